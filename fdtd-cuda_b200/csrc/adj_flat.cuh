// The transposed Yee sub-steps of the adjoint as direct passes (flat.cuh): one
// launch each, CPML included.
//
// adj_h_flat adds to lambda_H what the E sub-step read from H: each updated E
// component, through the coefficient of each of its two H differences (sg ceh
// ik lambda_E, plus the psi adjoint's share in a CPML slab), adj_gather_h's
// sums.  adj_e_flat is the same for the H sub-step.  A cell needs its own six
// coefficients and two each of its three neighbours.  The pass computes all of
// them: those of the neighbour plane are carried in registers, those of the
// neighbour along x come from the next lane, those of the neighbour row are
// computed again from its adjoint and psi adjoint.  The psi adjoints have two
// buffers, by step parity, since a neighbour reads a psi adjoint that its own
// cell moves on.  Dispersive cells have their coefficients in the arrays a.a
// (adj_e_design, adj_hydro_e).  The scalings cee and chh are 1 (no losses in
// the reference's coefficients, setup.cu:2015-2062), which the host checks.
// Arithmetic and summation order are those of adj_e_coef / adj_gather_h /
// adj_h_coef / adj_gather_e.
//
// What this replaced: slab kernels that wrote coefficient arrays for the CPML
// cells, and gathers that read flags and arrays for every cell (19 to 24 values
// a cell and sub-step there against 9).  Backward, us a step: FP32 96^3 56.5 to
// 25.9, 65x71x61 36.8 to 22.4, 184x168x129 hydrodynamic 263 to 167; FP64 160^3
// 331 to 211.  Bound by latency up to 128^3, above it by DRAM with 16 warps a
// multiprocessor; the copy-ahead ring of flat.cuh gave nothing here (168 to 169),
// nor did the transposed current update as blocks of adj_h_flat (167 to 166).
#pragma once
#include "adjoint.cuh"
#include "flat.cuh"

namespace fdtd {

// Coefficient of one difference: sg ceh ik lambda; lam is zero on the lanes
// that are not updated.
template <typename T, typename C, typename K>
__device__ __forceinline__ Vec<T> adj_base(const Vec<T>& lam, T sg, const C& ceh, const K& ik) {
  Vec<T> r;
#pragma unroll
  for (int l = 0; l < Vec<T>::N; l++) r.v[l] = adj_mul(sg * lane_of(ceh, l) * lane_of(ik, l), lam.v[l]);
  return r;
}
// The CPML's part of it; the psi adjoint one step back goes to out (null: the
// cell is another thread's).
template <typename T, typename C, typename B>
__device__ __forceinline__ void adj_psi_vec(Vec<T>& coef, const Vec<T>& old, const Vec<T>& lam, T sg, const C& ceh,
                                            const B& b, const B& c, T inv_d, T* out) {
  Vec<T> nw;
#pragma unroll
  for (int l = 0; l < Vec<T>::N; l++) {
    const T tot = old.v[l] + sg * lane_of(ceh, l) * lam.v[l];
    nw.v[l] = lane_of(b, l) * tot;
    coef.v[l] += lane_of(c, l) * inv_d * tot;
  }
  if (out) stv(out, nw);
}
// lanes of dispersive cells take their coefficient from the array
template <typename T>
__device__ __forceinline__ void adj_array_lanes(Vec<T>& coef, unsigned m, const T* p) {
#pragma unroll
  for (int l = 0; l < Vec<T>::N; l++)
    if ((m >> l) & 1) coef.v[l] = p[l];
}

// dispersive bits per component and the E coefficient of a vector's cells
template <typename T>
struct AdjCells {
  unsigned m[3];
  Vec<T> ceh;
  __device__ __forceinline__ void load(const SimView<T>& s, int i0, int j, int k, unsigned id) {
    constexpr int N = Vec<T>::N;
    m[0] = m[1] = m[2] = 0;
#pragma unroll
    for (int l = 0; l < N; l++) ceh.v[l] = s.ceh[0];
    if (i0 + N > s.mat_lo[0] && i0 < s.mat_hi[0] && j >= s.mat_lo[1] && j < s.mat_hi[1] && k >= s.mat_lo[2] &&
        k < s.mat_hi[2]) {
#pragma unroll
      for (int l = 0; l < N; l++) {
        const unsigned x = s.mat[id + l];
#pragma unroll
        for (int c = 0; c < 3; c++) m[c] |= ((x >> c) & 1u) << l;
        if (x >> 3) ceh.v[l] = s.ceh[x >> 3];
      }
    }
  }
};

// x-axis coefficient of E component c (Ez slot 0, Ey slot 1) of one cell: the
// neighbour of a warp's last lane.
template <typename T>
__device__ __forceinline__ T adj_e_edge(const SimView<T>& s, const AdjView<T>& a, int par, int c, int i, int j, int k) {
  const int sl = c == 2 ? 0 : 1;
  if (!adj_e_act(s, c, i, j, k)) return T(0);
  const size_t id = fidx(s.PX, s.plane, i, j, k);
  const unsigned m = adj_mat(s, i, j, k, id);
  if (m & (1u << c)) return a.a[c][sl][id];
  const T sg = sl == 0 ? T(1) : T(-1), ceh = s.ceh[m >> 3], lam = a.lE[c][id];
  T coef = adj_mul(sg * ceh * ldg(s.cp[0].inv_ked + i), lam);
  const int xs = i < s.cp[0].Wn ? i : (i >= s.cp[0].fb ? i - s.cp[0].fb + s.cp[0].Wn : -1);
  if (xs >= 0) {
    const T tot = a.fE[c][sl][(size_t)par * a.fEn[c][sl] + ((size_t)k * s.NY + j) * s.cp[0].W + xs] + sg * ceh * lam;
    coef += ldg((c == 1 ? s.cp[0].ce_ey : s.cp[0].ce) + i) * s.cp[0].inv_d * tot;
  }
  return coef;
}
// the same of H component h (Hz slot 0, Hy slot 1): the neighbour of a warp's
// first lane
template <typename T>
__device__ __forceinline__ T adj_h_edge(const SimView<T>& s, const AdjView<T>& a, int par, int h, int i, int j, int k) {
  const int sl = h == 2 ? 0 : 1;
  if (!adj_h_act(s, h, i, j, k)) return T(0);
  const size_t id = fidx(s.PX, s.plane, i, j, k);
  const T sg = sl == 0 ? T(-1) : T(1), lam = a.lH[h][id];
  T coef = adj_mul(sg * s.che * ldg(s.cp[0].inv_khd + i), lam);
  const int xs = i < s.cp[0].Wn ? i : (i >= s.cp[0].fb ? i - s.cp[0].fb + s.cp[0].Wn : -1);
  if (xs >= 0 && j < s.NY - 1 && k < s.NZ - 1) {
    const T tot = a.fH[h][sl][(size_t)par * a.fHn[h][sl] + ((size_t)k * s.NY + j) * s.cp[0].W + xs] + sg * s.che * lam;
    coef += ldg(s.cp[0].ch + i) * s.cp[0].inv_d * tot;
  }
  return coef;
}

// z-slab plane of the psi arrays (near then far), -1 outside
template <typename T>
__device__ __forceinline__ int adj_zs(const CpmlAxis<T>& a, int k, int w) {
  return k < w ? k : (k >= a.F ? k - a.F + w : -1);
}
// row of a y slab in its psi array (plane 0): near rows, then NZ planes on the
// far ones; -1 outside
template <typename T>
__device__ __forceinline__ int adj_ys(const CpmlAxis<T>& a, int j, int w, int NZ) {
  return j < w ? j : (j >= a.F ? j - a.F + NZ * w : -1);
}

template <typename T>
__global__ void __launch_bounds__(kFlatThreads, 2)
    adj_h_flat(const __grid_constant__ SimView<T> s, const __grid_constant__ AdjView<T> a, unsigned nbx, int kz) {
  constexpr int N = Vec<T>::N;
  const int n = a.step[0], par = n & 1;
  if (blockIdx.x == 0 && threadIdx.x == 0) a.step[1] = n;  // adj_e_flat's
  const unsigned kb = blockIdx.x / nbx, xb = blockIdx.x - kb * nbx;
  const int NX = s.NX, NY = s.NY, NZ = s.NZ, PX = s.PX;
  const unsigned PXV = (unsigned)PX / N, NV = PXV * (unsigned)NY, plane = (unsigned)s.plane;
  unsigned vq = xb * blockDim.x + threadIdx.x;
  const bool in = vq < NV;
  if (!in) vq = NV - 1;
  const int j = (int)(vq / PXV), i0 = (int)(vq - (unsigned)j * PXV) * N;
  const unsigned c0 = vq * N;
  const unsigned onx = lanes_in<N>(i0, 0, NX - 1), onyz = onx & ~(i0 == 0 ? 1u : 0u);
  const bool last = (threadIdx.x & 31) == 31;
  const bool jlo = j > 0, jhi = j < NY - 1, j1 = j + 1 < NY, jhi1 = j + 1 < NY - 1;
  const int w0 = s.cp[1].Nc + 1, wz = s.cp[2].Nc + 1;
  const int xs = i0 < s.cp[0].Wn ? i0 : (i0 + N > s.cp[0].fb ? i0 - s.cp[0].fb + s.cp[0].Wn : -1);
  const int ys = adj_ys(s.cp[1], j, w0, NZ), ys1 = j1 ? adj_ys(s.cp[1], j + 1, w0, NZ) : -1;
  const T idx = s.cp[0].inv_d, idy = s.cp[1].inv_d, idz = s.cp[2].inv_d;
  const Vec<T> ikx = ldgv(s.cp[0].inv_ked + i0);
  const T iky = ldg(s.cp[1].inv_ked + j), iky1 = j1 ? ldg(s.cp[1].inv_ked + j + 1) : T(0);
  auto rd = [&](int c, int sl) { return a.fE[c][sl] + (par ? a.fEn[c][sl] : 0); };
  auto wr = [&](int c, int sl) { return a.fE[c][sl] + (par ? 0 : a.fEn[c][sl]); };
  const int k0 = (int)kb * kz, k1 = min(k0 + kz, NZ);
  // z-axis coefficients of Ey (slot 0) and Ex (slot 1) of plane k
  auto zcoef = [&](int k, const Vec<T>& lx, const Vec<T>& ly, const AdjCells<T>& m, bool own, Vec<T>& ay, Vec<T>& ax) {
    const T ik = ldg(s.cp[2].inv_ked + k);
    const unsigned id = (unsigned)k * plane + c0;
    ay = adj_base(ly, T(1), m.ceh, ik);
    ax = adj_base(lx, T(-1), m.ceh, ik);
    const int zs = adj_zs(s.cp[2], k, wz);
    if (zs >= 0) {
      const unsigned o = (unsigned)zs * plane + c0;
      const T b = ldg(s.cp[2].be + k), c = ldg(s.cp[2].ce + k);
      adj_psi_vec(ay, ldgv(rd(1, 0) + o), ly, T(1), m.ceh, b, c, idz, own ? wr(1, 0) + o : nullptr);
      adj_psi_vec(ax, ldgv(rd(0, 1) + o), lx, T(-1), m.ceh, b, c, idz, own ? wr(0, 1) + o : nullptr);
    }
    if (m.m[0] | m.m[1]) {
      adj_array_lanes(ay, m.m[1], a.a[1][0] + id);
      adj_array_lanes(ax, m.m[0], a.a[0][1] + id);
    }
  };
  Vec<T> ayn = zerov<T>(), axn = zerov<T>();  // of plane k + 1
  if (k1 < NZ) {
    const unsigned id = (unsigned)k1 * plane + c0;
    const bool act = jhi && k1 > 0 && k1 < NZ - 1;
    AdjCells<T> m;
    m.load(s, i0, j, k1, id);
    const Vec<T> lx = keep_lanes<T>(act && jlo ? onx & ~m.m[0] : 0u, ldgv(a.lE[0] + id));
    const Vec<T> ly = keep_lanes<T>(act ? onyz & ~m.m[1] : 0u, ldgv(a.lE[1] + id));
    zcoef(k1, lx, ly, m, false, ayn, axn);
  }
#pragma unroll 1
  for (int k = k1 - 1; k >= k0; k--) {
    const unsigned id = (unsigned)k * plane + c0;
    const bool klo = k > 0, khi = k < NZ - 1;
    Vec<T> ex = ldgv(a.lE[0] + id), ey = ldgv(a.lE[1] + id), ez = ldgv(a.lE[2] + id);
    Vec<T> exj = zerov<T>(), ezj = zerov<T>();
    if (j1) { exj = ldgv(a.lE[0] + id + PX); ezj = ldgv(a.lE[2] + id + PX); }
    Vec<T> hx = ldv(a.lH[0] + id), hy = ldv(a.lH[1] + id), hz = ldv(a.lH[2] + id);
    AdjCells<T> m, mj;
    m.load(s, i0, j, k, id);
    mj.load(s, i0, j + 1, k, j1 ? id + PX : id);
    T e20 = T(0), e11 = T(0);
    if (last) {
      e20 = adj_e_edge(s, a, par, 2, i0 + N, j, k);
      e11 = adj_e_edge(s, a, par, 1, i0 + N, j, k);
    }
    // the adjoints, zero where the component is not updated
    ex = keep_lanes<T>(jlo && jhi && klo && khi ? onx & ~m.m[0] : 0u, ex);
    ey = keep_lanes<T>(jhi && klo && khi ? onyz & ~m.m[1] : 0u, ey);
    ez = keep_lanes<T>(jlo && jhi && khi ? onyz & ~m.m[2] : 0u, ez);
    exj = keep_lanes<T>(jhi1 && klo && khi ? onx & ~mj.m[0] : 0u, exj);
    ezj = keep_lanes<T>(jhi1 && khi ? onyz & ~mj.m[2] : 0u, ezj);
    // z: Ey slot 0, Ex slot 1
    Vec<T> a10, a01;
    zcoef(k, ex, ey, m, in, a10, a01);
    // y: Ex slot 0, Ez slot 1, here and in the next row
    Vec<T> a00 = adj_base(ex, T(1), m.ceh, iky), a21 = adj_base(ez, T(-1), m.ceh, iky);
    Vec<T> a00y = adj_base(exj, T(1), mj.ceh, iky1), a21y = adj_base(ezj, T(-1), mj.ceh, iky1);
    if (ys >= 0) {
      const unsigned o = ((unsigned)k * w0 + ys) * PX + i0;
      const T b = ldg(s.cp[1].be + j), c = ldg(s.cp[1].ce + j);
      adj_psi_vec(a00, ldgv(rd(0, 0) + o), ex, T(1), m.ceh, b, c, idy, in ? wr(0, 0) + o : nullptr);
      adj_psi_vec(a21, ldgv(rd(2, 1) + o), ez, T(-1), m.ceh, b, c, idy, in ? wr(2, 1) + o : nullptr);
    }
    if (ys1 >= 0) {
      const unsigned o = ((unsigned)k * w0 + ys1) * PX + i0;
      const T b = ldg(s.cp[1].be + j + 1), c = ldg(s.cp[1].ce + j + 1);
      adj_psi_vec<T>(a00y, ldgv(rd(0, 0) + o), exj, T(1), mj.ceh, b, c, idy, nullptr);
      adj_psi_vec<T>(a21y, ldgv(rd(2, 1) + o), ezj, T(-1), mj.ceh, b, c, idy, nullptr);
    }
    // x: Ez slot 0, Ey slot 1
    Vec<T> a20 = adj_base(ez, T(1), m.ceh, ikx), a11 = adj_base(ey, T(-1), m.ceh, ikx);
    if (xs >= 0) {
      const unsigned o = ((unsigned)k * NY + j) * s.cp[0].W + xs;
      const Vec<T> b = ldgv(s.cp[0].be + i0), c = ldgv(s.cp[0].ce + i0), cey = ldgv(s.cp[0].ce_ey + i0);
      adj_psi_vec(a20, ldgv(rd(2, 0) + o), ez, T(1), m.ceh, b, c, idx, in ? wr(2, 0) + o : nullptr);
      adj_psi_vec(a11, ldgv(rd(1, 1) + o), ey, T(-1), m.ceh, b, cey, idx, in ? wr(1, 1) + o : nullptr);
    }
    if (m.m[0] | m.m[1] | m.m[2]) {
      adj_array_lanes(a00, m.m[0], a.a[0][0] + id);
      adj_array_lanes(a21, m.m[2], a.a[2][1] + id);
      adj_array_lanes(a20, m.m[2], a.a[2][0] + id);
      adj_array_lanes(a11, m.m[1], a.a[1][1] + id);
    }
    if (mj.m[0] | mj.m[2]) {
      adj_array_lanes(a00y, mj.m[0], a.a[0][0] + id + PX);
      adj_array_lanes(a21y, mj.m[2], a.a[2][1] + id + PX);
    }
    {
      const T p = __shfl_down_sync(0xFFFFFFFFu, a20.v[0], 1), q = __shfl_down_sync(0xFFFFFFFFu, a11.v[0], 1);
      if (!last) { e20 = p; e11 = q; }
    }
#pragma unroll
    for (int l = 0; l < N; l++) {
      const T a20x = l + 1 < N ? a20.v[l + 1 < N ? l + 1 : 0] : e20, a11x = l + 1 < N ? a11.v[l + 1 < N ? l + 1 : 0] : e11;
      hx.v[l] = hx.v[l] + (a10.v[l] - ayn.v[l] + a21.v[l] - a21y.v[l]);
      hy.v[l] = hy.v[l] + (a01.v[l] - axn.v[l] + a20.v[l] - a20x);
      hz.v[l] = hz.v[l] + (a00.v[l] - a00y.v[l] + a11.v[l] - a11x);
    }
    if (in) {
      stv(a.lH[0] + id, hx);
      stv(a.lH[1] + id, hy);
      stv(a.lH[2] + id, hz);
    }
    ayn = a10;
    axn = a01;
  }
}

template <typename T>
__global__ void __launch_bounds__(kFlatThreads, 2)
    adj_e_flat(const __grid_constant__ SimView<T> s, const __grid_constant__ AdjView<T> a, unsigned nbx, int kz) {
  constexpr int N = Vec<T>::N;
  const int n = a.step[1], par = n & 1;
  if (blockIdx.x == 0 && threadIdx.x == 0) a.step[0] = n - 1;  // the step is done: the next one's
  const unsigned kb = blockIdx.x / nbx, xb = blockIdx.x - kb * nbx;
  const int NX = s.NX, NY = s.NY, NZ = s.NZ, PX = s.PX;
  const unsigned PXV = (unsigned)PX / N, NV = PXV * (unsigned)NY, plane = (unsigned)s.plane;
  unsigned vq = xb * blockDim.x + threadIdx.x;
  const bool in = vq < NV;
  if (!in) vq = NV - 1;
  const int j = (int)(vq / PXV), i0 = (int)(vq - (unsigned)j * PXV) * N;
  const unsigned c0 = vq * N;
  const unsigned on = lanes_in<N>(i0, 0, NX - 1), all = lanes_in<N>(i0, 0, NX);
  const bool first = (threadIdx.x & 31) == 0;
  const bool jhi = j < NY - 1, j1 = j > 0;
  const int w0 = s.cp[1].Nc, wz = s.cp[2].Nc;
  const int xs = s.cp[0].Nc <= 0 ? -1 : i0 < s.cp[0].Wn ? i0 : (i0 + N > s.cp[0].fb ? i0 - s.cp[0].fb + s.cp[0].Wn : -1);
  // (the H slabs end at index N - 2)
  const int ys = jhi ? adj_ys(s.cp[1], j, w0, NZ) : -1, ys1 = j1 ? adj_ys(s.cp[1], j - 1, w0, NZ) : -1;
  const T idx = s.cp[0].inv_d, idy = s.cp[1].inv_d, idz = s.cp[2].inv_d, che = s.che;
  const Vec<T> ikx = ldgv(s.cp[0].inv_khd + i0);
  const T iky = ldg(s.cp[1].inv_khd + j), iky1 = j1 ? ldg(s.cp[1].inv_khd + j - 1) : T(0);
  auto rd = [&](int c, int sl) { return a.fH[c][sl] + (par ? a.fHn[c][sl] : 0); };
  auto wr = [&](int c, int sl) { return a.fH[c][sl] + (par ? 0 : a.fHn[c][sl]); };
  const int k0 = (int)kb * kz, k1 = min(k0 + kz, NZ);
  // z-axis coefficients of Hy (slot 0) and Hx (slot 1) of plane k
  auto zcoef = [&](int k, const Vec<T>& lx, const Vec<T>& ly, bool own, Vec<T>& ay, Vec<T>& ax) {
    const T ik = ldg(s.cp[2].inv_khd + k);
    ay = adj_base(ly, T(-1), che, ik);
    ax = adj_base(lx, T(1), che, ik);
    const int zs = jhi && k < NZ - 1 ? adj_zs(s.cp[2], k, wz) : -1;
    if (zs >= 0) {
      const unsigned o = (unsigned)zs * plane + c0;
      const T b = ldg(s.cp[2].bh + k), c = ldg(s.cp[2].ch + k);
      adj_psi_vec(ay, ldgv(rd(1, 0) + o), ly, T(-1), che, b, c, idz, own ? wr(1, 0) + o : nullptr);
      adj_psi_vec(ax, ldgv(rd(0, 1) + o), keep_lanes<T>(on, lx), T(1), che, b, c, idz, own ? wr(0, 1) + o : nullptr);
    }
  };
  Vec<T> ayn = zerov<T>(), axn = zerov<T>();  // of plane k - 1
  if (k0 > 0) {
    const unsigned id = (unsigned)(k0 - 1) * plane + c0;
    const Vec<T> lx = keep_lanes<T>(jhi && k0 - 1 < NZ - 1 ? all : 0u, ldgv(a.lH[0] + id));
    const Vec<T> ly = keep_lanes<T>(k0 - 1 < NZ - 1 ? on : 0u, ldgv(a.lH[1] + id));
    zcoef(k0 - 1, lx, ly, false, ayn, axn);
  }
#pragma unroll 1
  for (int k = k0; k < k1; k++) {
    const unsigned id = (unsigned)k * plane + c0;
    const bool khi = k < NZ - 1;
    Vec<T> hx = ldgv(a.lH[0] + id), hy = ldgv(a.lH[1] + id), hz = ldgv(a.lH[2] + id);
    Vec<T> hxj = zerov<T>(), hzj = zerov<T>();
    if (j1) { hxj = ldgv(a.lH[0] + id - PX); hzj = ldgv(a.lH[2] + id - PX); }
    Vec<T> ex = ldv(a.lE[0] + id), ey = ldv(a.lE[1] + id), ez = ldv(a.lE[2] + id);
    T e20 = T(0), e11 = T(0);
    if (first && i0 > 0) {
      e20 = adj_h_edge(s, a, par, 2, i0 - 1, j, k);
      e11 = adj_h_edge(s, a, par, 1, i0 - 1, j, k);
    }
    // Yee range: the two other indices below N-1 (row j - 1 always is along y)
    hx = keep_lanes<T>(jhi && khi ? all : 0u, hx);
    hy = keep_lanes<T>(khi ? on : 0u, hy);
    hz = keep_lanes<T>(jhi ? on : 0u, hz);
    hxj = keep_lanes<T>(khi ? all : 0u, hxj);
    hzj = keep_lanes<T>(on, hzj);
    Vec<T> a10, a01;
    zcoef(k, hx, hy, in, a10, a01);
    // y: Hx slot 0, Hz slot 1, here and in the row before
    Vec<T> a00 = adj_base(hx, T(-1), che, iky), a21 = adj_base(hz, T(1), che, iky);
    Vec<T> a00y = adj_base(hxj, T(-1), che, iky1), a21y = adj_base(hzj, T(1), che, iky1);
    if (ys >= 0 && khi) {
      const unsigned o = ((unsigned)k * w0 + ys) * PX + i0;
      const T b = ldg(s.cp[1].bh + j), c = ldg(s.cp[1].ch + j);
      adj_psi_vec(a00, ldgv(rd(0, 0) + o), keep_lanes<T>(on, hx), T(-1), che, b, c, idy, in ? wr(0, 0) + o : nullptr);
      adj_psi_vec(a21, ldgv(rd(2, 1) + o), hz, T(1), che, b, c, idy, in ? wr(2, 1) + o : nullptr);
    }
    if (ys1 >= 0 && khi) {
      const unsigned o = ((unsigned)k * w0 + ys1) * PX + i0;
      const T b = ldg(s.cp[1].bh + j - 1), c = ldg(s.cp[1].ch + j - 1);
      adj_psi_vec<T>(a00y, ldgv(rd(0, 0) + o), keep_lanes<T>(on, hxj), T(-1), che, b, c, idy, nullptr);
      adj_psi_vec<T>(a21y, ldgv(rd(2, 1) + o), hzj, T(1), che, b, c, idy, nullptr);
    }
    // x: Hz slot 0, Hy slot 1
    Vec<T> a20 = adj_base(hz, T(-1), che, ikx), a11 = adj_base(hy, T(1), che, ikx);
    if (xs >= 0 && jhi && khi) {
      const unsigned o = ((unsigned)k * NY + j) * s.cp[0].W + xs;
      const Vec<T> b = ldgv(s.cp[0].bh + i0), c = ldgv(s.cp[0].ch + i0);
      adj_psi_vec(a20, ldgv(rd(2, 0) + o), hz, T(-1), che, b, c, idx, in ? wr(2, 0) + o : nullptr);
      adj_psi_vec(a11, ldgv(rd(1, 1) + o), hy, T(1), che, b, c, idx, in ? wr(1, 1) + o : nullptr);
    }
    {
      const T p = __shfl_up_sync(0xFFFFFFFFu, a20.v[N - 1], 1), q = __shfl_up_sync(0xFFFFFFFFu, a11.v[N - 1], 1);
      if (!first) { e20 = p; e11 = q; }
    }
#pragma unroll
    for (int l = 0; l < N; l++) {
      const T a20x = l > 0 ? a20.v[l > 0 ? l - 1 : 0] : e20, a11x = l > 0 ? a11.v[l > 0 ? l - 1 : 0] : e11;
      ex.v[l] += ayn.v[l] - a10.v[l] + a21y.v[l] - a21.v[l];
      ey.v[l] += axn.v[l] - a01.v[l] + a20x - a20.v[l];
      ez.v[l] += a00y.v[l] - a00.v[l] + a11x - a11.v[l];
    }
    if (in) {
      stv(a.lE[0] + id, ex);
      stv(a.lE[1] + id, ey);
      stv(a.lE[2] + id, ez);
    }
    ayn = a10;
    axn = a01;
  }
}

}  // namespace fdtd
