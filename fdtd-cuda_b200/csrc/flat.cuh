// Direct E and H passes: the Yee updates with the CPML recursions and, for a
// plane wave at normal incidence, the TFSF corrections, one launch per pass
// over the whole grid.
//
// A field plane is contiguous in memory (NY rows of PX values), so a thread
// takes one 16-byte vector of it (4 FP32 or 2 FP64 cells along x) counted
// over the whole plane, whatever NX is, and KZ planes of it one after the
// other.  Every neighbour is then a load at a constant offset (+-PX, +-plane)
// or the next lane's register (+-1), and nothing is staged: the loads of a
// plane do not depend on one another, and the +-1 rows and planes come out
// of L1 and L2.
//
// Why this form: the passes are bound by the bytes of the six fields (9
// values a cell and pass) at large grids and by latency at small ones.  The
// ring of shared-memory stages (staged.cuh) walks 8 to 32 planes per CTA
// with a barrier each; a small grid fills the GPU only for a short chain of
// such steps, and the CPML tiles of a large one stall on their psi loads.
// Pass times, us, H / E, staged against this form: FP32 64^3 10.3/10.3 and
// 6.2/6.2, 96^3 12.8/16.5 and 8.3/9.3, 128^3 24.5/23.2 and 16.1/17.1, 256^3
// 131/141 and 120/124 (5.7 and 5.5 TB/s of algorithmic bytes), 384x384x256
// 270/289 and 248/262; FP64 256^3 236/240 and 227/237 (6.0 and 5.8 TB/s).
// What bounds it: up to 128^3 the latency of one thread's few planes, above it
// DRAM, short of the copy rate because 16 warps a multiprocessor (128 registers)
// hold the loads in flight.  Fewer registers spill (80: twice the time), psi
// loaded after the fields costs the 256^3 E pass 124 -> 156, one plane a thread
// everywhere re-reads planes from DRAM (H 120 -> 159), L2 prefetches of the
// planes ahead 121 -> 130.
//
// The line, the dispersive cells and the TFSF increments ride in the two
// launches: a step in seven launches on side streams was 13.5 us at 64^3 and
// 292 us for the 256^3 dimer with these passes, in two 9.1 and 267.  (Beyond one
// wave of blocks the dispersive cells have launches of their own: cells_apart,
// fdtd.cu.)
#pragma once
#include "kernels.cuh"

namespace fdtd {

template <typename T>
struct alignas(16) Vec {
  static constexpr int N = 16 / (int)sizeof(T);
  T v[N];
};
template <typename T>
__device__ __forceinline__ Vec<T> ldv(const T* p) {
  return *reinterpret_cast<const Vec<T>*>(p);
}
// the same through the read-only path: values no thread of the launch writes
__device__ __forceinline__ Vec<float> ldgv(const float* p) {
  const float4 x = __ldg(reinterpret_cast<const float4*>(p));
  return Vec<float>{{x.x, x.y, x.z, x.w}};
}
__device__ __forceinline__ Vec<double> ldgv(const double* p) {
  const double2 x = __ldg(reinterpret_cast<const double2*>(p));
  return Vec<double>{{x.x, x.y}};
}
template <typename T>
__device__ __forceinline__ void stv(T* p, const Vec<T>& x) {
  *reinterpret_cast<Vec<T>*>(p) = x;
}
template <typename T>
__device__ __forceinline__ Vec<T> zerov() {
  Vec<T> r;
#pragma unroll
  for (int l = 0; l < Vec<T>::N; l++) r.v[l] = T(0);
  return r;
}

// Threads per block of the forms with a ring, and the most the others take: those
// also run with 128, which fills the last wave of a small grid better.
constexpr int kFlatThreads = 256;

// A thread's own vectors of the planes to come, copied into shared memory
// asynchronously S - 1 planes ahead.  No other thread reads them, so the ring
// needs no barrier: it stands in for registers that would hold the loads of
// several planes.
constexpr int kFlatRing = 4;
constexpr int kFlatRingBytes = kFlatRing * 6 * kFlatThreads * 16;
template <typename T>
struct FlatRing {
  unsigned base;
  __device__ __forceinline__ void init() {
    extern __shared__ __align__(16) unsigned char flat_smem[];
    base = (unsigned)__cvta_generic_to_shared(flat_smem) + threadIdx.x * 16u;
  }
  __device__ __forceinline__ void issue(int st, int a, const T* p) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(base + (unsigned)((st * 6 + a) * kFlatThreads * 16)),
                 "l"(p));
  }
  __device__ __forceinline__ Vec<float> get(int st, int a, float) {
    Vec<float> r;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n"
                 : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3])
                 : "r"(base + (unsigned)((st * 6 + a) * kFlatThreads * 16)));
    return r;
  }
  __device__ __forceinline__ Vec<double> get(int st, int a, double) {
    Vec<double> r;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];\n"
                 : "=d"(r.v[0]), "=d"(r.v[1])
                 : "r"(base + (unsigned)((st * 6 + a) * kFlatThreads * 16)));
    return r;
  }
  __device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
  __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(kFlatRing - 2) : "memory"); }
};
// a line another plane of this thread will need, into L2
template <typename T>
__device__ __forceinline__ void flat_touch(const T* p) {
  asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}

// CPML of one vector and one axis: psi <- b psi + c diff / d per lane, and the
// field += sg coef psi.  Lanes whose cell is not updated come with c = 0 (their
// psi is and stays zero); skip = lanes of dispersive cells, whose psi belongs to
// the dispersive-cell update.
template <typename T>
__device__ __forceinline__ T lane_of(const T& x, int) { return x; }
template <typename T>
__device__ __forceinline__ T lane_of(const Vec<T>& x, int l) { return x.v[l]; }
template <typename T, typename B, typename C>
__device__ __forceinline__ void psi_vec(T* p, const Vec<T>& old, const B& b, const Vec<T>& c, T inv_d,
                                        const Vec<T>& diff, Vec<T>& v, T sg, const C& coef, unsigned skip = 0) {
  constexpr int N = Vec<T>::N;
  Vec<T> ps;
#pragma unroll
  for (int l = 0; l < N; l++) {
    ps.v[l] = rfma(lane_of(b, l), old.v[l], rmul(rmul(c.v[l], diff.v[l]), inv_d));
    v.v[l] = rfma(sg * lane_of(coef, l), ps.v[l], v.v[l]);
  }
  if (!skip) stv(p, ps);
  else {
#pragma unroll
    for (int l = 0; l < N; l++)
      if (!((skip >> l) & 1)) p[l] = ps.v[l];
  }
}
template <typename T>
__device__ __forceinline__ T sum(const Vec<T>& x) {
  T r = x.v[0];
#pragma unroll
  for (int l = 1; l < Vec<T>::N; l++) r += x.v[l];
  return r;
}
// a coefficient on the lanes of m, 0 on the others
template <typename T, typename C>
__device__ __forceinline__ Vec<T> keep_lanes(unsigned m, const C& c) {
  Vec<T> r;
#pragma unroll
  for (int l = 0; l < Vec<T>::N; l++) r.v[l] = (m >> l) & 1 ? lane_of(c, l) : T(0);
  return r;
}

// Lanes of the vector at i0 whose cell index lies in [lo, hi).
template <int N>
__device__ __forceinline__ unsigned lanes_in(int i0, int lo, int hi) {
  unsigned m = 0;
#pragma unroll
  for (int l = 0; l < N; l++) m |= (i0 + l >= lo && i0 + l < hi) ? 1u << l : 0u;
  return m;
}
template <typename T>
__device__ __forceinline__ void add_lanes(Vec<T>& v, unsigned m, T x) {
#pragma unroll
  for (int l = 0; l < Vec<T>::N; l++)
    if ((m >> l) & 1) v.v[l] += x;
}

// The step's TFSF increments (tfsf_inc_at, kernels.cuh) in a pass.  The wave
// runs along z, so that on the x and y faces only the z component takes one: a
// lane of the vector on an x face and the lanes of a row on a y face.  Which,
// and on which side, is fixed along a thread's planes and kept in one word:
// bits 0-3 the x face's lane, 4-7 the y face's lanes, 8 / 9 their sides
// (finding them per plane cost the 256^3 H pass 8 us of 121, as did keeping
// masks and pointers apart, which spills).  One side a vector is enough because
// the passes take boxes of 4 cells and more only (tfsf_box_fuses, fdtd.cu).  The
// z faces are two planes of the grid.  half = 0: hz, half-open in x and y; half = 1: ez, closed in x and y.
template <typename T>
__device__ __forceinline__ unsigned flat_faces(const SimView<T>& s, int half, int i0, int j) {
  constexpr int N = Vec<T>::N;
  const int NX = s.NX, NY = s.NY, Tx = s.tf.Tx, Ty = s.tf.Ty, off = half ? 0 : 1;
  unsigned m = 0;
  if (j >= Ty && j < NY - Ty + half) {
    const int lo = Tx - off - i0, hi = NX - Tx - i0;
    if (lo >= 0 && lo < N) m |= 1u << lo;
    if (hi >= 0 && hi < N) m |= 1u << hi | 256u;
  }
  if (j == Ty - off || j == NY - Ty) m |= lanes_in<N>(i0, Tx, NX - Tx + half) << 4 | (j == NY - Ty ? 512u : 0u);
  return m;
}
// H pass (UPDATE_hx/hy/hz, main.cu:762-1044) of the vector vq of the plane,
// planes k0 .. k0+KZ-1.  Same arithmetic and order per cell as h_pass_tile
// (staged.cuh); the H half of CORRECT_X/Y/Z is added to the updated value
// from the step's increments (incH) when the view carries them.
template <typename T, bool RING, bool TFSF>
__device__ __forceinline__ void h_flat_cells(const SimView<T>& s, unsigned vq, int k0, int kz) {
  constexpr int N = Vec<T>::N;
  const int NX = s.NX, NY = s.NY, NZ = s.NZ, PX = s.PX;
  const unsigned PXV = (unsigned)PX / N, NV = PXV * (unsigned)NY;
  const bool in = vq < NV;
  if (!in) vq = NV - 1;  // takes part in the shuffles, stores nothing
  const int j = (int)(vq / PXV), i0 = (int)(vq - (unsigned)j * PXV) * N;
  const unsigned plane = (unsigned)s.plane, c0 = vq * N;  // 32-bit cell offsets (the host checks the range)
  const bool per = s.periodic != 0;
  const bool hasy = per || j + 1 < NY;
  // offset of the +y row; the last row of a bounded grid reads itself (its
  // hx and hz are not updated)
  const int oj = j + 1 < NY ? PX : (per ? -(NY - 1) * PX : 0);
  const unsigned lane = threadIdx.x & 31;
  const unsigned on = lanes_in<N>(i0, 0, per ? NX : NX - 1);  // lanes with a +x neighbour
  const Vec<T> ikx = ldgv(s.cp[0].inv_khd + i0);
  const T iky = ldg(s.cp[1].inv_khd + j);
  const T che = s.che, chh = s.chh;
  // CPML slabs of this vector
  const int xs = s.cp[0].Nc <= 0 ? -1 : i0 < s.cp[0].Wn ? i0 : (i0 + N > s.cp[0].fb ? i0 - s.cp[0].fb + s.cp[0].Wn : -1);
  const bool yfar = j >= s.cp[1].F;
  // (the far y slab follows the near one, NZ planes of Nc rows on)
  const int ys = s.cp[1].Nc <= 0 ? -1 : j < s.cp[1].Nc ? j : (yfar && j < NY - 1 ? j - s.cp[1].F + NZ * s.cp[1].Nc : -1);
  const int Ncz = s.cp[2].Nc, Fz = s.cp[2].F;
  // next vector's first value along x, from the next lane
  const bool edge = lane == 31 || i0 + N >= PX;
  const int ox = i0 + N < PX ? N : (per ? N - PX : 0);
  const T* incH = TFSF && s.incH ? s.incH + (size_t)(s.clk->th & 1) * 12 * NZ : nullptr;
  const unsigned face = incH ? flat_faces(s, 0, i0, j) : 0u;
  // downwards: Ex and Ey of plane k + 1 come in registers, and the plane's own
  // loads are all of plane k, with the +y row's just loaded by its own thread
  const int k1 = min(k0 + kz, NZ);
  const unsigned b1 = (unsigned)min(k1, NZ - 1) * plane + c0;
  Vec<T> exn = ldgv(s.E[0] + b1), eyn = ldgv(s.E[1] + b1);
  FlatRing<T> ring;
  int st = 0;
  auto issue = [&](int stage, int k) {
    if (k >= k0) {
      const unsigned b = (unsigned)k * plane + c0;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        ring.issue(stage, c, s.E[c] + b);
        ring.issue(stage, 3 + c, s.H[c] + b);
      }
    }
    ring.commit();
  };
  if (RING) {
    ring.init();
#pragma unroll
    for (int q = 0; q < kFlatRing - 1; q++) issue(q, k1 - 1 - q);
  }
#pragma unroll 1
  for (int k = k1 - 1; k >= k0; k--) {
    const unsigned b = (unsigned)k * plane + c0;
    const bool hask = k + 1 < NZ;
    // every load of the plane
    const Vec<T> exj = ldgv(s.E[0] + b + oj), ezj = ldgv(s.E[2] + b + oj);
    Vec<T> ex, ey, ez, hx, hy, hz;
    if (!RING) {
      ex = ldgv(s.E[0] + b); ey = ldgv(s.E[1] + b); ez = ldgv(s.E[2] + b);
      hx = ldv(s.H[0] + b); hy = ldv(s.H[1] + b); hz = ldv(s.H[2] + b);
    }
    T eyi = T(0), ezi = T(0);
    if (edge) { eyi = ldg(s.E[1] + b + ox); ezi = ldg(s.E[2] + b + ox); }
    const T ikz = ldg(s.cp[2].inv_khd + k);
    unsigned ozo = 0, oxo = 0, oyo = 0;  // offsets in the psi arrays
    Vec<T> ox0, ox1, oy0, oy1, oz0, oz1;
    int zs = -1;
    if (hask && Ncz > 0) zs = k < Ncz ? k : (k >= Fz ? k - Fz + Ncz : -1);
    if (zs >= 0) {
      ozo = (unsigned)zs * plane + c0;
      oz0 = ldv(s.psiH_N[0][1] + ozo); oz1 = ldv(s.psiH_N[1][0] + ozo);
    }
    if (xs >= 0 && hask) {
      oxo = ((unsigned)k * NY + j) * s.cp[0].W + xs;
      ox0 = ldv(s.psiH_N[1][1] + oxo); ox1 = ldv(s.psiH_N[2][0] + oxo);
    }
    if (ys >= 0 && hask) {
      oyo = ((unsigned)k * s.cp[1].Nc + ys) * PX + i0;
      oy0 = ldv(s.psiH_N[0][0] + oyo); oy1 = ldv(s.psiH_N[2][1] + oyo);
    }
    if (RING) {
      if (k > k0) {  // the next plane's psi
        if (xs >= 0) {
          const unsigned o = ((unsigned)(k - 1) * NY + j) * s.cp[0].W + xs;
          flat_touch(s.psiH_N[1][1] + o);
          flat_touch(s.psiH_N[2][0] + o);
        }
        if (ys >= 0) {
          const unsigned o = ((unsigned)(k - 1) * s.cp[1].Nc + ys) * PX + i0;
          flat_touch(s.psiH_N[0][0] + o);
          flat_touch(s.psiH_N[2][1] + o);
        }
      }
      ring.wait();
      issue(st == 0 ? kFlatRing - 1 : st - 1, k - (kFlatRing - 1));
      ex = ring.get(st, 0, T(0)); ey = ring.get(st, 1, T(0)); ez = ring.get(st, 2, T(0));
      hx = ring.get(st, 3, T(0)); hy = ring.get(st, 4, T(0)); hz = ring.get(st, 5, T(0));
      st = st == kFlatRing - 1 ? 0 : st + 1;
    }
    T fx = T(0), fy = T(0);  // TFSF increments (loaded last: they wait for the clock)
    if (TFSF && face && k >= s.tf.Tz && k <= NZ - s.tf.Tz) {
      if (face & 15u) fx = incH[tfsf_inc_at(0, (face >> 8) & 1, 1, NZ) + k];
      if (face & 240u) fy = incH[tfsf_inc_at(1, (face >> 9) & 1, 0, NZ) + k];
    }
    {
      const T a = __shfl_down_sync(0xFFFFFFFFu, ey.v[0], 1), c = __shfl_down_sync(0xFFFFFFFFu, ez.v[0], 1);
      if (!edge) { eyi = a; ezi = c; }
    }
    // differences
    Vec<T> dzy, dzx, dyz, dyx, dxz, dxy;  // d(ey)/dz, d(ex)/dz, d(ez)/dy, d(ex)/dy, d(ez)/dx, d(ey)/dx
#pragma unroll
    for (int l = 0; l < N; l++) {
      dzy.v[l] = rsub(eyn.v[l], ey.v[l]);
      dzx.v[l] = rsub(exn.v[l], ex.v[l]);
      dyz.v[l] = rsub(ezj.v[l], ez.v[l]);
      dyx.v[l] = rsub(exj.v[l], ex.v[l]);
      dxz.v[l] = rsub(l + 1 < N ? ez.v[l + 1 < N ? l + 1 : 0] : ezi, ez.v[l]);
      dxy.v[l] = rsub(l + 1 < N ? ey.v[l + 1 < N ? l + 1 : 0] : eyi, ey.v[l]);
    }
    Vec<T> vx, vy, vz;
#pragma unroll
    for (int l = 0; l < N; l++) {
      vx.v[l] = rfma(che, rcurl(dzy.v[l], ikz, dyz.v[l], iky), rmul(chh, hx.v[l]));
      vy.v[l] = rfma(che, rcurl(dxz.v[l], ikx.v[l], dzx.v[l], ikz), rmul(chh, hy.v[l]));
      vz.v[l] = rfma(che, rcurl(dyx.v[l], iky, dxy.v[l], ikx.v[l]), rmul(chh, hz.v[l]));
    }
    // CPML (cells with every index below N-1, main.cu:829); per axis in the
    // order z, x, y
    if (hasy && in) {
      if (zs >= 0) {
        const T bz = ldg(s.cp[2].bh + k);
        const Vec<T> cz = keep_lanes<T>(on, ldg(s.cp[2].ch + k));
        psi_vec(s.psiH_N[0][1] + ozo, oz0, bz, cz, s.cp[2].inv_d, dzy, vx, T(1), che);
        psi_vec(s.psiH_N[1][0] + ozo, oz1, bz, cz, s.cp[2].inv_d, dzx, vy, T(-1), che);
      }
      if (xs >= 0 && hask) {
        const Vec<T> bx = ldgv(s.cp[0].bh + i0), cx = ldgv(s.cp[0].ch + i0);  // zero at NX-1
        psi_vec(s.psiH_N[1][1] + oxo, ox0, bx, cx, s.cp[0].inv_d, dxz, vy, T(1), che);
        psi_vec(s.psiH_N[2][0] + oxo, ox1, bx, cx, s.cp[0].inv_d, dxy, vz, T(-1), che);
      }
      if (ys >= 0 && hask) {
        const T by = ldg(s.cp[1].bh + j);
        const Vec<T> cy = keep_lanes<T>(on, ldg(s.cp[1].ch + j));
        psi_vec(s.psiH_N[0][0] + oyo, oy0, by, cy, s.cp[1].inv_d, dyz, vx, T(-1), che);
        psi_vec(s.psiH_N[2][1] + oyo, oy1, by, cy, s.cp[1].inv_d, dyx, vz, T(1), che);
      }
    }
#pragma unroll
    for (int l = 0; l < N; l++) {
      hx.v[l] = vx.v[l];
      if ((on >> l) & 1) { hy.v[l] = vy.v[l]; hz.v[l] = vz.v[l]; }
    }
    // the H half of CORRECT_X/Y/Z
    if (TFSF && face) {
      add_lanes(hz, face & 15u, fx);
      add_lanes(hz, (face >> 4) & 15u, fy);
    }
    if (TFSF && incH && (k == s.tf.Tz - 1 || k == NZ - s.tf.Tz)) {
      const int side = k == NZ - s.tf.Tz, Tx = s.tf.Tx, Ty = s.tf.Ty;
      if (j >= Ty && j < NY - Ty) add_lanes(hx, lanes_in<N>(i0, Tx, min(NX, NX - Tx + 1)), incH[tfsf_inc_at(2, side, 0, NZ) + k]);
      if (j >= Ty && j <= NY - Ty) add_lanes(hy, lanes_in<N>(i0, Tx, NX - Tx), incH[tfsf_inc_at(2, side, 1, NZ) + k]);
    }
    if (in) {
      if (hasy && hask) stv(s.H[0] + b, hx);
      if (hask) stv(s.H[1] + b, hy);
      if (hasy) stv(s.H[2] + b, hz);
    }
    exn = ex;
    eyn = ey;
  }
}

// Which blocks of a launch do what: block 0 the 1D line (H launches with
// line = 1), the next nrole blocks the dispersive cells, the others the
// grid's vectors, nbx blocks a group of kz planes.
struct FlatGrid {
  unsigned nbx, nrole;
  int kz, line;
};

// The H launch of a step: the H pass, with it the 1D line's step (it reads E
// at the probe cell, the line and the clock, and writes the line's other E
// buffer, the line's H and the increments of the coming E and H launches, none
// of which the pass reads) and the hydrodynamic currents (they read E^n, the
// currents and densities).
template <typename T, bool RING, bool TFSF, bool HYDRO>
__global__ void __launch_bounds__(kFlatThreads, 2)
    h_flat(const __grid_constant__ SimView<T> s, const __grid_constant__ MetalView<T> m,
           const __grid_constant__ LineArgs line, size_t probe_id, const __grid_constant__ FlatGrid g) {
  unsigned b = blockIdx.x;
  if (g.line) {
    if (b == 0) {
      line_step_body(line, s, probe_id, line.clk->th);
      return;
    }
    b--;
  }
  if (HYDRO) {
    if (b < g.nrole) {
      hydro_p_any(s, m, s.clk->th, (int)(b * blockDim.x + threadIdx.x));
      return;
    }
    b -= g.nrole;
  }
  const unsigned kb = b / g.nbx, xb = b - kb * g.nbx;
  h_flat_cells<T, RING, TFSF>(s, xb * blockDim.x + threadIdx.x, (int)kb * g.kz, g.kz);
}

// E pass (UPDATE_ex/ey/ez, main.cu:1048-1912) of the vector vq, planes k0 ..
// k0+KZ-1: e_pass_tile's arithmetic and order per cell (CPML per axis in the
// order z, y, x).  The E half of CORRECT_X/Y/Z goes in before the update.
// Dispersive components are left to the dispersive-cell kernels, which run
// beside this one: a vector with such a cell stores lane by lane.
template <typename T, bool RING, bool TFSF>
__device__ __forceinline__ void e_flat_cells(const SimView<T>& s, unsigned vq, int k0, int kz) {
  constexpr int N = Vec<T>::N;
  const int NX = s.NX, NY = s.NY, NZ = s.NZ, PX = s.PX;
  const unsigned PXV = (unsigned)PX / N, NV = PXV * (unsigned)NY;
  const bool in = vq < NV;
  if (!in) vq = NV - 1;
  const int j = (int)(vq / PXV), i0 = (int)(vq - (unsigned)j * PXV) * N;
  const unsigned plane = (unsigned)s.plane, c0 = vq * N;
  const bool per = s.periodic != 0;
  const int oj = j > 0 ? -PX : (per ? (NY - 1) * PX : 0);
  const unsigned lane = threadIdx.x & 31;
  // lanes whose ex, ey, ez are updated in this column (main.cu:1172, 1476,
  // 1767; every column when periodic, main.cu:1072, 1364, 1668)
  const bool jlo = per || j > 0, jhi = per || j < NY - 1;
  const unsigned onx = lanes_in<N>(i0, 0, per ? NX : NX - 1), onyz = onx & ~(!per && i0 == 0 ? 1u : 0u);
  const bool rowy = in && jhi, rowxz = rowy && jlo;
  const Vec<T> ikx = ldgv(s.cp[0].inv_ked + i0);
  const T iky = ldg(s.cp[1].inv_ked + j);
  const T cee0 = s.cee[0], ceh0 = s.ceh[0];
  const bool inbox = i0 + N > s.mat_lo[0] && i0 < s.mat_hi[0] && j >= s.mat_lo[1] && j < s.mat_hi[1];
  const int xs = s.cp[0].Nc <= 0 ? -1 : i0 < s.cp[0].Wn ? i0 : (i0 + N > s.cp[0].fb ? i0 - s.cp[0].fb + s.cp[0].Wn : -1);
  const bool yfar = j >= s.cp[1].F;
  const int ys = s.cp[1].Nc <= 0 ? -1 : j <= s.cp[1].Nc ? j : (yfar ? j - s.cp[1].F + NZ * (s.cp[1].Nc + 1) : -1);
  const int Ncz = s.cp[2].Nc, Fz = s.cp[2].F;
  const bool edge = lane == 0 || i0 == 0;
  const int ox = i0 > 0 ? -1 : (per ? PX - 1 : 0);
  const unsigned face = TFSF && s.incE ? flat_faces(s, 1, i0, j) : 0u;
  T check = T(0);
  const unsigned bm = (unsigned)min(max(k0 - 1, 0), NZ - 1) * plane + c0;  // (a batch block's groups may start past NZ)
  Vec<T> hxm = ldgv(s.H[0] + bm), hym = ldgv(s.H[1] + bm);
  const int k1 = min(k0 + kz, NZ);
  FlatRing<T> ring;
  int st = 0;
  auto issue = [&](int stage, int k) {
    if (k < k1) {
      const unsigned b = (unsigned)k * plane + c0;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        ring.issue(stage, c, s.H[c] + b);
        ring.issue(stage, 3 + c, s.E[c] + b);
      }
    }
    ring.commit();
  };
  if (RING) {
    ring.init();
#pragma unroll
    for (int q = 0; q < kFlatRing - 1; q++) issue(q, k0 + q);
  }
#pragma unroll 1
  for (int k = k0; k < k1; k++) {
    const unsigned b = (unsigned)k * plane + c0;
    const bool okz = k < NZ - 1, hasz = k > 0;
    // every load of the plane
    const Vec<T> hxj = ldgv(s.H[0] + b + oj), hzj = ldgv(s.H[2] + b + oj);
    Vec<T> hx, hy, hz, ex, ey, ez;
    if (!RING) {
      hx = ldgv(s.H[0] + b); hy = ldgv(s.H[1] + b); hz = ldgv(s.H[2] + b);
      ex = ldv(s.E[0] + b); ey = ldv(s.E[1] + b); ez = ldv(s.E[2] + b);
    }
    T hyi = T(0), hzi = T(0);
    if (edge) { hyi = ldg(s.H[1] + b + ox); hzi = ldg(s.H[2] + b + ox); }
    const T ikz = ldg(s.cp[2].inv_ked + k);
    unsigned ozo = 0, oxo = 0, oyo = 0;  // offsets in the psi arrays
    Vec<T> ox0, ox1, oy0, oy1, oz0, oz1;
    int zs = -1;
    if (okz && Ncz > 0) zs = k <= Ncz ? k : (k >= Fz ? k - Fz + Ncz + 1 : -1);
    if (zs >= 0) {
      ozo = (unsigned)zs * plane + c0;
      oz0 = ldv(s.psiE_N[0][1] + ozo); oz1 = ldv(s.psiE_N[1][0] + ozo);
    }
    if (ys >= 0 && okz) {
      oyo = ((unsigned)k * (s.cp[1].Nc + 1) + ys) * PX + i0;
      oy0 = ldv(s.psiE_N[0][0] + oyo); oy1 = ldv(s.psiE_N[2][1] + oyo);
    }
    if (xs >= 0 && okz) {
      oxo = ((unsigned)k * NY + j) * s.cp[0].W + xs;
      ox0 = ldv(s.psiE_N[1][1] + oxo); ox1 = ldv(s.psiE_N[2][0] + oxo);
    }
    // dielectric classes and dispersive components
    Vec<T> ceh;
    unsigned mx = 0, my = 0, mz = 0;
#pragma unroll
    for (int l = 0; l < N; l++) ceh.v[l] = ceh0;
    if (inbox && k >= s.mat_lo[2] && k < s.mat_hi[2]) {
      const uint8_t* mp = s.mat + b;
#pragma unroll
      for (int l = 0; l < N; l++) {
        const unsigned m = mp[l];
        mx |= (m & 1u) << l;
        my |= ((m >> 1) & 1u) << l;
        mz |= ((m >> 2) & 1u) << l;
        if (m >> 3) ceh.v[l] = s.ceh[m >> 3];
      }
    }
    if (RING) {
      if (k + 1 < k1) {  // the next plane's psi
        if (xs >= 0) {
          const unsigned o = ((unsigned)(k + 1) * NY + j) * s.cp[0].W + xs;
          flat_touch(s.psiE_N[1][1] + o);
          flat_touch(s.psiE_N[2][0] + o);
        }
        if (ys >= 0) {
          const unsigned o = ((unsigned)(k + 1) * (s.cp[1].Nc + 1) + ys) * PX + i0;
          flat_touch(s.psiE_N[0][0] + o);
          flat_touch(s.psiE_N[2][1] + o);
        }
      }
      ring.wait();
      issue(st == 0 ? kFlatRing - 1 : st - 1, k + (kFlatRing - 1));
      hx = ring.get(st, 0, T(0)); hy = ring.get(st, 1, T(0)); hz = ring.get(st, 2, T(0));
      ex = ring.get(st, 3, T(0)); ey = ring.get(st, 4, T(0)); ez = ring.get(st, 5, T(0));
      st = st == kFlatRing - 1 ? 0 : st + 1;
    }
    T fx = T(0), fy = T(0);  // TFSF increments
    if (TFSF && face && k >= s.tf.Tz && k < NZ - s.tf.Tz) {
      if (face & 15u) fx = s.incE[tfsf_inc_at(0, (face >> 8) & 1, 1, NZ) + k];
      if (face & 240u) fy = s.incE[tfsf_inc_at(1, (face >> 9) & 1, 0, NZ) + k];
    }
    {
      const T a = __shfl_up_sync(0xFFFFFFFFu, hy.v[N - 1], 1), c = __shfl_up_sync(0xFFFFFFFFu, hz.v[N - 1], 1);
      if (!edge) { hyi = a; hzi = c; }
    }
    const bool upx = rowxz && hasz && okz, upy = rowy && hasz && okz, upz = rowxz && okz;
    // the E half of CORRECT_X/Y/Z, before the update
    if (TFSF && face) {
      add_lanes(ez, face & 15u, fx);
      add_lanes(ez, (face >> 4) & 15u, fy);
    }
    if (TFSF && s.incE && (k == s.tf.Tz || k == NZ - s.tf.Tz)) {
      const int side = k == NZ - s.tf.Tz, Tx = s.tf.Tx, Ty = s.tf.Ty;
      if (j >= Ty && j <= NY - Ty) add_lanes(ex, lanes_in<N>(i0, Tx, NX - Tx), s.incE[tfsf_inc_at(2, side, 0, NZ) + k]);
      if (j >= Ty && j < NY - Ty) add_lanes(ey, lanes_in<N>(i0, Tx, min(NX, NX - Tx + 1)), s.incE[tfsf_inc_at(2, side, 1, NZ) + k]);
    }
    Vec<T> dyz, dzy, dzx, dxz, dxy, dyx;  // d(hz)/dy, d(hy)/dz, d(hx)/dz, d(hz)/dx, d(hy)/dx, d(hx)/dy
#pragma unroll
    for (int l = 0; l < N; l++) {
      dyz.v[l] = rsub(hz.v[l], hzj.v[l]);
      dzy.v[l] = rsub(hy.v[l], hym.v[l]);
      dzx.v[l] = rsub(hx.v[l], hxm.v[l]);
      dxz.v[l] = rsub(hz.v[l], l > 0 ? hz.v[l > 0 ? l - 1 : 0] : hzi);
      dxy.v[l] = rsub(hy.v[l], l > 0 ? hy.v[l > 0 ? l - 1 : 0] : hyi);
      dyx.v[l] = rsub(hx.v[l], hxj.v[l]);
    }
    Vec<T> vx, vy, vz;
#pragma unroll
    for (int l = 0; l < N; l++) {
      vx.v[l] = rfma(ceh.v[l], rcurl(dyz.v[l], iky, dzy.v[l], ikz), rmul(cee0, ex.v[l]));
      vy.v[l] = rfma(ceh.v[l], rcurl(dzx.v[l], ikz, dxz.v[l], ikx.v[l]), rmul(cee0, ey.v[l]));
      vz.v[l] = rfma(ceh.v[l], rcurl(dxy.v[l], ikx.v[l], dyx.v[l], iky), rmul(cee0, ez.v[l]));
    }
    // CPML (cells with i < NX-1, j < NY-1, k < NZ-1)
    if (zs >= 0) {
      const T bz = ldg(s.cp[2].be + k), cz = ldg(s.cp[2].ce + k);
      if (upx) psi_vec(s.psiE_N[0][1] + ozo, oz0, bz, keep_lanes<T>(onx, cz), s.cp[2].inv_d, dzy, vx, T(-1), ceh, mx);
      if (upy) psi_vec(s.psiE_N[1][0] + ozo, oz1, bz, keep_lanes<T>(onyz, cz), s.cp[2].inv_d, dzx, vy, T(1), ceh, my);
    }
    if (ys >= 0 && okz) {
      const T by = ldg(s.cp[1].be + j), cy = ldg(s.cp[1].ce + j);
      if (upx) psi_vec(s.psiE_N[0][0] + oyo, oy0, by, keep_lanes<T>(onx, cy), s.cp[1].inv_d, dyz, vx, T(1), ceh, mx);
      if (upz) psi_vec(s.psiE_N[2][1] + oyo, oy1, by, keep_lanes<T>(onyz, cy), s.cp[1].inv_d, dyx, vz, T(-1), ceh, mz);
    }
    if (xs >= 0 && okz) {
      const Vec<T> bx = ldgv(s.cp[0].be + i0);
      if (upy) psi_vec(s.psiE_N[1][1] + oxo, ox0, bx, keep_lanes<T>(onyz, ldgv(s.cp[0].ce_ey + i0)), s.cp[0].inv_d, dxz, vy, T(-1), ceh, my);
      if (upz) psi_vec(s.psiE_N[2][0] + oxo, ox1, bx, keep_lanes<T>(onyz, ldgv(s.cp[0].ce + i0)), s.cp[0].inv_d, dxy, vz, T(1), ceh, mz);
    }
#pragma unroll
    for (int l = 0; l < N; l++) {
      if ((onx >> l) & 1) ex.v[l] = vx.v[l];
      if ((onyz >> l) & 1) { ey.v[l] = vy.v[l]; ez.v[l] = vz.v[l]; }
    }
    if (!(mx | my | mz)) {
      if (upx) { stv(s.E[0] + b, ex); check += sum(ex); }
      if (upy) { stv(s.E[1] + b, ey); check += sum(ey); }
      if (upz) { stv(s.E[2] + b, ez); check += sum(ez); }
    } else {
#pragma unroll
      for (int l = 0; l < N; l++) {
        if (upx && !((mx >> l) & 1)) { s.E[0][b + l] = ex.v[l]; check += ex.v[l]; }
        if (upy && !((my >> l) & 1)) { s.E[1][b + l] = ey.v[l]; check += ey.v[l]; }
        if (upz && !((mz >> l) & 1)) { s.E[2][b + l] = ez.v[l]; check += ez.v[l]; }
      }
    }
    hxm = hx;
    hym = hy;
  }
  // NaN/Inf watchdog: a non-finite value makes the running sum non-finite
  if (!isfinite(check)) atomicOr(s.nonfinite, 1);
}

// The E launch of a step: the E pass and the dispersive cells (KIND 1 = the
// local model, 2 = the hydrodynamic model), which write disjoint cells.
template <typename T, bool RING, bool TFSF, int KIND>
__global__ void __launch_bounds__(kFlatThreads, 2)
    e_flat(const __grid_constant__ SimView<T> s, const __grid_constant__ MetalView<T> m,
           const __grid_constant__ FlatGrid g) {
  unsigned b = blockIdx.x;
  if (b == 0 && threadIdx.x == 0) s.clk->th = s.clk->t;
  if (KIND) {
    if (b < g.nrole) {
      const int q = (int)(b * blockDim.x + threadIdx.x), t = s.clk->t - 1;
      if (KIND == 1) metal_e_cell(s, m, t, q);
      else hydro_e_any(s, m, t, q);
      return;
    }
    b -= g.nrole;
  }
  const unsigned kb = b / g.nbx, xb = b - kb * g.nbx;
  e_flat_cells<T, RING, TFSF>(s, xb * blockDim.x + threadIdx.x, (int)kb * g.kz, g.kz);
}

}  // namespace fdtd
