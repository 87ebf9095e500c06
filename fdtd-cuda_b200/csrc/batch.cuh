// Batched independent simulations (no counterpart in the reference: its
// trials loop, main.cu:2435, runs one simulation after another, and FP64
// builds allow one trial, main.cu:2386-2389).
//
// Every member is an ordinary fdtd_sim (its own fields, tables, DFT and
// clock); the batch adds, in device memory, one descriptor per member and the
// block lists of its two launches per time step.  A block of a list is the line
// step of a member, a share of its dispersive cells, or vectors and planes of
// its grid (the direct passes, flat.cuh):
//   h_flat_batch      line steps, hydrodynamic currents, H pass
//   tfsf_apply_batch  only with members at oblique incidence
//   e_flat_batch      dispersive cells, E pass
//   metal_e_batch, hydro_p_batch, hydro_e_batch  the dispersive cells beside the
//                     E pass where they are many (cells_apart, fdtd.cu)
//   dft_sample        one launch every dft_every steps, blockIdx.z = member
//   the DFT contraction (job, phasors, product, reset), one launch each,
//                     every 32 samples; it contracts each member's first
//                     ring half once that holds 64 samples
// so the launch count per step does not grow with the member count, and
// small members that could not fill the GPU alone share it.  A step, us, against
// persistent staged passes over a work queue with the other kernels in launches
// of their own: 16 members of 48-128 381 to 305, 4 of 44-60 51.7 to 22.6, 40 of
// 48-128 875 to 700, 8 of 80-140 FP64 697 to 473; bound by DRAM for the large
// members (16 warps a multiprocessor).  Runs of
// 32 * dft_every steps are captured into one CUDA graph and replayed.  A batch
// with a member that the direct passes do not take (the staged ones are forced,
// or it is beyond their 32-bit offsets) steps its members one after another.
//
// This file is included at the end of fdtd.cu (it uses the simulation
// internals defined there).

namespace fdtd {

template <typename T>
struct BatchSim {
  SimView<T> v;
  MetalView<T> m;
  LineArgs line;
  DftView dft;
  TfsfTable tf_h, tf_e;
  T* ring;
  double2* tw;
  DevClock* clk;
  size_t probe_id;
};

template <typename T>
__global__ void tfsf_apply_batch(const BatchSim<T>* __restrict__ b) {
  const BatchSim<T>& x = b[blockIdx.y];
  tfsf_apply_body(x.v, x.tf_h, x.tf_e, x.line);
}

// A block of a batch launch: (member | role << 20, first vector's block or the
// block of the role, first plane, planes per thread | z groups << 16).  A grid
// block's 256 threads are z groups of 256 / groups vectors each, one above the
// other.
enum { kItemGrid = 0, kItemLine = 1, kItemCells = 2 };

// The member's view in shared memory: the passes read it where a single
// simulation's kernel reads its parameters.
template <typename T>
__device__ __forceinline__ void batch_view(SimView<T>& dst, const SimView<T>& src) {
  static_assert(sizeof(SimView<T>) % 8 == 0, "copied in 8-byte words");
  const unsigned long long* p = reinterpret_cast<const unsigned long long*>(&src);
  unsigned long long* q = reinterpret_cast<unsigned long long*>(&dst);
  for (int w = threadIdx.x; w < (int)(sizeof(SimView<T>) / 8); w += kFlatThreads) q[w] = __ldg(p + w);
  __syncthreads();
}

template <typename T, bool RING, bool HYDRO>
__global__ void __launch_bounds__(kFlatThreads, 2)
    h_flat_batch(const BatchSim<T>* __restrict__ b, const int4* __restrict__ items) {
  __shared__ SimView<T> s;
  const int4 it = items[blockIdx.x];
  const BatchSim<T>& x = b[it.x & 0xFFFFF];
  const int role = it.x >> 20;
  if (role == kItemLine) {
    line_step_body(x.line, x.v, x.probe_id, x.clk->th);
    return;
  }
  if (HYDRO && role == kItemCells) {
    hydro_p_any(x.v, x.m, x.clk->th, it.y * kFlatThreads + (int)threadIdx.x);
    return;
  }
  batch_view(s, x.v);
  const int kz = it.w & 0xFFFF, vx = kFlatThreads / (it.w >> 16), tz = threadIdx.x / vx;
  h_flat_cells<T, RING, true>(s, (unsigned)(it.y * vx + (threadIdx.x - tz * vx)), it.z + tz * kz, kz);
}
template <typename T, bool RING, bool HYDRO>
__global__ void __launch_bounds__(kFlatThreads, 2)
    e_flat_batch(const BatchSim<T>* __restrict__ b, const int4* __restrict__ items) {
  __shared__ SimView<T> s;
  const int4 it = items[blockIdx.x];
  const BatchSim<T>& x = b[it.x & 0xFFFFF];
  if ((it.x >> 20) == kItemCells) {
    const int q = it.y * kFlatThreads + (int)threadIdx.x, t = x.clk->t - 1;
    if (HYDRO) hydro_e_any(x.v, x.m, t, q);
    else metal_e_cell(x.v, x.m, t, q);
    return;
  }
  if (it.y == 0 && it.z == 0 && threadIdx.x == 0) x.clk->th = x.clk->t;
  batch_view(s, x.v);
  const int kz = it.w & 0xFFFF, vx = kFlatThreads / (it.w >> 16), tz = threadIdx.x / vx;
  e_flat_cells<T, RING, true>(s, (unsigned)(it.y * vx + (threadIdx.x - tz * vx)), it.z + tz * kz, kz);
}
template <typename T>
__global__ void metal_e_batch(const BatchSim<T>* __restrict__ b) {
  const BatchSim<T>& x = b[blockIdx.y];
  metal_e_cell(x.v, x.m, x.clk->t - 1, (int)(blockIdx.x * blockDim.x + threadIdx.x));
}
template <typename T>
__global__ void hydro_p_batch(const BatchSim<T>* __restrict__ b) {
  const BatchSim<T>& x = b[blockIdx.y];
  hydro_p_any(x.v, x.m, x.clk->t - 1, (int)(blockIdx.x * blockDim.x + threadIdx.x));
}
template <typename T, int PART>
__global__ void hydro_e_batch(const BatchSim<T>* __restrict__ b) {
  const BatchSim<T>& x = b[blockIdx.y];
  hydro_e_part<T, PART>(x.v, x.m, x.clk->t - 1, (int)(blockIdx.x * blockDim.x + threadIdx.x));
}
template <typename T>
__global__ void dft_sample_batch(const BatchSim<T>* __restrict__ b) {
  const BatchSim<T>& x = b[blockIdx.z];
  dft_sample_body(x.v, x.dft, x.ring, x.clk);
}
// The members keep filling the first half of their rings: every launch
// period each member's job is its samples once the half cannot take
// another period (dft_job_ready_body), contracted, then the half emptied.
// A flush before the spectra are read goes through the member's own
// contraction kernels (fdtd_spectral_finalize) and takes the samples no job
// has taken.
template <typename T>
__global__ void dft_job_ready_batch(const BatchSim<T>* __restrict__ b) {
  dft_job_ready_body(b[blockIdx.y].clk);
}
template <typename T>
__global__ void dft_twiddles_batch(const BatchSim<T>* __restrict__ b) {
  const BatchSim<T>& x = b[blockIdx.y];
  dft_twiddles_body(x.dft, x.clk, x.tw);
}
template <typename T>
__global__ void __launch_bounds__(128) dft_contract_batch(const BatchSim<T>* __restrict__ b) {
  const BatchSim<T>& x = b[blockIdx.y];
  dft_contract_body(x.dft, x.ring, x.clk, x.tw);
}
template <typename T>
__global__ void dft_job_done_batch(const BatchSim<T>* __restrict__ b) {
  dft_job_done_body(b[blockIdx.y].clk);
}

}  // namespace fdtd

constexpr int kBatchBucket = 16;  // members bucketed by their largest edge, 16 cells a bucket
constexpr int kBatchMaxBuckets = FDTD_BATCH_MAX_BUCKETS;

struct fdtd_batch {
  int device = 0;
  bool fp64 = false, hydro = false;
  std::vector<std::unique_ptr<fdtd_sim>> sims;
  std::vector<std::unique_ptr<DevBuf>> bufs;
  void* descs = nullptr;  // BatchSim<T>[n]
  // block lists of the two launches (H, E), kept and grown: the graph of the
  // step holds their addresses
  int4* items[2] = {nullptr, nullptr};
  int nitems[2] = {0, 0};
  size_t items_cap[2] = {0, 0};
  bool direct = true;  // every member takes the direct passes
  bool tail = false;   // the last blocks take fewer planes (batch_split_tail)
  bool ring = false;   // their planes are copied ahead
  // size buckets and their planes per thread; member -> bucket
  int nbuckets = 0;
  int bucket_lo[kBatchMaxBuckets] = {}, bucket_members[kBatchMaxBuckets] = {}, bucket_kz[kBatchMaxBuckets] = {};
  float bucket_ms[kBatchMaxBuckets] = {};
  std::vector<int> member_bucket;
  int sms = 0;
  bool tuned = false;
  bool cells_apart = false;  // the dispersive cells run as launches of their own
  unsigned g_m = 0;          // their blocks of 128 (the largest member's)
  cudaStream_t side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  unsigned g_f = 0, g_s = 0, g_tw = 0, g_c = 0;
  int t = 0, host_nsamp = 0, dft_every = 0, tend = 0;
  long long kernels = 0, graph_launches = 0, graph_kernels = 0;
  cudaGraphExec_t graph = nullptr;
  cudaStream_t cap = nullptr;

  ~fdtd_batch() {
    if (graph) cudaGraphExecDestroy(graph);
    if (cap) cudaStreamDestroy(cap);
    if (side) cudaStreamDestroy(side);
    if (fork) cudaEventDestroy(fork);
    if (join) cudaEventDestroy(join);
  }
  template <typename U>
  cudaError_t alloc(U** out, size_t count) {
    auto b = std::make_unique<DevBuf>();
    cudaError_t e = b->alloc(count * sizeof(U));
    if (e != cudaSuccess) return e;
    *out = static_cast<U*>(b->p);
    bufs.push_back(std::move(b));
    return cudaSuccess;
  }
};

// Planes per thread as blocks: a block spans up to 8 planes, or one run where
// that is longer (its z-chunk), short runs of planes as 2, 4 or 8 groups of
// threads above one another.
static int batch_groups(int kz) { return kz == 1 ? 8 : kz == 2 ? 4 : kz <= 4 ? 2 : 1; }
static int batch_kchunk(int kz) { return kz * batch_groups(kz); }

// The grid blocks of member i with kz planes per thread.
template <typename T>
static void batch_member_items(const fdtd_sim* s, int i, int kz, std::vector<int4>& out) {
  const int kc = batch_kchunk(kz), groups = batch_groups(kz), vx = kFlatThreads / groups;
  const int nv = (int)(s->plane / Vec<T>::N), nx = (nv + vx - 1) / vx;
  for (int k = 0; k < s->NZ; k += kc)
    for (int x = 0; x < nx; x++) out.push_back(make_int4(i, x, k, kz | groups << 16));
}

template <typename T>
static fdtd_status batch_build(fdtd_batch* b) {
  const int n = (int)b->sims.size();
  std::vector<BatchSim<T>> d(n);
  long long cells = 0;
  for (int i = 0; i < n; i++) {
    fdtd_sim* s = b->sims[i].get();
    BatchSim<T>& x = d[i];
    x.v = view<T>(s);
    x.m = mview<T>(s);
    x.line = s->line;
    x.dft = s->dft;
    if (!s->fused_tfsf) {  // else the passes apply the corrections
      x.tf_h = s->tf_h;
      x.tf_e = s->tf_e;
    }
    b->direct = b->direct && s->hcfg.kz > 0;
    x.ring = static_cast<T*>(s->ring);
    x.tw = s->twiddles;
    x.clk = s->clk;
    x.probe_id = s->probe_id;
    auto blocks = [](long long cells, int per) { return (unsigned)((cells + per - 1) / per); };
    const long long nc = (long long)s->nmetal[0] + s->nmetal[1] + s->nmetal[2];
    cells += nc;
    b->g_m = std::max(b->g_m, blocks(nc, 128));
    b->g_f = std::max(b->g_f, blocks((long long)x.tf_h.n + x.tf_e.n, 256));
    int maxn = 0;
    for (int f = 0; f < 12; f++) maxn = std::max(maxn, s->dft.face[f].na * s->dft.face[f].nb);
    b->g_s = std::max(b->g_s, blocks(maxn, 256));
    b->g_tw = std::max(b->g_tw, blocks(2LL * kRingSlots * s->dft.nf, 256));
    b->g_c = std::max(b->g_c, (unsigned)(s->dft.rows / kDftRows));
  }
  BatchSim<T>* dd;
  CUDA_TRY(b->alloc(&dd, n));
  CUDA_TRY(cudaMemcpy(dd, d.data(), n * sizeof(BatchSim<T>), cudaMemcpyHostToDevice));
  b->descs = dd;
  // size buckets by the largest edge
  b->member_bucket.assign(n, 0);
  std::vector<int> key(n);
  for (int i = 0; i < n; i++) {
    const fdtd_sim* s = b->sims[i].get();
    key[i] = (std::max(s->NX, std::max(s->NY, s->NZ)) - 1) / kBatchBucket;
  }
  std::vector<int> keys(key);
  std::sort(keys.begin(), keys.end());
  keys.erase(std::unique(keys.begin(), keys.end()), keys.end());
  if ((int)keys.size() > kBatchMaxBuckets) {  // merge the largest ones into the last bucket
    keys.resize(kBatchMaxBuckets);
  }
  b->nbuckets = (int)keys.size();
  for (int q = 0; q < b->nbuckets; q++) {
    b->bucket_lo[q] = keys[q] * kBatchBucket + 1;
    b->bucket_kz[q] = 8;
    b->bucket_members[q] = 0;
  }
  for (int i = 0; i < n; i++) {
    int q = (int)(std::lower_bound(keys.begin(), keys.end(), key[i]) - keys.begin());
    q = std::min(q, b->nbuckets - 1);
    b->member_bucket[i] = q;
    b->bucket_members[q]++;
  }
  CUDA_TRY(cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, b->device));
  b->cells_apart = cells_apart(cells, b->sms, 8);
  if (b->cells_apart) {
    CUDA_TRY(cudaStreamCreateWithFlags(&b->side, cudaStreamNonBlocking));
    CUDA_TRY(cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming));
    CUDA_TRY(cudaEventCreateWithFlags(&b->join, cudaEventDisableTiming));
  }
  {
    const void* k[4] = {(const void*)h_flat_batch<T, true, false>, (const void*)h_flat_batch<T, true, true>,
                        (const void*)e_flat_batch<T, true, false>, (const void*)e_flat_batch<T, true, true>};
    for (const void* f : k)
      CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kFlatRingBytes));
  }
  CUDA_TRY(cudaFuncSetAttribute(dft_contract_batch<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)dft_smem_bytes<T>()));
  return FDTD_OK;
}

// A launch ends when its last blocks do, and those started up to a whole block's
// time apart: the blocks that the GPU starts last get a quarter of the planes
// each, four in the place of one (each re-reads a plane at its end, which is why
// not all blocks are that short).  Kept where it measures faster: a step, us, 16
// members of 48-128 304.6 to 301.6, 40 of 48-128 700 to 687, 8 of 80-140 FP64
// 473.4 to 467.6; 10 of 60-100 144.8 either way.
static void batch_split_tail(fdtd_batch* b, std::vector<int4>& v) {
  const size_t last = std::min(v.size(), (size_t)2 * b->sms);
  std::vector<int4> t(v.end() - last, v.end());
  v.resize(v.size() - last);
  for (const int4& it : t) {
    const int kz = it.w & 0xFFFF, groups = it.w >> 16;
    if ((it.x >> 20) != kItemGrid || kz < 8 || kz % 4) { v.push_back(it); continue; }
    const int NZ = b->sims[it.x & 0xFFFFF]->NZ;
    for (int p = 0; p < 4; p++) {
      const int z = it.z + p * groups * (kz / 4);
      if (z < NZ) v.push_back(make_int4(it.x, it.y, z, kz / 4 | groups << 16));
    }
  }
}

// The block lists for the current planes per thread, uploaded.  only: a bucket,
// or -1 for all of them; grid: the grid blocks alone (for timing).
template <typename T>
static fdtd_status batch_upload_items(fdtd_batch* b, int only = -1, bool grid = false) {
  const int n = (int)b->sims.size();
  for (int p = 0; p < 2; p++) {
    std::vector<int4> v;
    if (!grid && p == 0)
      for (int i = 0; i < n; i++) v.push_back(make_int4(i | kItemLine << 20, 0, 0, 0));
    if (!grid && !b->cells_apart && (p == 1 || b->hydro))
      for (int i = 0; i < n; i++) {
        const fdtd_sim* s = b->sims[i].get();
        const int nb = (s->nmetal[0] + s->nmetal[1] + s->nmetal[2] + kFlatThreads - 1) / kFlatThreads;
        for (int q = 0; q < nb; q++) v.push_back(make_int4(i | kItemCells << 20, q, 0, 0));
      }
    for (int i = 0; i < n; i++)
      if (only < 0 || b->member_bucket[i] == only)
        batch_member_items<T>(b->sims[i].get(), i, b->bucket_kz[b->member_bucket[i]], v);
    if (only < 0 && b->tail) batch_split_tail(b, v);
    b->nitems[p] = (int)v.size();
    if (v.empty()) continue;
    if (!b->items[p] || b->items_cap[p] < v.size()) {
      int4* d;
      CUDA_TRY(b->alloc(&d, v.size()));
      b->items[p] = d;
      b->items_cap[p] = v.size();
    }
    CUDA_TRY(cudaMemcpy(b->items[p], v.data(), v.size() * sizeof(int4), cudaMemcpyHostToDevice));
  }
  return FDTD_OK;
}

template <typename T, bool RING, bool HYDRO>
static void batch_launch_form(fdtd_batch* b, int p, cudaStream_t st) {
  const BatchSim<T>* d = static_cast<const BatchSim<T>*>(b->descs);
  const dim3 g(b->nitems[p]), blk(kFlatThreads);
  const size_t smem = RING ? kFlatRingBytes : 0;
  if (p == 0) h_flat_batch<T, RING, HYDRO><<<g, blk, smem, st>>>(d, b->items[0]);
  else e_flat_batch<T, RING, HYDRO><<<g, blk, smem, st>>>(d, b->items[1]);
}
template <typename T>
static void batch_launch(fdtd_batch* b, int p, cudaStream_t st) {
  if (b->ring) {
    if (b->hydro) batch_launch_form<T, true, true>(b, p, st);
    else batch_launch_form<T, true, false>(b, p, st);
  } else {
    if (b->hydro) batch_launch_form<T, false, true>(b, p, st);
    else batch_launch_form<T, false, false>(b, p, st);
  }
}

template <typename T>
static void batch_enqueue_step(fdtd_batch* b, cudaStream_t st) {
  if (!b->direct) {
    for (auto& s : b->sims) {
      const long long k0 = s->kernels;
      enqueue_step<T>(s.get(), st);
      b->kernels += s->kernels - k0;
    }
    b->t++;
    return;
  }
  const int n = (int)b->sims.size();
  const BatchSim<T>* d = static_cast<const BatchSim<T>*>(b->descs);
  int k = 2;
  batch_launch<T>(b, 0, st);
  if (b->g_f) { tfsf_apply_batch<T><<<dim3(b->g_f, n), 256, 0, st>>>(d); k++; }
  if (b->cells_apart) {
    const dim3 g(b->g_m, n);
    cudaEventRecord(b->fork, st);
    cudaStreamWaitEvent(b->side, b->fork, 0);
    if (!b->hydro) {
      metal_e_batch<T><<<g, 128, 0, b->side>>>(d);
      k++;
    } else {
      hydro_p_batch<T><<<g, 128, 0, b->side>>>(d);
      hydro_e_batch<T, 1><<<g, 128, 0, b->side>>>(d);
      hydro_e_batch<T, 2><<<g, 128, 0, b->side>>>(d);
      k += 3;
    }
    cudaEventRecord(b->join, b->side);
  }
  batch_launch<T>(b, 1, st);
  if (b->cells_apart) cudaStreamWaitEvent(st, b->join, 0);
  if (b->dft_every > 0 && b->t % b->dft_every == 0) {
    dft_sample_batch<T><<<dim3(b->g_s, 12, n), 256, 0, st>>>(d);
    k++;
    if (++b->host_nsamp == kSampleBlock) {
      // the members' rings fill together: these contract once they are full
      dft_job_ready_batch<T><<<dim3(1, n), 1, 0, st>>>(d);
      dft_twiddles_batch<T><<<dim3(b->g_tw, n), 256, 0, st>>>(d);
      dft_contract_batch<T><<<dim3(b->g_c, n), 128, dft_smem_bytes<T>(), st>>>(d);
      dft_job_done_batch<T><<<dim3(1, n), 1, 0, st>>>(d);
      k += 4;
      b->host_nsamp = 0;
    }
  }
  b->kernels += k;
  b->t++;
}

// Mean device time of `reps` runs of both passes over the current block lists
// (grid blocks), after one untimed run.  On the zero state the passes leave the
// fields at zero.
template <typename T>
static fdtd_status batch_time_passes(fdtd_batch* b, int reps, float* ms) {
  cudaEvent_t e0, e1;
  CUDA_TRY(cudaEventCreate(&e0));
  CUDA_TRY(cudaEventCreate(&e1));
  auto go = [&]() {
    batch_launch<T>(b, 0, 0);
    batch_launch<T>(b, 1, 0);
  };
  go();
  cudaEventRecord(e0, 0);
  for (int r = 0; r < reps; r++) go();
  cudaEventRecord(e1, 0);
  cudaError_t e = cudaEventSynchronize(e1);
  float t = 0.f;
  if (e == cudaSuccess) e = cudaEventElapsedTime(&t, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (e != cudaSuccess) return fail(FDTD_ERR_CUDA, std::string("batch tuning: ") + cudaGetErrorString(e));
  *ms = t / reps;
  return FDTD_OK;
}

// The autotuner of the batch's passes (no counterpart in the reference): per
// size bucket the planes per thread (2, 4, 8 or 16) with the bucket's members
// alone, then the same number for every bucket over the whole batch: members
// alone want short runs, which fill the GPU, a full batch longer ones, which
// re-read less.  FDTD_TUNE=0, or a batch under 2^20 cells, takes the most
// planes, up to 8, that leave two blocks a multiprocessor.
// FDTD_PASS=flat:KZ[:RING] fixes both (blocks have 256 threads whatever else it
// says), FDTD_BATCH_TAIL=0 / 1 whether the last blocks are split.
template <typename T>
static fdtd_status batch_tune(fdtd_batch* b) {
  if (!b->direct) return FDTD_OK;
  long long cells = 0, vecs = 0;
  for (const auto& s : b->sims) {
    cells += s->ncell;
    vecs += (long long)(s->ncell / Vec<T>::N);
  }
  int kz = 1;
  while (kz < 8 && vecs / (2 * kz * kFlatThreads) >= 2LL * b->sms) kz *= 2;
  for (int q = 0; q < b->nbuckets; q++) b->bucket_kz[q] = kz;
  const char* env = std::getenv("FDTD_TUNE");
  const char* tail = std::getenv("FDTD_BATCH_TAIL");
  const char* force = std::getenv("FDTD_PASS");
  b->tail = tail && tail[0] == '1';
  int fz = 0, fring = 0;
  if (force && std::sscanf(force, "flat:%d:%d", &fz, &fring) >= 1) {  // (the members' creation has checked it)
    for (int q = 0; q < b->nbuckets; q++) b->bucket_kz[q] = std::min(fz, 0x7FFF);
    b->ring = fring != 0;
    return batch_upload_items<T>(b);
  }
  fdtd_status st;
  if ((env && env[0] == '0') || cells < (1LL << 20)) return batch_upload_items<T>(b);
  std::vector<int> chosen(b->nbuckets, kz);
  float ms;
  for (int q = 0; q < b->nbuckets; q++) {
    float best = 1e30f;
    for (int z : {2, 4, 8, 16}) {
      b->bucket_kz[q] = z;
      if ((st = batch_upload_items<T>(b, q, true)) != FDTD_OK) return st;
      if ((st = batch_time_passes<T>(b, 3, &ms)) != FDTD_OK) return st;
      if (ms < best) { best = ms; chosen[q] = z; }
    }
    b->bucket_ms[q] = best;
  }
  // -1: each bucket's own; with and without the ring
  float best = 1e30f;
  int best_z = -1;
  bool best_ring = false;
  for (int z : {-1, 4, 8, 16, 32}) {
    for (int q = 0; q < b->nbuckets; q++) b->bucket_kz[q] = z < 0 ? chosen[q] : z;
    if ((st = batch_upload_items<T>(b, -1, true)) != FDTD_OK) return st;
    for (int ring = 0; ring < 2; ring++) {
      if (ring ? z >= 0 && z < 8 : z == 32) continue;
      b->ring = ring;
      if ((st = batch_time_passes<T>(b, 3, &ms)) != FDTD_OK) return st;
      if (ms < best) { best = ms; best_z = z; best_ring = ring; }
    }
  }
  for (int q = 0; q < b->nbuckets; q++) b->bucket_kz[q] = best_z < 0 ? chosen[q] : best_z;
  b->ring = best_ring;
  b->tuned = true;
  if (tail) return batch_upload_items<T>(b);
  b->tail = true;
  if ((st = batch_upload_items<T>(b, -1, true)) != FDTD_OK) return st;
  if ((st = batch_time_passes<T>(b, 3, &ms)) != FDTD_OK) return st;
  b->tail = ms < best;
  CUDA_TRY(cudaGetLastError());
  return batch_upload_items<T>(b);
}

template <typename T>
static fdtd_status batch_step(fdtd_batch* b, int nsteps, cudaStream_t st) {
  const int every = b->dft_every > 0 ? b->dft_every : 1;
  const int G = every * kSampleBlock;
  int done = 0;
  while (done < nsteps) {
    const bool aligned = b->direct && b->t % G == 0 && b->host_nsamp == 0 && nsteps - done >= G;
    if (aligned) {
      if (!b->graph) {
        if (!b->cap) CUDA_TRY(cudaStreamCreateWithFlags(&b->cap, cudaStreamNonBlocking));
        cudaGraph_t g;
        const int t_save = b->t, n_save = b->host_nsamp;
        const long long k_save = b->kernels;
        CUDA_TRY(cudaStreamBeginCapture(b->cap, cudaStreamCaptureModeThreadLocal));
        for (int q = 0; q < G; q++) batch_enqueue_step<T>(b, b->cap);
        CUDA_TRY(cudaStreamEndCapture(b->cap, &g));
        b->graph_kernels = b->kernels - k_save;
        b->kernels = k_save;
        b->t = t_save;
        b->host_nsamp = n_save;
        cudaError_t e = cudaGraphInstantiate(&b->graph, g, 0);
        cudaGraphDestroy(g);
        CUDA_TRY(e);
      }
      CUDA_TRY(cudaGraphLaunch(b->graph, st));
      b->kernels += b->graph_kernels;
      b->graph_launches++;
      b->t += G;
      done += G;
    } else {
      batch_enqueue_step<T>(b, st);
      done++;
    }
  }
  // the members' host mirrors follow the batch clock
  for (auto& s : b->sims) {
    if (b->direct) {
      s->t = b->t;
      s->host_nsamp = b->host_nsamp;
    }
    s->steps_done += nsteps;
  }
  CUDA_TRY(cudaGetLastError());
  return FDTD_OK;
}

static fdtd_status batch_create_impl(const fdtd_params* ps, int n, int device, fdtd_batch** out) {
  if (!ps || !out || n <= 0) return fail(FDTD_ERR_INVALID, "bad argument");
  auto b = std::make_unique<fdtd_batch>();
  b->device = device;
  CUDA_TRY(cudaSetDevice(device));
  for (int i = 0; i < n; i++)
    if (ps[i].periodic_xy) return fail(FDTD_ERR_UNSUPPORTED, "periodic_xy simulations do not batch (member " + std::to_string(i) + ")");
  for (int i = 0; i < n; i++) {
    fdtd_sim* s = nullptr;
    const fdtd_status st = create_impl(&ps[i], device, &s, /*member*/ true);
    if (st != FDTD_OK) return fail(st, "batch member " + std::to_string(i) + ": " + g_err);
    b->sims.emplace_back(s);
    if (i == 0) {
      b->fp64 = s->fp64;
      b->hydro = s->su.hydro;
      b->dft_every = s->line.dft_every;
      b->tend = s->su.p.Tend;
    } else if (s->fp64 != b->fp64 || s->su.hydro != b->hydro || s->line.dft_every != b->dft_every ||
               s->su.p.Tend != b->tend) {
      return fail(FDTD_ERR_INVALID, "batch members must share precision, hydrodynamic model, "
                                    "DFT sampling period and Tend (member " + std::to_string(i) + ")");
    }
  }
  fdtd_status st = b->fp64 ? batch_build<double>(b.get()) : batch_build<float>(b.get());
  if (st != FDTD_OK) return st;
  st = b->fp64 ? batch_tune<double>(b.get()) : batch_tune<float>(b.get());
  if (st != FDTD_OK) return st;
  CUDA_TRY(cudaDeviceSynchronize());
  *out = b.release();
  return FDTD_OK;
}

extern "C" fdtd_status fdtd_batch_create(const fdtd_params* ps, int n, int device, fdtd_batch** out) {
  try {
    return batch_create_impl(ps, n, device, out);
  } catch (const std::bad_alloc&) {
    return fail(FDTD_ERR_ALLOC, "host allocation failed");
  }
}

extern "C" fdtd_status fdtd_batch_step(fdtd_batch* b, int nsteps, void* stream) {
  if (!b || nsteps < 0) return fail(FDTD_ERR_INVALID, "bad argument");
  CUDA_TRY(cudaSetDevice(b->device));
  return b->fp64 ? batch_step<double>(b, nsteps, as_stream(stream)) : batch_step<float>(b, nsteps, as_stream(stream));
}

extern "C" fdtd_status fdtd_batch_run(fdtd_batch* b, void* stream) {
  if (!b) return fail(FDTD_ERR_INVALID, "null argument");
  const int left = b->tend + 1 - b->t;
  if (left <= 0) return FDTD_OK;
  return fdtd_batch_step(b, left, stream);
}

extern "C" fdtd_status fdtd_batch_sim(fdtd_batch* b, int idx, fdtd_sim** out) {
  if (!b || !out || idx < 0 || idx >= (int)b->sims.size()) return fail(FDTD_ERR_INVALID, "bad argument");
  *out = b->sims[idx].get();
  return FDTD_OK;
}

extern "C" fdtd_status fdtd_batch_spectra(fdtd_batch* b, int idx, double* out19) {
  if (!b || !out19 || idx < 0 || idx >= (int)b->sims.size()) return fail(FDTD_ERR_INVALID, "bad argument");
  return fdtd_spectral_finalize(b->sims[idx].get(), out19);
}

extern "C" fdtd_status fdtd_batch_get_stats(const fdtd_batch* b, long long* kernels, long long* graph_launches) {
  if (!b) return fail(FDTD_ERR_INVALID, "null argument");
  if (kernels) *kernels = b->kernels;
  if (graph_launches) *graph_launches = b->graph_launches;
  return FDTD_OK;
}

extern "C" fdtd_status fdtd_batch_get_tuning(const fdtd_batch* b, fdtd_batch_tuning* out) {
  if (!b || !out) return fail(FDTD_ERR_INVALID, "null argument");
  std::memset(out, 0, sizeof(*out));
  out->tuned = b->tuned ? 1 : 0;
  out->nbuckets = b->nbuckets;
  for (int q = 0; q < b->nbuckets; q++) {
    out->edge_lo[q] = b->bucket_lo[q];
    out->edge_hi[q] = q + 1 < b->nbuckets ? b->bucket_lo[q + 1] - 1 : INT_MAX;
    out->members[q] = b->bucket_members[q];
    out->kchunk[q] = batch_kchunk(b->bucket_kz[q]);
    out->bucket_ms[q] = b->bucket_ms[q];
  }
  out->tile_x = 32;
  out->tile_y = b->fp64 ? Vec<double>::N : Vec<float>::N;
  for (int p = 0; p < 2; p++)
    for (int e = 0; e < 2; e++) {
      out->minb[p][e] = 2;
      out->stages[p][e] = b->ring ? kFlatRing : 1;
    }
  return FDTD_OK;
}

extern "C" fdtd_status fdtd_batch_destroy(fdtd_batch* b) {
  if (!b) return FDTD_OK;
  cudaSetDevice(b->device);
  cudaDeviceSynchronize();
  delete b;
  return FDTD_OK;
}
