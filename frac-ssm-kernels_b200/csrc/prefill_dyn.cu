// dyn[rows, N] = x[rows, K] W[N, K]^T in bf16 with float32 accumulation, N <= 192: the dynamic projection of a mixer
// (three values a head) next to its convolution, which reads the same x (frac_ssm/models/modeling_frac.py, FracMixer:
// dyn_proj).
//
// Bound by the bytes of x when there are many rows, by the latency of one pass over K when there are few: 128 rows are
// one tensor-core tile, so 4000 rows are 32 blocks, and a block that walks all of K alone waits for one load after the
// other.  K is therefore cut among the blocks of a cluster (up to 8); the partial sums go to the block that owns their
// rows through the cluster's shared memory and are added in the order of the blocks (no atomics: the same bits each
// time).  Tiles arrive by TMA: rows beyond the last one, weight rows beyond N and columns beyond K read as zero, so no
// operand has to be padded.
//
// The grid lets the convolution start at once, which needs nothing of it; the convolution's first block waits for it, so
// that what follows the convolution follows both.  us for K = 1536, the convolution alone / with the library's product
// behind it / with this kernel beside it:
//   rows            5                 397                4000                16000               65536
//   36 columns   3.0 / 12.7 / 4.9   4.2 / 16.5 / 6.5   11.3 / 28.9 / 12.5   36.3 / 56.6 / 38.1   127 / 204 / 164
//   72 columns   3.1 /  7.1 / 5.4   4.2 /  8.3 / 7.3   11.2 / 16.2 / 12.6   36.3 / 44.3 / 38.8   126 / 178 / 165
// (The library takes an old kernel where N is no multiple of 8: 17 us for 4000 rows and 36 columns, 4.6 for 72.)
#include <mutex>

#include "common.cuh"
#include "prefill_dyn.cuh"
#include "tmap.cuh"
#include "umma.cuh"

namespace fracssm {
namespace {

constexpr int kDynRows = 128;        // rows of a tile: the tensor-core instruction's M
constexpr int kDynK = 64;            // columns of K a step: one 128-byte row of the operand layout
constexpr int kDynThreads = 128;
constexpr int kDynMaxSplit = 8;
constexpr int kDynMaxStages = 8;
constexpr size_t kDynMaxSmem = 224 * 1024;
constexpr int64_t kDynFewBlocks = 64;

struct DynArgs {
  __nv_bfloat16 *out;
  int64_t rows;
  int N, n16, cols;    // columns; rounded up to 16; of tensor memory (a power of two)
  int steps, split, stages;
  uint64_t wait_ns;
  int withhold;        // self-test: the first block of a cluster leaves out its last tile of x
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// the address of `addr` of this block in block `rank` of the cluster
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, int rank) {
  uint32_t there;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(addr), "r"(rank));
  return there;
}
__device__ __forceinline__ void st_peer(uint32_t addr, float x, float y, float z, float w) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

template <int SPLIT>
__global__ void __launch_bounds__(kDynThreads)
prefill_dyn_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const DynArgs a) {
  extern __shared__ uint8_t raw_smem[];
  __shared__ uint64_t full[kDynMaxStages], done[kDynMaxStages];
  __shared__ uint32_t tmem;
  __shared__ int failed;
  const int warp = threadIdx.x >> 5;
  // (the same offset in every block of the cluster)
  uint8_t *ring = raw_smem + ((1024u - (umma::smem_u32(raw_smem) & 1023u)) & 1023u);
  const uint32_t a_bytes = kDynRows * 128, stage_bytes = a_bytes + (uint32_t)a.n16 * 128;
  const int rank = (int)(blockIdx.x % SPLIT);
  const int64_t row0 = (int64_t)(blockIdx.x / SPLIT) * kDynRows;
  const int k0 = a.steps * rank / SPLIT, n_steps = a.steps * (rank + 1) / SPLIT - k0;   // at least one

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    umma::prefetch_tmap(&x_map);
    umma::prefetch_tmap(&w_map);
    failed = 0;
    for (int s = 0; s < a.stages; ++s) {
      umma::mbar_init(&full[s], 1);
      umma::mbar_init(&done[s], 1);
    }
    umma::fence_mbar_init();
  }
  // Nobody who holds tensor memory waits for a block that may yet want some (another stream's kernel may hold it there,
  // and wait in turn): a block says that it has started before it asks for its own, and gives it back before it waits for
  // the others' sums.
  if (SPLIT > 1) cluster_arrive();
  if (warp == 1) umma::tmem_alloc(&tmem, (uint32_t)a.cols);
  umma::tc_fence_before();
  __syncthreads();
  umma::tc_fence_after();

  // One thread loads, one of another warp multiplies.
  if (warp == 0 && umma::elect_one()) {
    uint32_t s = 0, phase = 0;
    bool late = false;
#pragma unroll 1
    for (int k = 0; k < n_steps; ++k) {
      if (k >= a.stages && !umma::mbar_wait_parked(&done[s], phase ^ 1, a.wait_ns)) { late = true; break; }
      uint8_t *stage = ring + s * stage_bytes;
      umma::mbar_expect_tx(&full[s], stage_bytes);
      if (!(a.withhold && rank == 0 && k == n_steps - 1)) umma::tma_load_3d(stage, &x_map, &full[s], (k0 + k) * kDynK, (int)row0, 0);
      umma::tma_load_3d(stage + a_bytes, &w_map, &full[s], (k0 + k) * kDynK, 0, 0);
      if (++s == (uint32_t)a.stages) {
        s = 0;
        phase ^= 1;
      }
    }
    if (late) failed = 1;
  }
  if (warp == 2 && umma::elect_one()) {
    const uint32_t idesc = umma::make_idesc(kDynRows, a.n16, false, false);
    const uint64_t d0 = umma::make_sdesc(umma::smem_u32(ring), 16, 1024);   // (addresses count in units of 16 bytes)
    uint32_t s = 0, phase = 0, last = 0, last_phase = 0;
    bool late = false;
#pragma unroll 1
    for (int k = 0; k < n_steps; ++k) {
      // (after a wait that ran out the others are still made: a load that is on its way lands before the block ends)
      if (!umma::mbar_wait_parked(&full[s], phase, a.wait_ns)) late = true;
      umma::tc_fence_after();
      const uint64_t da = d0 + (s * stage_bytes >> 4), db = da + (a_bytes >> 4);
#pragma unroll
      for (int q = 0; q < kDynK / 16; ++q) umma::mma_ss(tmem, da + q * 2, db + q * 2, idesc, (k | q) != 0);
      umma::mma_commit(&done[s]);
      last = s;
      last_phase = phase;
      if (++s == (uint32_t)a.stages) {
        s = 0;
        phase ^= 1;
      }
    }
    // the last commit follows all products
    if (!umma::mbar_wait_parked(&done[last], last_phase, a.wait_ns)) late = true;
    if (late) failed = 1;
  }
  __syncthreads();
  umma::tc_fence_after();

  // Each row's sums go to the block that owns the row, into a slot behind its ring for each block they come from.  (A
  // block alone has its slots in the ring.)
  if (SPLIT > 1) cluster_wait();      // all blocks have started
  constexpr int kPer = kDynRows / SPLIT;
  const int pitch = a.n16 + 4;      // (16-byte stores of eight rows fall into different banks)
  const float *part = reinterpret_cast<const float *>(ring + (SPLIT > 1 ? (uint32_t)a.stages * stage_bytes : 0u));
  const uint32_t slot = umma::smem_u32(part) + (uint32_t)((rank * kPer + (int)threadIdx.x % kPer) * pitch) * 4u;
  const uint32_t to = peer_addr(slot, (int)threadIdx.x / kPer);
  const bool bad = failed != 0, wanted = row0 + (int)threadIdx.x < a.rows;
  for (int c = 0; c < a.n16; c += 16) {
    float v[16];
    umma::tmem_ld16(tmem + ((uint32_t)warp << 21) + (uint32_t)c, v);
    umma::tmem_ld_wait();
    if (bad) {
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = __int_as_float(0x7fc00000);
    }
#pragma unroll
    for (int i = 0; i < 16; i += 4)
      if (wanted) st_peer(to + (uint32_t)(c + i) * 4u, v[i], v[i + 1], v[i + 2], v[i + 3]);
  }
  umma::tc_fence_before();
  __syncthreads();
  if (warp == 1) umma::tmem_dealloc(tmem, (uint32_t)a.cols);
  if (SPLIT > 1) {
    cluster_arrive();
    cluster_wait();
  }

  // this block's rows: a warp four rows at a time, a lane a pair of columns
  const int64_t first = row0 + rank * kPer, left = a.rows - first;
  const int here = left <= 0 ? 0 : left < kPer ? (int)left : kPer, lane = (int)threadIdx.x & 31;
  __nv_bfloat16 *out = a.out + first * a.N;
  constexpr int kRun = 4;
  for (int r0 = warp * kRun; r0 < here; r0 += kRun * kDynThreads / 32) {
    for (int c = 2 * lane; c < a.N; c += 64) {
      float2 sum[kRun];
#pragma unroll
      for (int j = 0; j < kRun; ++j) sum[j] = *reinterpret_cast<const float2 *>(part + (r0 + j) * pitch + c);
#pragma unroll
      for (int q = 1; q < SPLIT; ++q) {
#pragma unroll
        for (int j = 0; j < kRun; ++j) {
          const float2 v = *reinterpret_cast<const float2 *>(part + (q * kPer + r0 + j) * pitch + c);
          sum[j].x += v.x;
          sum[j].y += v.y;
        }
      }
#pragma unroll
      for (int j = 0; j < kRun; ++j) {
        if (r0 + j >= here) break;
        __nv_bfloat16 *o = out + (r0 + j) * a.N + c;
        if ((a.N & 1) == 0) {      // (c + 1 < N, and o lies on 4 bytes)
          *reinterpret_cast<__nv_bfloat162 *>(o) = __floats2bfloat162_rn(sum[j].x, sum[j].y);
        } else {
          o[0] = __float2bfloat16_rn(sum[j].x);
          if (c + 1 < a.N) o[1] = __float2bfloat16_rn(sum[j].y);
        }
      }
    }
  }
}

}  // namespace

int prefill_dyn_launch(const void *x, int64_t x_sl, const void *w, void *out, int64_t rows, int64_t K, int64_t N,
                       cudaStream_t st, uint64_t wait_ns, bool withhold) {
  if (!x || !w || !out) return fail(FRACSSM_ERR_ARG, "prefill_dyn: null pointer");
  if (rows <= 0 || K <= 0 || N <= 0 || x_sl < K) return fail(FRACSSM_ERR_ARG, "prefill_dyn: bad sizes");
  if (N > 192 || K % 8 != 0 || x_sl % 8 != 0 || rows > (1ll << 30) || K > (1ll << 30) ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) != 0 ||
      (reinterpret_cast<uintptr_t>(out) & 3) != 0)
    return fail(FRACSSM_ERR_UNSUPPORTED, "prefill_dyn: at most 192 columns, rows and weights on 16 bytes");
  // per device, once: its number of SMs, and the large dynamic shared memory
  using Kernel = void (*)(const CUtensorMap, const CUtensorMap, const DynArgs);
  static constexpr Kernel kernels[4] = {prefill_dyn_kernel<1>, prefill_dyn_kernel<2>, prefill_dyn_kernel<4>,
                                        prefill_dyn_kernel<8>};
  static std::mutex mu;
  static int count[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev >= 64) return fail(FRACSSM_ERR_CUDA, "prefill_dyn: %s", cudaGetErrorString(e));
  int sms = 0;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!count[dev]) {
      int n = 0;
      e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
      if (e == cudaSuccess) {
        for (auto kernel : kernels)
          if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDynMaxSmem);
      }
      if (e != cudaSuccess) return fail(FRACSSM_ERR_CUDA, "prefill_dyn: %s", cudaGetErrorString(e));
      count[dev] = n;
    }
    sms = count[dev];
  }
  DynArgs a{};
  a.out = reinterpret_cast<__nv_bfloat16 *>(out);
  a.rows = rows;
  a.N = (int)N;
  a.n16 = (int)ceil_div(N, 16) * 16;
  a.cols = 32;
  while (a.cols < a.n16) a.cols *= 2;
  a.steps = (int)ceil_div(K, kDynK);
  a.wait_ns = wait_ns;
  a.withhold = withhold;
  // K is cut as long as the grid has one block per SM and a block two steps.  The kernel alone, us, 72 columns:
  //   blocks a tile        1      2      4      8
  //     397 rows         10.4    8.1    7.0    6.5
  //    4000 rows         10.5    8.2    8.1   10.2   (8: 256 blocks)
  //    9000 rows         10.7   10.0   11.1          (4: 284 blocks)
  //   16000 rows         10.9   12.6   19.7          (2: 250 blocks)
  const int64_t tiles = ceil_div(rows, kDynRows);
  a.split = 1;
  while (a.split < kDynMaxSplit && tiles * a.split * 2 <= sms && a.steps >= a.split * 4) a.split *= 2;
  const size_t stage = kDynRows * 128 + (size_t)a.n16 * 128, sums = (size_t)kDynRows * (a.n16 + 4) * 4;
  // As many stages as half an SM has room for, or the whole where blocks are few or that is less than two.  (128 blocks in
  // clusters of 8 find no place with an SM each: 2000 rows with the convolution 16.4 us instead of 9.9.  128 blocks in
  // clusters of 4 do, and are 0.5 us faster alone, but the convolution beside them is slower: 4 x 1000 tokens through 24
  // layers 3152 us instead of 3090.)  1 KB aligns the ring.
  const int most = (int)ceil_div(a.steps, a.split);
  const size_t behind = a.split > 1 ? sums : 0;
  auto fit = [&](size_t room) { return room < 1024 + behind ? 0 : (int)((room - 1024 - behind) / stage); };
  a.stages = tiles * a.split <= kDynFewBlocks ? 0 : fit(kDynMaxSmem / 2);
  if (a.stages < 2) a.stages = fit(kDynMaxSmem);
  if (a.stages > kDynMaxStages) a.stages = kDynMaxStages;
  if (a.stages > most) a.stages = most;
  size_t smem = a.stages * stage + behind;
  smem = 1024 + (smem > sums ? smem : sums);

  CUtensorMap x_map, w_map;
  int rc = make_tmap_bf16_rows(&x_map, x, (uint64_t)K, (uint64_t)rows, (uint64_t)x_sl, kDynK, kDynRows);
  if (!rc) rc = make_tmap_bf16_rows(&w_map, w, (uint64_t)K, (uint64_t)N, (uint64_t)K, kDynK, (uint32_t)a.n16);
  if (rc) return rc;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(tiles * a.split));
  cfg.blockDim = dim3(kDynThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)a.split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, kernels[a.split == 1 ? 0 : a.split == 2 ? 1 : a.split == 4 ? 2 : 3], x_map, w_map, a);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(FRACSSM_ERR_CUDA, "prefill_dyn: %s", cudaGetErrorString(e));
  }
  return FRACSSM_OK;
}

}  // namespace fracssm
