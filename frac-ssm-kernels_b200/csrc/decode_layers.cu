// One decode token through all layers of the model, bfloat16, up to 64 sequences.  A layer has four stages:
//
//   kIn    in_proj of the normalised hidden state -> x | gate; the rows of x also take the causal convolution step + SiLU (a
//          channel needs its own history only)
//   kProj  rw_proj of x_conv and dyn_proj of x, whose rows also take the nonlinearities of the time step, alpha and lambda
//   kMix   the scan parameters of a (sequence, head), its state one token further, readout, D skip, gate
//   kOut   out_proj of the normalised result -> + hidden state
// and decode_first_kernel, once, does for the embedding what kOut does for the next layer's norm.
//
// What bounds a step: reading the weights (27 MB a layer at hidden 768, 128 modes) and, from some 16 sequences
// on, the float32 state in and out; at few sequences the length of the chain of stages.  Hence
//   * elementwise work sits in the epilogue of the product that writes its rows.  A norm is split: whoever writes
//     the row also writes it times the norm's weight and the sums of squares of its part of the row, and the product
//     that reads it scales its results by 1 / rms, so no block has to see a whole row before it can start.  What
//     passes between the stages without going through a product (hidden state, gate, readout) stays float32;
//   * the products stream the weights once, straight into the fragments of mma.sync (16 weight rows x 16 of the
//     contraction x 8 sequences): with at most 64 sequences they are far below the tensor-core ridge, and a lane
//     reads 8 consecutive weights of a row because the contraction order is free as long as both operands share
//     it.  A team of 8 warps splits the contraction of a 16-row tile, so even 768 output rows keep 48 teams busy;
//   * what a stage needs and no stage of this call writes (weights, the old state and convolution history, parameters) is
//     requested before the stage in front of it is waited for.
//
// Two forms of the same code (struct Step), with the same results:
//   * a kernel a stage, launched with programmatic stream serialisation: 97 launches at 24 layers;
//   * one kernel (a launch per 32 layers) whose blocks, at most one per SM, meet at a barrier between the stages.  The host makes
//     the 97 launches in more time than the device takes for them at few sequences.  A stage takes 2 to 5 us here, of which
//     the barrier is 1.3; what bounds it is the number of instructions a warp gets through with cold instruction
//     caches, since every stage passes through its code once per layer.  So it is ONE loop over the stages with one copy of each
//     piece of code, little of it unrolled (with the products and their requests inlined for each stage 117 KB of code and
//     0.86 ms at one sequence; 68 KB and 0.50 ms as here).
//     Nothing makes all blocks run at the same time: kernels of other streams may hold SMs, for long, and may wait for this very
//     step.  So the blocks that have started make up a list and share the work among themselves (see join); a block that comes
//     later finds the list closed and leaves.  Nobody waits for a block that has not started.
// Where either is used: see one_kernel_pays.
#include <mutex>

#include "common.cuh"
#include "scan_tile.cuh"

namespace fracssm {
namespace {

constexpr int kWarps = 8, kTeam = 32 * kWarps;   // warps that share a tile's contraction, and their threads
constexpr int kTileRows = 16, kMaxSeq = 64;
constexpr int kRedStride = 20;       // floats per sequence in the exchange buffer: 16 rows, bank-conflict free
constexpr int kPassTiles = 2;        // groups of 8 sequences exchanged at a time
constexpr int kSums = 6;             // partial sums of squares a thread reads at a time
constexpr uint32_t kMostSmem = 227 * 1024;

constexpr int kPre = 6;              // 32-wide steps of the contraction a warp holds weights for
constexpr int kMaxHidden = 8192;     // longest hidden state
enum { kIn = 0, kProj = 1, kMix = 2, kOut = 3 };   // the stages of a layer

__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ uint4 ldg_weights(const void *p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float bf(uint32_t lo16) { return __uint_as_float(lo16 << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
__device__ __forceinline__ float sum_warp(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float sigmoid_(float x) { return 1.f / (1.f + __expf(-x)); }

// a parameter's bits, and its value: the second waits for the first, so it is taken where the value is needed
__device__ __forceinline__ uint32_t ld_bits(const void *p, int64_t i, int dt) {
  return dt == FRACSSM_F32 ? __ldg(reinterpret_cast<const uint32_t *>(p) + i)
                           : (uint32_t)__ldg(reinterpret_cast<const unsigned short *>(p) + i);
}
__device__ __forceinline__ float as_f32(uint32_t bits, int dt) { return __uint_as_float(dt == FRACSSM_F32 ? bits : bits << 16); }

// 16 bytes to shared memory, zeros where `on` is false
__device__ __forceinline__ void copy_async16(uint32_t dst, const void *src, bool on) {
  const int n = on ? 16 : 0;   // (0: nothing is read)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

__host__ __device__ inline int tiles_of(int n) { return (n + kTileRows - 1) / kTileRows; }
// bytes from row to row of the activations in shared memory: 64 mod 128, so that a quarter-warp's 16-byte reads cover all banks
__host__ __device__ inline uint32_t act_stride(int K) { return K * 2 + ((K * 2) % 128 == 0 ? 64 : 128); }

// Sum of a row's partial sums of squares over the 16 threads that share it (lane e of them); none where `on` is false.  All of
// a thread's reads are on their way together: one after the other they were up to six waits for L2 behind every norm.
__device__ __forceinline__ float row_sum(const float *ss, int n, int e, bool on) {
  const int mine = on ? n : 0;
  float t = 0.f;
#pragma unroll 1
  for (int i0 = e; i0 < mine; i0 += 16 * kSums) {
    float y[kSums];
#pragma unroll
    for (int i = 0; i < kSums; ++i) y[i] = i0 + 16 * i < mine ? __ldcg(ss + i0 + 16 * i) : 0.f;
#pragma unroll
    for (int i = 0; i < kSums; ++i) t += y[i];
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// the layers' pointer and number tables of fracssm_decode_layers
enum LayerPtr { kNormW, kInW, kConvW, kConvB, kDynW, kDynB, kRwW, kDtBias, kReadLogit, kWriteLogit, kLogTau, kD,
                kOutNormW, kOutW, kOldState, kOldConv, kNewState, kNewConv, kF32Mask, kLayerPtrs };
enum LayerNum { kEpsIn, kEpsOut, kReadTemp, kDtMin, kDtMax, kAMin, kAMax, kLMin, kLMax, kGateBias, kLayerNums };

// Where a thread stands: a block is `teams` teams of 8 warps, each of which works on tiles or heads of its own; the blocks that
// share the work are numbered 0 .. blocks - 1.
struct Place {
  int team, teams, tid, lane, w;   // tid, w: inside the team
  int block, blocks;
  __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(kTeam) : "memory"); }
};

constexpr int kMixPre = 8;             // float4 pieces of the old state a thread requests ahead
constexpr int kMixItems = 4;           // items whose parameters a team's warps work out side by side
struct MixShape {                      // what does not change from layer to layer, worked out on the host
  int cols, quads, groups, fold;       // columns of an item, float4 pieces of them, modes worked on side by side
  int items, batch, parts;             // parts: sums of squares an item leaves
};

// What the blocks of the one-kernel form count together.
struct Meeting {
  unsigned arrived;    // at the barriers, over the whole launch
  unsigned started;    // blocks that asked to be on the list; kClosed once it is closed
  unsigned members;    // blocks on the closed list, 0 before
  unsigned left;       // blocks at their end
  unsigned failed;     // set once a wait has run out, for the whole call
  unsigned spare[3];
};
constexpr size_t kPerLaunch = 16;      // bytes of it that every launch starts with as zeros: all but `failed`
constexpr unsigned kClosed = 0x80000000u;

// The embedding times the first norm's weight, and its sums of squares (one part per row); clears what the one-kernel form's
// blocks count.
__global__ void __launch_bounds__(kTeam)
decode_first_kernel(const __nv_bfloat16 *h, const void *w, int w_dt, float *h_f32, __nv_bfloat16 *h_w, float *ss, int d,
                    Meeting *meeting) {
  __shared__ float red[kWarps];
  const int64_t b = blockIdx.x;
  grid_dep_launch();
  if (b == 0 && threadIdx.x == 0) *meeting = Meeting{};
  float sq = 0.f;
  for (int i = threadIdx.x; i < d; i += kTeam) {
    const float v = __bfloat162float(h[b * d + i]);
    h_f32[b * d + i] = v;
    h_w[b * d + i] = __float2bfloat16_rn(v * ld_f32(w, i, w_dt));
    sq = fmaf(v, v, sq);
  }
  sq = sum_warp(sq);
  if (threadIdx.x % 32 == 0) red[threadIdx.x / 32] = sq;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) t += red[i];
    ss[b] = t;
  }
}

constexpr int kTabLayers = 32;       // layers of one launch of the one-kernel form
struct LayerTab {
  uint64_t p[kLayerPtrs];
  float f[kLayerNums];
};
// LAYERS layers of the model; their table is a kernel argument (a graph keeps it)
template <int LAYERS>
struct StepArgs {
  LayerTab tab[LAYERS];
  const void *after_w;               // the norm weight behind the last of them, or null: the model's last layer
  int after_dt;
  int layers, first;                 // first: index of tab[0] in the model
  int B, d, H, R, M, splits, l2_state, blocks2;   // blocks2: blocks that take dyn_proj's tiles (the kernel of a stage)
  MixShape mix;
  __nv_bfloat16 *x, *x_conv, *vals, *hid_w, *out;
  float *gate, *rw, *dyn, *ss, *hid[2], *hid_ss;
  Meeting *meeting;
  unsigned long long work_ns;        // what the launch takes one block per SM, about
  unsigned long long wait_ns;        // limit of a wait for the other blocks
  int lost;                          // self-test: at this barrier, counted from 1, block 0 waits for the next one's arrivals too
  uint32_t act_bytes, red_bytes, mix_bytes;
};

// Teams of a block, and with them registers a thread: up to 8 sequences 255, beyond 128.  (24 layers of hidden 768 at one
// sequence: 0.51 ms with one team, 0.54 with two, 0.63 with three, which spill; at 32 sequences 1.00 with one, 0.87 with two.)
template <int NT>
constexpr int max_teams() { return NT == 1 ? 1 : 2; }

// A team's work on the stages, NT groups of 8 sequences.
template <int NT, int LAYERS>
struct Step {
  static constexpr int kPasses = (NT + kPassTiles - 1) / kPassTiles;
  static constexpr int kExtra = 3 + 3 * kPasses > 8 ? 3 + 3 * kPasses : 8;

  const StepArgs<LAYERS> &a;
  Place at;
  uint8_t *smem;
  // What a team holds of a stage before it begins, requested before the barrier in front of it: everything that the stage
  // before does not write.  A product's: the fragments of the first tile's weights [2 i], [2 i + 1], and what the
  // epilogue needs; the mix: pieces of the first item's old state, and parameters.
  uint4 hold[2 * kPre];
  uint32_t extra[kExtra];
  // the product of a stage as this team sees it
  const __nv_bfloat16 *W, *act;
  int N, K, tile0, tile_step, tiles, k_lo, k_hi;
  bool second, any;   // second: dyn_proj's tiles; any: a team of this block has a tile
  int blocks2;        // blocks that take dyn_proj's tiles

  __device__ __forceinline__ const __nv_bfloat16 *bfp(int l, int i) const {
    return reinterpret_cast<const __nv_bfloat16 *>(a.tab[l].p[i]);
  }
  __device__ __forceinline__ const void *raw(int l, int i) const { return reinterpret_cast<const void *>(a.tab[l].p[i]); }
  __device__ __forceinline__ int dt(int l, int i) const {
    return (static_cast<uint32_t>(a.tab[l].p[kF32Mask]) >> i) & 1 ? FRACSSM_F32 : FRACSSM_BF16;
  }

  // ---------------------------------------------------------------------------------------------- the products
  // (`rest`, a block alone: rw_proj's tiles, after dyn_proj's)
  __device__ __forceinline__ void product(int l, int kind, int team, bool rest = false) {
    const int di = a.H * a.R;
    int blk = at.block, blocks = at.blocks;
    second = kind == kProj && blk < blocks2 && !rest;
    if (kind == kIn) {
      W = bfp(l, kInW); act = a.hid_w; N = 2 * di; K = a.d;
    } else if (kind == kOut) {
      W = bfp(l, kOutW); act = a.vals; N = a.d; K = di;
    } else {
      K = di;
      if (second) {
        W = bfp(l, kDynW); act = a.x; N = 3 * a.H;
        blocks = blocks2;
      } else {
        W = bfp(l, kRwW); act = a.x_conv; N = 2 * a.H * a.M;
        if (!rest) { blk -= blocks2; blocks -= blocks2; }
      }
    }
    tiles = tiles_of(N);
    tile0 = blk + team * blocks;
    tile_step = blocks * at.teams;
    any = blk < tiles;
    const int steps = K / 32, share = (steps + kWarps - 1) / kWarps;
    k_lo = min(at.w * share, steps); k_hi = min(k_lo + share, steps);
  }
  __device__ __forceinline__ void request(int tile, int k0) {
    const int g = at.lane >> 2, tig = at.lane & 3;
    const int r0 = min(tile * kTileRows + g, N - 1), r1 = min(tile * kTileRows + g + 8, N - 1);
    const __nv_bfloat16 *p0 = W + (int64_t)r0 * K + 8 * tig, *p1 = W + (int64_t)r1 * K + 8 * tig;
#pragma unroll
    for (int i = 0; i < kPre; ++i) {
      if (k0 + i < k_hi) {
        hold[2 * i] = ldg_weights(p0 + (k0 + i) * 32);
        hold[2 * i + 1] = ldg_weights(p1 + (k0 + i) * 32);
      }
    }
  }
  // what the epilogue of a tile needs, for all of this thread's sequences.  kIn: the channel's convolution weights (0, 1) and
  // bias (2) and history; kOut: the next norm's weight (0) and the hidden state (written four barriers ago)
  __device__ __forceinline__ void epilogue_inputs(int l, int kind, int tile) {
    const int n = tile * kTileRows + (at.tid & 15), e_seq = at.tid >> 4, di = a.H * a.R;
    if (kind == kIn) {
      if (n >= di) return;
      const uint2 cw = __ldg(reinterpret_cast<const uint2 *>(bfp(l, kConvW) + (int64_t)n * 4));
      extra[0] = cw.x; extra[1] = cw.y;
      extra[2] = a.tab[l].p[kConvB] ? ld_bits(raw(l, kConvB), n, FRACSSM_BF16) : 0u;
#pragma unroll
      for (int p = 0; p < kPasses; ++p) {
        const int b = 8 * kPassTiles * p + e_seq;
        const bool on = a.tab[l].p[kOldConv] && b < a.B;
#pragma unroll
        for (int i = 0; i < 3; ++i)
          extra[3 + 3 * p + i] = on ? ld_bits(raw(l, kOldConv), ((int64_t)b * di + n) * 3 + i, FRACSSM_BF16) : 0u;
      }
    } else if (kind == kProj) {
      if (!second || n >= N) return;   // dyn_proj's bias (0) and the heads' dt_bias (1)
      extra[0] = a.tab[l].p[kDynB] ? ld_bits(raw(l, kDynB), n, FRACSSM_BF16) : 0u;
      extra[1] = n < a.H ? ld_bits(raw(l, kDtBias), n, dt(l, kDtBias)) : 0u;
    } else {
      const void *next_w = l + 1 < a.layers ? raw(l + 1, kNormW) : a.after_w;
      extra[0] = next_w && n < N ? ld_bits(next_w, n, l + 1 < a.layers ? dt(l + 1, kNormW) : a.after_dt) : 0u;
      const float *res = a.hid[(a.first + l) & 1];
#pragma unroll
      for (int p = 0; p < kPasses; ++p) {
        const int b = 8 * kPassTiles * p + e_seq;
        extra[3 + 3 * p] = b < a.B && n < N ? __float_as_uint(__ldcg(res + (int64_t)b * N + n)) : 0u;
      }
    }
  }
  // a team's tiles to L2, by one thread
  __device__ __forceinline__ void product_to_l2(int l, int kind, int team) {
    product(l, kind, team);
#pragma unroll 1
    for (int tile = tile0; tile < tiles; tile += tile_step)
      umma::prefetch_l2(W + (int64_t)tile * kTileRows * K, min(kTileRows, N - tile * kTileRows) * K * 2);
  }

  __device__ __forceinline__ void ahead_product(int l, int kind) {
    product(l, kind, at.team);
    if (tile0 >= tiles) return;
    request(tile0, k_lo);
    epilogue_inputs(l, kind, tile0);
  }
  __device__ __forceinline__ void ahead_epilogue(int l, int kind) {
    if (tile0 < tiles) epilogue_inputs(l, kind, tile0);
  }
  // (the fields that `product` set for the requests still hold)
  __device__ __forceinline__ void run_product(int l, int kind) {
    // act_smem: the activations of all teams (NT > 1); red: this team's exchange buffer
    float *red = reinterpret_cast<float *>(smem + a.act_bytes + at.team * a.red_bytes);
    const int g = at.lane >> 2, tig = at.lane & 3, e_row = at.tid & 15, e_seq = at.tid >> 4;
    const uint32_t stride = act_stride(K);   // 64 mod 128 bytes: a quarter-warp's 16-byte reads cover all banks
    // ---- activations (bf16, zeros beyond B).  Up to 8 sequences straight into the fragments; beyond, every tile reads
    // them again, so they go to shared memory once for all teams.
    if (NT > 1 && any) {
      const uint32_t act_s = (uint32_t)__cvta_generic_to_shared(smem);
      const int pieces = K / 8;
#pragma unroll 1
      for (int b = at.team * kWarps + at.w; b < 8 * NT; b += at.teams * kWarps) {
        const __nv_bfloat16 *src = act + (int64_t)min(b, a.B - 1) * K;
#pragma unroll 4
        for (int i = at.lane; i < pieces; i += 32) copy_async16(act_s + b * stride + i * 16, src + i * 8, b < a.B);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    }
    // (the activations' and the sums' reads are on their way together)
    uint4 xs[NT == 1 ? kPre : 1];
    auto activations = [&](int k0) {
      const __nv_bfloat16 *src = act + (int64_t)g * K + k0 * 32 + 8 * tig;
#pragma unroll
      for (int i = 0; i < kPre; ++i) {
        xs[i] = make_uint4(0, 0, 0, 0);
        if (k0 + i < k_hi && g < a.B) xs[i] = __ldcg(reinterpret_cast<const uint4 *>(src + i * 32));
      }
    };
    if constexpr (NT == 1) {
      if (any) activations(k_lo);
    }
    // 1 / rms of this thread's sequences: 16 threads share one
    float rs[kPasses];
    if (kind != kProj && any) {
      const float *ss = kind == kIn ? a.hid_ss : a.ss;
      const int nss = kind == kOut ? a.H * a.splits * a.mix.parts : a.first + l == 0 ? 1 : tiles_of(a.d);
      const float eps = a.tab[l].f[kind == kIn ? kEpsIn : kEpsOut];
#pragma unroll
      for (int p = 0; p < kPasses; ++p) {
        const int b = 8 * kPassTiles * p + e_seq;
        const float t = row_sum(ss + (int64_t)b * nss, nss, e_row, b < a.B);
        rs[p] = rsqrtf(t / (float)K + eps);
      }
    } else {
#pragma unroll
      for (int p = 0; p < kPasses; ++p) rs[p] = 1.f;
    }
    if (NT > 1 && any) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }

#pragma unroll 1
    for (int tile = tile0; tile < tiles; tile += tile_step) {
      float acc[NT][4];
#pragma unroll
      for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
#pragma unroll 1
      for (int k0 = k_lo; k0 < k_hi; k0 += kPre) {
        if (k0 != k_lo) request(tile, k0);
        if constexpr (NT == 1) {
          if (k0 != k_lo || (tile != tile0 && k_hi - k_lo > kPre)) activations(k0);
        }
#pragma unroll
        for (int i = 0; i < kPre; ++i) {
          if (k0 + i < k_hi) {
            const uint4 w0 = hold[2 * i], w1 = hold[2 * i + 1];
#pragma unroll
            for (int t = 0; t < NT; ++t) {
              const uint4 x = NT == 1 ? xs[NT == 1 ? i : 0]
                                      : *reinterpret_cast<const uint4 *>(smem + (8 * t + g) * stride + (k0 + i) * 64 + 16 * tig);
              mma_bf16(acc[t], w0.x, w1.x, w0.y, w1.y, x.x, x.y);
              mma_bf16(acc[t], w0.z, w1.z, w0.w, w1.w, x.z, x.w);
            }
          }
        }
      }
      if (tile + tile_step < tiles) request(tile + tile_step, k_lo);   // on their way during the epilogue
      if (tile != tile0) epilogue_inputs(l, kind, tile);
      // ---- the warps' shares of the contraction are added, a value per thread
      const int n = tile * kTileRows + e_row;
#pragma unroll
      for (int p = 0; p < NT; p += kPassTiles) {
#pragma unroll
        for (int t = p; t < p + kPassTiles && t < NT; ++t) {
          float *d = red + (at.w * 8 * kPassTiles + 8 * (t - p) + 2 * tig) * kRedStride + g;
          d[0] = acc[t][0];
          d[kRedStride] = acc[t][1];
          d[8] = acc[t][2];
          d[kRedStride + 8] = acc[t][3];
        }
        at.sync();
        const int b = 8 * p + e_seq, pass = p / kPassTiles;
        const bool on = e_seq < 8 * (NT - p) && b < a.B && n < N;
        float v = 0.f;
#pragma unroll
        for (int i = 0; i < kWarps; ++i) v += red[(i * 8 * kPassTiles + e_seq) * kRedStride + e_row];
        finish(l, kind, tile, n, b, on, v, rs[pass], extra[3 + 3 * pass], extra[4 + 3 * pass], extra[5 + 3 * pass]);
        at.sync();
      }
    }
  }
  // One result times rs (1 for kProj): sequence b, row n.  (Here and in the mix every fused multiply-add is written out: both
  // forms of the step are to round alike.)
  __device__ __forceinline__ void finish(int l, int kind, int tile, int n, int b, bool on, float v, float rs, uint32_t x0, uint32_t x1,
                                         uint32_t x2) {
    const int di = a.H * a.R;
    const uint32_t o = (uint32_t)b * N + n;
    if (kind == kIn) {
      if (on && n < di) {
        const __nv_bfloat16 xb = __float2bfloat16_rn(__fmul_rn(v, rs));
        float y = bf(extra[2]);
        y = fmaf(bf(extra[0]), bf(x0), y);
        y = fmaf(bf_hi(extra[0]), bf(x1), y);
        y = fmaf(bf(extra[1]), bf(x2), y);
        y = fmaf(bf_hi(extra[1]), __bfloat162float(xb), y);
        const uint32_t c = (uint32_t)b * di + n;
        a.x[c] = xb;
        a.x_conv[c] = __float2bfloat16_rn(y / (1.f + __expf(-y)));
        if (a.tab[l].p[kNewConv]) {
          unsigned short *q = reinterpret_cast<unsigned short *>(a.tab[l].p[kNewConv]) + c * 3;
          q[0] = (unsigned short)x1;
          q[1] = (unsigned short)x2;
          q[2] = __bfloat16_as_ushort(xb);
        }
      } else if (on) {
        a.gate[(uint32_t)b * di + n - di] = __fmul_rn(v, rs);
      }
    } else if (kind == kProj) {
      // dyn_proj's rows are the heads' time step, alpha and lambda before their nonlinearity, which is taken here (the
      // formulas of compute_params_kernel): a value per thread instead of one after the other in the mix
      if (on && second) {
        const float *f = a.tab[l].f;
        const float y = v + bf(extra[0]);
        float r;
        if (n < a.H) {
          const float d0 = y + as_f32(extra[1], dt(l, kDtBias));
          r = fminf(fmaxf(d0 > 20.f ? d0 : log1pf(expf(d0)), f[kDtMin]), f[kDtMax]);
        } else {
          const int lo = n < 2 * a.H ? kAMin : kLMin, hi = n < 2 * a.H ? kAMax : kLMax;
          r = fmaf(sigmoid_(y), f[hi] - f[lo], f[lo]);
        }
        a.dyn[o] = r;
      } else if (on) {
        a.rw[o] = v;
      }
    } else {
      // + hidden state; for the next layer's norm the row times its weight, and a sum of squares per tile
      const bool more = l + 1 < a.layers || a.after_w;
      float sq = 0.f;
      if (on) {
        const float hv = fmaf(v, rs, __uint_as_float(x0));
        if (more) {
          a.hid[(a.first + l + 1) & 1][o] = hv;
          a.hid_w[o] = __float2bfloat16_rn(hv * as_f32(extra[0], l + 1 < a.layers ? dt(l + 1, kNormW) : a.after_dt));
          sq = __fmul_rn(hv, hv);
        } else {
          a.out[o] = __float2bfloat16_rn(hv);
        }
      }
      if (more) {   // the tile's 16 rows of a sequence lie in 16 neighbouring lanes
#pragma unroll
        for (int i = 8; i > 0; i >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, i);
        if (on && (at.tid & 15) == 0) a.hid_ss[(uint32_t)b * tiles + tile] = sq;
      }
    }
  }

  // ------------------------------------------------------------------------------------------------- the mix
  // The scan parameters, state and readout of (sequence, head, share of the head's columns) items.  A team takes up to
  // four items at a time: first every pair of warps works out the parameters of one (the read and the write side, a
  // softmax within a warp, so that nothing waits for a block), then the team goes through their states.
  struct Item { int b, h, sp; };
  __device__ __forceinline__ Item item_at(int item) const {
    const int bh = a.splits == 1 ? item : item / a.splits, b = bh / a.H;
    return Item{b, bh - b * a.H, item - bh * a.splits};
  }
  __device__ __forceinline__ int64_t head_of(const Item &i) const { return (int64_t)i.b * a.H + i.h; }
  __device__ __forceinline__ void state_to_l2(int l, int team) const {
    const float *old = reinterpret_cast<const float *>(a.tab[l].p[kOldState]);
    if (!old || !a.l2_state) return;
#pragma unroll 1
    for (int item = at.block + team * at.blocks; item < a.mix.items; item += at.blocks * at.teams)
      if (item % a.splits == 0) umma::prefetch_l2(old + (int64_t)(item / a.splits) * a.M * a.R, a.M * a.R * 4);
  }
  __device__ __forceinline__ void request_state(int l, int q, int mg) {
    const int first = at.block + at.team * at.blocks;
    const float *old = reinterpret_cast<const float *>(a.tab[l].p[kOldState]);
    if (first >= a.mix.items) return;
    const bool have = old && mg < a.mix.groups;
    const Item i0 = item_at(first);
    old += head_of(i0) * a.M * a.R + i0.sp * a.mix.cols + 4 * q + mg * a.R;
    const int hop = a.mix.groups * a.R;
#pragma unroll
    for (int i = 0; i < kMixPre; ++i) {
      hold[i] = make_uint4(0, 0, 0, 0);
      if (have && mg + i * a.mix.groups < a.M) hold[i] = __ldcs(reinterpret_cast<const uint4 *>(old));
      old += hop;
    }
  }
  // What an item's modes have in shared memory: rho, kappa's weight (its factor 1 - rho is applied where the state is), c,
  // log_tau.  Beside it, requested or written before the barrier: log_tau, and the logits (extra 4 read, 5 write), D (6),
  // norm weight (7).
  __device__ __forceinline__ float4 *modes_of(int slot) const {
    return reinterpret_cast<float4 *>(smem + at.team * a.mix_bytes) + slot * a.M;
  }
  __device__ __forceinline__ void mix_inputs(int l) {
    const int first = at.block + at.team * at.blocks;
    if (first >= a.mix.items) return;
    const Item i0 = item_at(first);
    extra[4] = ld_bits(raw(l, kReadLogit), 0, dt(l, kReadLogit));
    extra[5] = ld_bits(raw(l, kWriteLogit), 0, dt(l, kWriteLogit));
    const int64_t c = (int64_t)i0.h * a.R + i0.sp * a.mix.cols + at.tid;
    if (at.tid < a.mix.cols) {
      extra[6] = ld_bits(raw(l, kD), c, dt(l, kD));
      extra[7] = ld_bits(raw(l, kOutNormW), c, dt(l, kOutNormW));
    }
#pragma unroll 1
    for (int m = at.tid; m < a.M; m += kTeam) {
      const float lt = as_f32(ld_bits(raw(l, kLogTau), m, dt(l, kLogTau)), dt(l, kLogTau));
      for (int slot = 0; slot < a.mix.batch; ++slot) modes_of(slot)[m].w = lt;
    }
  }
  // An item's read and write weights (softmax over the modes) by one warp, its decays by another (the formulas of
  // compute_params_kernel).  Loops of a mode a lane, not unrolled: what counts is how many instructions are fetched.
  __device__ __forceinline__ void weights(int l, const Item &it, float4 *P) {
    const float *f = a.tab[l].f;
    const int M = a.M, lane = at.lane;
    const float *rd = a.rw + (int64_t)it.b * 2 * a.H * M + (int64_t)it.h * M, *wr = rd + (int64_t)a.H * M;
    const float alpha = __ldcg(a.dyn + (int64_t)it.b * 3 * a.H + a.H + it.h);
#pragma unroll 4
    for (int m = lane; m < M; m += 32) {
      P[m].y = __ldcg(wr + m);
      P[m].z = __ldcg(rd + m);
    }
    const float read = sigmoid_(as_f32(extra[4], dt(l, kReadLogit))), write = sigmoid_(as_f32(extra[5], dt(l, kWriteLogit)));
    const float inv_temp = 1.f / f[kReadTemp];
    float cx = -INFINITY, kx = -INFINITY;
#pragma unroll 1
    for (int m = lane; m < M; m += 32) {
      const float prior = __fmul_rn(-alpha, P[m].w);
      const float c = __fmul_rn(fmaf(read, P[m].z, prior), inv_temp), k = fmaf(write, P[m].y, prior);
      P[m].z = c;
      P[m].y = k;
      cx = fmaxf(cx, c);
      kx = fmaxf(kx, k);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      cx = fmaxf(cx, __shfl_xor_sync(0xffffffffu, cx, o));
      kx = fmaxf(kx, __shfl_xor_sync(0xffffffffu, kx, o));
    }
    float cs = 0.f, ks = 0.f;
#pragma unroll 1
    for (int m = lane; m < M; m += 32) {
      cs += P[m].z = __expf(P[m].z - cx);
      ks += P[m].y = __expf(P[m].y - kx);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      cs += __shfl_xor_sync(0xffffffffu, cs, o);
      ks += __shfl_xor_sync(0xffffffffu, ks, o);
    }
    cs = 1.f / cs;
    ks = 1.f / ks;
#pragma unroll 1
    for (int m = lane; m < M; m += 32) {
      P[m].z *= cs;
      P[m].y *= ks;
    }
  }
  __device__ __forceinline__ void decays(const Item &it, float4 *P) const {
    const float *dyn = a.dyn + (int64_t)it.b * 3 * a.H + it.h;
    const float step = __ldcg(dyn), alpha = __ldcg(dyn + a.H), lam = __ldcg(dyn + 2 * a.H);
    const float rate = powf(fmaxf(lam, 1e-4f), 1.f / fmaxf(alpha, 1e-4f));
#pragma unroll 1
    for (int m = at.lane; m < a.M; m += 32) {
      const float rho = expf(-step * (rate / fmaxf(expf(P[m].w), 1e-6f)));
      P[m].x = fminf(fmaxf(rho, 1e-6f), 1.f - 1e-6f);
    }
  }

  __device__ __forceinline__ void run_mix(int l, int q, int mg) {
    const int first = at.block + at.team * at.blocks, step = at.blocks * at.teams;
    if (first >= a.mix.items) return;
    const int M = a.M, R = a.R, cols = a.mix.cols, groups = a.mix.groups;
    const bool on = mg < groups;
    float *const part = reinterpret_cast<float *>(modes_of(a.mix.batch));   // two exchange buffers [rows][cols]
    const int tid = at.tid, lane = at.lane, w = at.w, rows = a.mix.fold ? kWarps : groups;
    const float *const old = reinterpret_cast<const float *>(a.tab[l].p[kOldState]);
    float *const fresh = reinterpret_cast<float *>(a.tab[l].p[kNewState]);
    // what an item needs beside its state: u of this thread's four columns; u, gate, D and norm weight of column tid
    struct Small { uint2 uw; uint32_t uc, D, nw; float gc; };
    auto small = [&](const Item &it) {
      const int64_t col = head_of(it) * R + it.sp * cols;
      Small x{};
      if (on) x.uw = __ldcg(reinterpret_cast<const uint2 *>(a.x_conv + col + 4 * q));
      if (tid < cols) {
        x.uc = __ldcg(reinterpret_cast<const unsigned short *>(a.x_conv) + col + tid);
        x.gc = __ldcg(a.gate + col + tid);
      }
      return x;
    };
    auto small_params = [&](Small &x, const Item &it, int c) {
      const int64_t at_c = (int64_t)it.h * R + it.sp * cols + c;
      x.D = ld_bits(raw(l, kD), at_c, dt(l, kD));
      x.nw = ld_bits(raw(l, kOutNormW), at_c, dt(l, kOutNormW));
    };
    Small here = small(item_at(first));
    here.D = extra[6];
    here.nw = extra[7];
    int buffer = 0;
#pragma unroll 1
    for (int item0 = first; item0 < a.mix.items; item0 += a.mix.batch * step) {
      const int mine = item0 + (w >> 1) * step;
      if ((w >> 1) < a.mix.batch && mine < a.mix.items) {
        const Item it = item_at(mine);
        if (w & 1) decays(it, modes_of(w >> 1));
        else weights(l, it, modes_of(w >> 1));
      }
      at.sync();
#pragma unroll 1
      for (int j = 0; j < a.mix.batch; ++j, buffer ^= 1) {
        const int item = item0 + j * step, next = item + step;
        if (item >= a.mix.items) break;
        const bool more = next < a.mix.items;
        const Item it = item_at(item), nx = item_at(more ? next : item);
        const float4 *P = modes_of(j);
        // ---- the state one token further, and the readout; the next item's state is requested on the way
        const int64_t sbase = head_of(it) * M * R + it.sp * cols + 4 * q;
        const float *const mine_old = old ? old + sbase : nullptr;
        const float *const next_old = old && more ? old + head_of(nx) * M * R + nx.sp * cols + 4 * q : nullptr;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        const float u0 = bf(here.uw.x), u1 = bf_hi(here.uw.x), u2 = bf(here.uw.y), u3 = bf_hi(here.uw.y);
        const float4 *pm = P + mg;
        float *to = fresh ? fresh + sbase + mg * R : nullptr;
        const float *from = next_old ? next_old + mg * R : nullptr;
        const int hop = groups * R;
        auto token = [&](const uint4 &x) {
          const float4 y = *pm;
          const float rho = y.x, kap = __fmul_rn(1.f - rho, y.y), c = y.z;
          float4 v;
          v.x = fmaf(rho, __uint_as_float(x.x), __fmul_rn(kap, u0));
          v.y = fmaf(rho, __uint_as_float(x.y), __fmul_rn(kap, u1));
          v.z = fmaf(rho, __uint_as_float(x.z), __fmul_rn(kap, u2));
          v.w = fmaf(rho, __uint_as_float(x.w), __fmul_rn(kap, u3));
          if (fresh) __stcs(reinterpret_cast<float4 *>(to), v);
          acc.x = fmaf(c, v.x, acc.x);
          acc.y = fmaf(c, v.y, acc.y);
          acc.z = fmaf(c, v.z, acc.z);
          acc.w = fmaf(c, v.w, acc.w);
          pm += groups;
          to += hop;
        };
        // modes that this thread has left: all its pieces lie at mg + i * groups
        const int mine = on ? (M - mg + groups - 1) / groups : 0;
#pragma unroll
        for (int i = 0; i < kMixPre; ++i) {
          if (i < mine) {
            token(hold[i]);
            if (next_old) hold[i] = __ldcs(reinterpret_cast<const uint4 *>(from));
            from += hop;
          }
        }
#pragma unroll 1
        for (int i = kMixPre; i < mine; ++i)
          token(mine_old ? __ldcs(reinterpret_cast<const uint4 *>(mine_old + (int64_t)(mg + i * groups) * R)) : make_uint4(0, 0, 0, 0));
        Small then{};
        if (more) {
          then = small(nx);
          if (tid < cols) small_params(then, nx, tid);
        }
        float *const px = part + buffer * kTeam * 4;
        if (a.mix.fold) {
#pragma unroll 1
          for (int o = a.mix.quads; o < 32; o *= 2) {
            acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
            acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
            acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
            acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
          }
          if (lane < a.mix.quads) *reinterpret_cast<float4 *>(px + w * cols + 4 * q) = acc;
        } else if (on) {
          *reinterpret_cast<float4 *>(px + mg * cols + 4 * q) = acc;
        }
        at.sync();
        const int64_t col = head_of(it) * R + it.sp * cols;
        float sq = 0.f;
#pragma unroll 1
        for (int c = tid; c < cols; c += kTeam) {
          if (c != tid) {   // (heads wider than a team)
            small_params(here, it, c);
            here.uc = __ldcg(reinterpret_cast<const unsigned short *>(a.x_conv) + col + c);
            here.gc = __ldcg(a.gate + col + c);
          }
          float o = 0.f;
#pragma unroll 4
          for (int i = 0; i < rows; ++i) o += px[i * cols + c];
          const float z = here.gc + a.tab[l].f[kGateBias];
          const float v = __fmul_rn(fmaf(bf(here.uc), as_f32(here.D, dt(l, kD)), o), __fmul_rn(z, sigmoid_(z)));
          a.vals[col + c] = __float2bfloat16_rn(v * as_f32(here.nw, dt(l, kOutNormW)));
          sq = fmaf(v, v, sq);
        }
        if (w < a.mix.parts) {
          sq = sum_warp(sq);
          if (lane == 0) a.ss[(head_of(it) * a.splits + it.sp) * a.mix.parts + w] = sq;
        }
        here = then;
      }
    }
  }
};

// Puts this block on the list of those that share the work, by one thread.  Nothing is set where the list was closed before; for
// want of an answer within the limit *gave_up is.
__device__ void join(Meeting *m, uint64_t work_ns, uint64_t wait_ns, Place *at, int *gave_up) {
  const unsigned mine = atomicAdd(&m->started, 1u);
  if (mine & kClosed) return;
  const unsigned grid = gridDim.x;
  unsigned n = 0;
  const uint64_t t0 = umma::global_ns();
  if (mine == 0) {
#pragma unroll 1
    do {
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(&m->started) : "memory");
    } while (n < grid && !umma::past_limit(t0, umma::global_ns(), list_patience_ns(n, grid, work_ns)));
    n = atomicOr(&m->started, kClosed);
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&m->members), "r"(n) : "memory");
  } else {
#pragma unroll 1
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(n) : "l"(&m->members) : "memory");
      if (n) break;
      if (umma::past_limit(t0, umma::global_ns(), wait_ns)) {
        *gave_up = 1;
        return;
      }
    }
  }
  at->block = (int)mine;
  at->blocks = (int)n;
}

// All blocks of the list wait for one another, in two parts: a block arrives when its writes are done, and does what needs no other
// block in between.
__device__ __forceinline__ void arrive(unsigned *counter) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
  }
}
// False when the limit ran out, for every thread of the block.
__device__ __forceinline__ bool wait_for_all(const unsigned *counter, unsigned target, uint64_t wait_ns) {
  int gave_up = 0;
  if (threadIdx.x == 0) {
    uint64_t t0 = 0;
#pragma unroll 1
    for (uint32_t spins = 0;; ++spins) {
      unsigned seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
      if (static_cast<int>(seen - target) >= 0) break;
      if (spins == 64) t0 = umma::global_ns();
      if (spins > 64 && umma::past_limit(t0, umma::global_ns(), wait_ns)) {
        gave_up = 1;
        break;
      }
    }
  }
  return __syncthreads_or(gave_up) == 0;
}

// What a step leaves where a wait ran out: NaN throughout, by one block.
template <typename T>
__device__ __noinline__ void fill(T *p, int64_t n, T v) {
  for (int64_t i = threadIdx.x; p && i < n; i += blockDim.x) p[i] = v;
}
template <int LAYERS>
__device__ void mark_failed(const StepArgs<LAYERS> &a) {
  const unsigned short nan16 = 0x7fc0;
  const int64_t di = (int64_t)a.H * a.R;
  if (!a.after_w) fill(reinterpret_cast<unsigned short *>(a.out), (int64_t)a.B * a.d, nan16);
#pragma unroll 1
  for (int l = 0; l < a.layers; ++l) {
    fill(reinterpret_cast<float *>(a.tab[l].p[kNewState]), a.B * di * a.M, __int_as_float(0x7fc00000));
    fill(reinterpret_cast<unsigned short *>(a.tab[l].p[kNewConv]), a.B * di * 3, nan16);
  }
}

template <int NT>
__global__ void __launch_bounds__(kTeam * max_teams<NT>(), 1) decode_step_kernel(const __grid_constant__ StepArgs<kTabLayers> a) {
  extern __shared__ __align__(16) uint8_t smem[];
  Place at{(int)(threadIdx.x / kTeam), (int)(blockDim.x / kTeam), (int)(threadIdx.x % kTeam), (int)(threadIdx.x % 32),
           (int)(threadIdx.x % kTeam / 32), 0, 0};
  int *const listed = reinterpret_cast<int *>(smem);
  if (threadIdx.x == 0) {
    int gave_up = 0;
    Place mine{};
    join(a.meeting, a.work_ns, a.wait_ns, &mine, &gave_up);
    listed[0] = mine.block;
    listed[1] = gave_up ? -1 : mine.blocks;
  }
  __syncthreads();
  // (through a reduction, whose result the compiler knows to be the same in the whole warp: 24 layers at one sequence 496 us
  // against 498, at 32 sequences 879 against 883; as blockIdx and gridDim they were 495 and 869)
  at.block = __reduce_max_sync(0xffffffffu, listed[0]);
  at.blocks = __reduce_max_sync(0xffffffffu, listed[1]);
  __syncthreads();
  const int q = at.tid % a.mix.quads, mg = at.tid / a.mix.quads;
  Step<NT, kTabLayers> x{a, at, smem};
  bool ok = at.blocks >= 0;
  unsigned target = 0;
  // dyn_proj's tiles take blocks in proportion (a block alone takes them all, and the others after them)
  const int t2 = tiles_of(3 * a.H), t12 = t2 + tiles_of(2 * a.H * a.M);
  x.blocks2 = max(1, min((at.blocks * t2 + t12 - 1) / t12, at.blocks - 1));
  const int stages = at.blocks > 0 ? 4 * a.layers : -1;   // (none for a block that is not on the list)
  // Stage -1 only requests what the first one needs.  Beside a barrier the teams' shares of the weights of a later product
  // and of the layer's old state go to L2 (a lane of the block's last warp for each team), so that no stage waits for HBM.
  const bool carrier = threadIdx.x >= blockDim.x - 32 && at.lane < at.teams;
#pragma unroll 1
  for (int stage = -1; stage < stages; ++stage) {
    const int kind = stage & 3, next = stage + 1, nl = next >> 2, nk = next & 3;
    if (stage >= 0) {
      if (kind == kMix) x.run_mix(stage >> 2, q, mg);
      else {
#pragma unroll 1
        for (;;) {
          x.run_product(stage >> 2, kind);
          if (at.blocks > 1 || !x.second) break;
          __syncthreads();   // (the activations in shared memory are written anew)
          x.product(stage >> 2, kind, at.team, true);
          if (x.tile0 < x.tiles) x.request(x.tile0, x.k_lo);
        }
      }
      if (next == stages) break;
      arrive(&a.meeting->arrived);
    }
    if (nk == kMix) {
      x.request_state(nl, q, mg);
      x.mix_inputs(nl);
    }
    else x.ahead_product(nl, nk);
    if (carrier) {
      // in front of in_proj (not the first) out_proj's weights, in front of rw_proj the old state, then the next layer's
      // in_proj and rw_proj with dyn_proj; at the start rw_proj, dyn_proj and out_proj
      Step<NT, kTabLayers> y{a, at, smem};
      y.blocks2 = x.blocks2;
      if (nk == kProj) y.state_to_l2(nl, at.lane);
      const int cl = nk == kIn ? nl : nl + 1;
#pragma unroll 1
      for (int k = nk == kIn ? (stage < 0 ? kProj : kOut) : nk == kMix ? kIn : nk == kOut ? kProj : kLayerPtrs;
           k <= kOut && cl < a.layers; k = k == kProj && stage < 0 ? kOut : kLayerPtrs)
        y.product_to_l2(cl, k, at.lane);
    }
    if (stage >= 0) {
      target += (unsigned)at.blocks;
      if (!(ok = wait_for_all(&a.meeting->arrived, target + (at.block == 0 && next == a.lost ? at.blocks : 0), a.wait_ns))) break;
    }
  }
  // A block that gave up says so, and whoever leaves last, when nobody writes any more, sees it.
  __syncthreads();
  int bad = 0;
  if (threadIdx.x == 0) {
    if (!ok) atomicExch(&a.meeting->failed, 1u);
    asm volatile("fence.acq_rel.gpu;" ::: "memory");
    if (atomicAdd(&a.meeting->left, 1u) + 1 == gridDim.x) {
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      bad = atomicAdd(&a.meeting->failed, 0u) != 0;
    }
  }
  if (__syncthreads_or(bad)) mark_failed(a);
}

// One stage of one layer as a kernel: a block is a team.  (Two blocks per SM for the products up to 32 sequences: with three, and
// 80 registers a thread, they spilled, and 24 layers at one sequence took 0.49 instead of 0.39 ms.)
template <int NT, int KIND>
__global__ void __launch_bounds__(kTeam, KIND == kMix ? 3 : NT <= 4 ? 2 : 1)
decode_stage_kernel(const __grid_constant__ StepArgs<1> a) {
  extern __shared__ __align__(16) uint8_t smem[];
  const Place at{0, 1, (int)threadIdx.x, (int)(threadIdx.x % 32), (int)(threadIdx.x / 32), (int)blockIdx.x, (int)gridDim.x};
  grid_dep_launch();
  Step<NT, 1> x{a, at, smem};
  x.blocks2 = a.blocks2;
  if constexpr (KIND == kMix) {
    const int q = at.tid % a.mix.quads, mg = at.tid / a.mix.quads;
    x.request_state(0, q, mg);
    x.mix_inputs(0);
    grid_dep_wait();
    __syncthreads();   // (the modes' log_tau, written by all threads)
    x.run_mix(0, q, mg);
  } else {
    x.product(0, KIND, 0);
    if (x.tile0 < x.tiles) x.request(x.tile0, x.k_lo);
    if (KIND != kOut) x.ahead_epilogue(0, KIND);
    grid_dep_wait();
    if (KIND == kOut) x.ahead_epilogue(0, KIND);   // (reads the hidden state of an earlier kernel)
    x.run_product(0, KIND);
  }
}

size_t lin_smem_bytes(int nt, int64_t K) {
  const size_t red = (size_t)kWarps * 8 * kPassTiles * kRedStride * 4;
  return (nt == 1 ? 0 : 8 * nt * (size_t)act_stride((int)K)) + red;
}
size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// the columns of a (sequence, head) are spread over 1, 2 or 4 blocks while there are fewer of them than SMs
int mix_splits(int64_t B, int64_t H, int64_t R) {
  int s = 1;
  while (s < 4 && B * H * s < 148 && R % (8 * s) == 0) s *= 2;
  return s;
}

struct Scratch {
  size_t x, gate, x_conv, rw, dyn, vals, ss, hid, hid_w, hid_ss, meeting, bytes;
};
Scratch scratch_layout(int64_t B, int64_t d, int64_t di, int64_t H, int64_t M) {
  Scratch s{};
  size_t off = 0;
  auto take = [&](size_t n) { const size_t at = off; off += align256(n); return at; };
  s.meeting = take(sizeof(Meeting));   // (at the start: fracssm_decode_layers_status)
  s.x = take((size_t)B * di * 2);
  s.gate = take((size_t)B * di * 4);
  s.x_conv = take((size_t)B * di * 2);
  s.rw = take((size_t)B * 2 * H * M * 4);
  s.dyn = take((size_t)B * 3 * H * 4);
  s.vals = take((size_t)B * di * 2);
  s.ss = take((size_t)B * H * 4 * kWarps * 4);
  s.hid = take(2 * align256((size_t)B * d * 4));
  s.hid_w = take((size_t)B * d * 2);
  s.hid_ss = take((size_t)B * tiles_of((int)d) * 4);
  s.bytes = off;
  return s;
}

size_t mix_smem_bytes(int64_t M, int batch) { return (size_t)(batch * 4 * M + 2 * kTeam * 4) * 4; }

template <int LAYERS>
void fill_table(StepArgs<LAYERS> &a, const uint64_t *ptrs, const float *nums, int64_t layers, int64_t l0) {
  a.layers = (int)(layers - l0 < LAYERS ? layers - l0 : LAYERS);
  a.first = (int)l0;
  for (int l = 0; l < a.layers; ++l) {
    for (int i = 0; i < kLayerPtrs; ++i) a.tab[l].p[i] = ptrs[(l0 + l) * kLayerPtrs + i];
    for (int i = 0; i < kLayerNums; ++i) a.tab[l].f[i] = nums[(l0 + l) * kLayerNums + i];
  }
  const uint64_t *after = l0 + a.layers < layers ? ptrs + (l0 + a.layers) * kLayerPtrs : nullptr;
  a.after_w = after ? reinterpret_cast<const void *>(after[kNormW]) : nullptr;
  a.after_dt = after && !(after[kF32Mask] & 1) ? FRACSSM_BF16 : FRACSSM_F32;
}

struct Shape {
  int64_t B, d, H, R, M;
};
int64_t layer_weights(const Shape &p) { return 2 * p.H * p.R * (3 * p.d + 2 * p.H * p.M + 3 * p.H); }   // bytes
template <int LAYERS>
void fill_shape(StepArgs<LAYERS> &a, int nt, const Shape &p, char *ws, void *hidden_out) {
  const int64_t di = p.H * p.R;
  const Scratch s = scratch_layout(p.B, p.d, di, p.H, p.M);
  auto bf = [&](size_t off) { return reinterpret_cast<__nv_bfloat16 *>(ws + off); };
  auto fl = [&](size_t off) { return reinterpret_cast<float *>(ws + off); };
  a.B = (int)p.B; a.d = (int)p.d; a.H = (int)p.H; a.R = (int)p.R; a.M = (int)p.M;
  a.splits = mix_splits(p.B, p.H, p.R);
  a.l2_state = p.B * p.H * p.M * p.R * 4 <= (int64_t(48) << 20);   // beside a layer's weights, in an L2 of 126 MB
  MixShape &x = a.mix;
  x.cols = (int)p.R / a.splits;
  x.quads = x.cols / 4;
  x.groups = kTeam / x.quads;
  x.fold = x.quads <= 32 && (x.quads & (x.quads - 1)) == 0;   // a warp's mode groups of the same columns: added by shuffles
  x.items = (int)(p.B * p.H * a.splits);
  x.batch = LAYERS > 1 && p.M <= 512 ? kMixItems : 1;
  x.parts = x.cols >= kTeam ? kWarps : (x.cols + 31) / 32;
  a.red_bytes = (uint32_t)lin_smem_bytes(1, 0);
  a.act_bytes = (uint32_t)lin_smem_bytes(nt, p.d > di ? p.d : di) - a.red_bytes;
  a.mix_bytes = (uint32_t)mix_smem_bytes(p.M, x.batch);
  a.x = bf(s.x); a.x_conv = bf(s.x_conv); a.vals = bf(s.vals); a.hid_w = bf(s.hid_w);
  a.out = reinterpret_cast<__nv_bfloat16 *>(hidden_out);
  a.gate = fl(s.gate); a.rw = fl(s.rw); a.dyn = fl(s.dyn); a.ss = fl(s.ss); a.hid_ss = fl(s.hid_ss);
  a.hid[0] = fl(s.hid); a.hid[1] = fl(s.hid + align256((size_t)p.B * p.d * 4));
  a.meeting = reinterpret_cast<Meeting *>(ws + s.meeting);
}

// SM count of the current device; calls `prepare` once per device.
template <typename F>
int device_sms(int *sms, F prepare) {
  static std::mutex mu;
  static int count[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return fail(FRACSSM_ERR_CUDA, "decode_layers: cannot identify the current device");
  std::lock_guard<std::mutex> lock(mu);
  if (!count[dev]) {
    int n = 0;
    cudaError_t e = prepare();
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return fail(FRACSSM_ERR_CUDA, "decode_layers: %s", cudaGetErrorString(e));
    count[dev] = n;
  }
  *sms = count[dev];
  return FRACSSM_OK;
}
template <typename K>
cudaError_t all_smem(K kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMostSmem);
}
template <typename Arg>
cudaError_t launch(void (*kernel)(const Arg), unsigned grid, int threads, size_t smem, cudaStream_t st, bool dependent,
                   const Arg &arg) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, arg);
}
int launched(cudaError_t e) {
  if (e == cudaSuccess) return check_launch("decode_layers");
  cudaGetLastError();
  return fail(FRACSSM_ERR_CUDA, "decode_layers: %s", cudaGetErrorString(e));
}

// Where one kernel is the form to take.  24 layers as the whole model call, us, a kernel per stage / one kernel:
//                                sequences   1           8          12          16          17          20          32          64
//   hidden 768, 128 modes   plain call   696 / 503   692 / 543   720 / 592   692 / 628   889 / 766   969 / 786  1055 / 880   1570 / 1750
//                           captured     394 / 495   440 / 532   496 / 574   527 / 620   846 / 743   935 / 772  1031 / 866   1520 / 1740
//   FracConfig()            plain call   693 / 451   703 / 461   712 / 460   696 / 460   704 / 551   711 / 540   707 / 574    860 / 1060
//                           captured     297 / 394   310 / 421   370 / 451   356 / 429   467 / 531   466 / 519   515 / 561    810 / 1040
// (a plain call of the kernels waits for the host up to some 20 sequences; a captured one has no launches to save.)  Between 17
// and 32 sequences it depends on the model which of the captured forms is the faster; MB of weights a layer, us at 20 sequences:
//   hidden  768, 24 heads, modes 16   9.7  574 / 566     hidden 768, 12 heads, modes  32   9.5  482 / 527
//                                32  12.0  590 / 568                                  64  11.9  531 / 554
//                                64  16.7  730 / 625                                 128  16.6  749 / 662
//   hidden 1536, 24 heads, modes  8  31.1  992 / 896     hidden 512, 16 heads, modes 128  11.6  504 / 585
//   hidden 1024, 32 heads, modes 32  21.4  832 / 761     (32 sequences)
//   hidden 1024, 16 heads, modes 64  21.2  614 / 675     the one of these on the slower side of the line
constexpr int64_t kCapturedWeights = 12000000;      // bytes
bool one_kernel_pays(const Shape &p, cudaStream_t st) {
  if (p.B > 32) return false;
  if (p.B > 16 && layer_weights(p) > kCapturedWeights) return true;
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &status) != cudaSuccess) {
    cudaGetLastError();   // (the legacy stream while another is captured: the launches themselves say so)
    return false;
  }
  return status == cudaStreamCaptureStatusNone;
}

template <int NT>
int run_one_kernel(const uint64_t *ptrs, const float *nums, int64_t layers, void *hidden_out, char *ws, const Shape &p,
                   cudaStream_t st, const DecodeForm &how) {
  int sms = 0;
  const int rc = device_sms(&sms, [] { return all_smem(decode_step_kernel<NT>); });
  if (rc) return rc;
  StepArgs<kTabLayers> a{};
  fill_shape(a, NT, p, ws, hidden_out);
  // as many teams a block as the shared memory holds
  int teams = max_teams<NT>();
  auto smem_of = [&](int t) -> uint32_t {
    const uint32_t lin = a.act_bytes + t * a.red_bytes, mix = t * a.mix_bytes;
    return lin > mix ? lin : mix;
  };
  while (teams > 1 && smem_of(teams) > kMostSmem) --teams;
  const int grid = how.blocks > 0 ? how.blocks : sms;
  cudaError_t e = cudaSuccess;
  for (int64_t l0 = 0; l0 < layers && e == cudaSuccess; l0 += kTabLayers) {
    fill_table(a, ptrs, nums, layers, l0);
    // (the first kernel clears it for the first launch)
    if (l0) e = cudaMemsetAsync(a.meeting, 0, kPerLaunch, st);
    a.lost = l0 ? 0 : how.lost;
    a.work_ns = a.layers * (20000ull + (unsigned long long)layer_weights(p) / 4);   // (latency; 4 TB/s)
    a.wait_ns = list_limit_ns(grid, a.work_ns, how.wait_ns);
    if (e == cudaSuccess) e = launch(decode_step_kernel<NT>, (unsigned)grid, kTeam * teams, smem_of(teams), st, false, a);
  }
  return launched(e);
}

template <int NT>
int run_stages(const uint64_t *ptrs, const float *nums, int64_t layers, void *hidden_out, char *ws, const Shape &p,
               cudaStream_t st) {
  int sms = 0;
  const int rc = device_sms(&sms, [] {
    cudaError_t e = all_smem(decode_stage_kernel<NT, kIn>);
    if (e == cudaSuccess) e = all_smem(decode_stage_kernel<NT, kProj>);
    if (e == cudaSuccess) e = all_smem(decode_stage_kernel<NT, kMix>);
    if (e == cudaSuccess) e = all_smem(decode_stage_kernel<NT, kOut>);
    return e;
  });
  if (rc) return rc;
  StepArgs<1> a{};
  fill_shape(a, NT, p, ws, hidden_out);
  const int64_t di = p.H * p.R;
  // (the exchange buffer lies behind the activations of the longer of the two contractions)
  const size_t smem = a.act_bytes + a.red_bytes;
  // Up to 8 sequences a block takes one tile.  Beyond, filling the activation tile costs as much as a
  // tile's weights: one or two blocks per SM walk over the tiles.
  auto blocks = [&](int64_t rows) -> unsigned {
    const int64_t tiles = tiles_of((int)rows), most = sms * (smem <= 110 * 1024 ? 2 : 1);
    return (unsigned)(NT == 1 ? tiles : ceil_div(tiles, ceil_div(tiles, most)));
  };
  a.blocks2 = tiles_of((int)(3 * p.H));
  cudaError_t e = cudaSuccess;
  for (int64_t l = 0; l < layers && e == cudaSuccess; ++l) {
    fill_table(a, ptrs, nums, layers, l);
    e = launch(decode_stage_kernel<NT, kIn>, blocks(2 * di), kTeam, smem, st, true, a);
    if (e == cudaSuccess) e = launch(decode_stage_kernel<NT, kProj>, a.blocks2 + blocks(2 * p.H * p.M), kTeam, smem, st, true, a);
    if (e == cudaSuccess) e = launch(decode_stage_kernel<NT, kMix>, (unsigned)a.mix.items, kTeam, a.mix_bytes, st, true, a);
    if (e == cudaSuccess) e = launch(decode_stage_kernel<NT, kOut>, blocks(p.d), kTeam, smem, st, true, a);
  }
  return launched(e);
}

template <int NT>
int run_layers(const uint64_t *ptrs, const float *nums, int64_t layers, void *hidden_out, char *ws, const Shape &p,
               cudaStream_t st, const DecodeForm &how) {
  if constexpr (NT <= 4) {
    if (how.form == DecodeForm::kOneKernel || (how.form == DecodeForm::kByRule && one_kernel_pays(p, st)))
      return run_one_kernel<NT>(ptrs, nums, layers, hidden_out, ws, p, st, how);
  }
  return run_stages<NT>(ptrs, nums, layers, hidden_out, ws, p, st);
}

}  // namespace
}  // namespace fracssm

extern "C" int fracssm_decode_layers_supported(int64_t B, int64_t hidden, int64_t H, int64_t R, int64_t M, int64_t K) {
  using namespace fracssm;
  if (B < 1 || B > kMaxSeq || hidden < 32 || hidden > kMaxHidden || H < 1 || R < 4 || M < 1 || K != 4) return 0;
  if (H > 65536 || R > 1024 || M > 2048) return 0;
  const int64_t di = H * R;
  if (hidden % 32 != 0 || di % 32 != 0 || di > 65536 || R % 4 != 0 || H * M > (1 << 24)) return 0;
  const int nt = B <= 8 ? 1 : B <= 16 ? 2 : B <= 32 ? 4 : 8;
  return lin_smem_bytes(nt, di) <= 227 * 1024 && lin_smem_bytes(nt, hidden) <= 227 * 1024;
}

extern "C" size_t fracssm_decode_layers_workspace_bytes(int64_t B, int64_t hidden, int64_t H, int64_t R, int64_t M) {
  if (B < 1 || hidden < 1 || H < 1 || R < 1 || M < 1) return 0;
  return fracssm::scratch_layout(B, hidden, H * R, H, M).bytes;
}

int fracssm::decode_layers_launch(const uint64_t *layer_ptrs, const float *layer_nums, int64_t layers, const void *hidden_in,
                                  void *hidden_out, void *workspace, size_t workspace_bytes, int64_t B, int64_t hidden,
                                  int64_t H, int64_t R, int64_t M, int64_t K, void *stream, const DecodeForm &how) {
  if (layers < 1 || !layer_ptrs || !layer_nums || !hidden_in || !hidden_out || !workspace)
    return fail(FRACSSM_ERR_ARG, "decode_layers: null pointer or no layer");
  if (!fracssm_decode_layers_supported(B, hidden, H, R, M, K))
    return fail(FRACSSM_ERR_UNSUPPORTED, "decode_layers: sizes not covered");
  if (workspace_bytes < fracssm_decode_layers_workspace_bytes(B, hidden, H, R, M))
    return fail(FRACSSM_ERR_ARG, "decode_layers: workspace too small");
  uint64_t bits = (uint64_t)(uintptr_t)hidden_in | (uint64_t)(uintptr_t)hidden_out;
  if ((uintptr_t)workspace & 255) return fail(FRACSSM_ERR_ARG, "decode_layers: workspace must be 256-byte aligned");
  for (int64_t l = 0; l < layers; ++l) {
    const uint64_t *p = layer_ptrs + l * kLayerPtrs;
    for (int i = 0; i < kOldState; ++i)
      if (!p[i] && i != kConvB && i != kDynB) return fail(FRACSSM_ERR_ARG, "decode_layers: null parameter");
    bits |= p[kInW] | p[kDynW] | p[kRwW] | p[kOutW] | p[kOldState] | p[kNewState];
    if (p[kConvW] & 7) return fail(FRACSSM_ERR_ARG, "decode_layers: the convolution weight must be 8-byte aligned");
  }
  if (bits & 15)
    return fail(FRACSSM_ERR_ARG, "decode_layers: hidden states, projection weights and states must be 16-byte aligned");
  const cudaStream_t st = (cudaStream_t)stream;
  char *ws = reinterpret_cast<char *>(workspace);
  const Scratch s = scratch_layout(B, hidden, H * R, H, M);
  decode_first_kernel<<<(unsigned)B, kTeam, 0, st>>>(
      reinterpret_cast<const __nv_bfloat16 *>(hidden_in), reinterpret_cast<const void *>(layer_ptrs[kNormW]),
      layer_ptrs[kF32Mask] & 1 ? FRACSSM_F32 : FRACSSM_BF16, reinterpret_cast<float *>(ws + s.hid),
      reinterpret_cast<__nv_bfloat16 *>(ws + s.hid_w), reinterpret_cast<float *>(ws + s.hid_ss), (int)hidden,
      reinterpret_cast<Meeting *>(ws + s.meeting));
  const int rc = check_launch("decode_layers");
  if (rc) return rc;
  const Shape p{B, hidden, H, R, M};
  if (B <= 8) return run_layers<1>(layer_ptrs, layer_nums, layers, hidden_out, ws, p, st, how);
  if (B <= 16) return run_layers<2>(layer_ptrs, layer_nums, layers, hidden_out, ws, p, st, how);
  if (B <= 32) return run_layers<4>(layer_ptrs, layer_nums, layers, hidden_out, ws, p, st, how);
  return run_layers<8>(layer_ptrs, layer_nums, layers, hidden_out, ws, p, st, how);
}

extern "C" int fracssm_decode_layers(const uint64_t *layer_ptrs, const float *layer_nums, int64_t layers,
                                     const void *hidden_in, void *hidden_out, void *workspace, size_t workspace_bytes,
                                     int64_t B, int64_t hidden, int64_t H, int64_t R, int64_t M, int64_t K, void *stream) {
  return fracssm::decode_layers_launch(layer_ptrs, layer_nums, layers, hidden_in, hidden_out, workspace, workspace_bytes, B,
                                       hidden, H, R, M, K, stream, fracssm::DecodeForm{});
}

extern "C" int fracssm_decode_layers_status(const void *workspace, void *stream) {
  using namespace fracssm;
  if (!workspace) return fail(FRACSSM_ERR_ARG, "decode_layers_status: null workspace");
  Meeting m{};
  cudaError_t e = cudaMemcpyAsync(&m, workspace, sizeof(m), cudaMemcpyDeviceToHost, (cudaStream_t)stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) return fail(FRACSSM_ERR_CUDA, "decode_layers_status: %s", cudaGetErrorString(e));
  if (m.failed) return fail(FRACSSM_ERR_WAIT, "decode step: a device-side wait ran out");
  return FRACSSM_OK;
}
