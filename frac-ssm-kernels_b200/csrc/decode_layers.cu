// One decode token through all layers of the model, bfloat16, up to 64 sequences: four kernels per layer.
//
//   decode_linear_kernel<.., kIn>    in_proj of the normalised hidden state -> x | gate; the rows of x also take
//                                    the causal convolution step + SiLU (a channel needs its own history only)
//   decode_linear_kernel<.., kProj>  rw_proj of x_conv and dyn_proj of x
//   decode_mix_kernel                the scan parameters of a (sequence, head), its state one token further,
//                                    readout, D skip, gate
//   decode_linear_kernel<.., kOut>   out_proj of the normalised result -> + hidden state
// and decode_first_kernel once, which does for the embedding what kOut does for the next layer's norm.
//
// What bounds a step: reading the weights (27 MB a layer at hidden 768, 128 modes) and, from some 16 sequences
// on, the float32 state in and out; at one sequence the length of the kernel chain.  As separate library and
// elementwise calls (about 30 launches a layer, most of them from Python) a step of 24 layers was bound by the
// host.  Hence
//   * elementwise stages sit in the epilogue of the product that writes their rows.  A norm is split: whoever writes
//     the row also writes it times the norm's weight and the sums of squares of its part of the row, and the product
//     that reads it scales its results by 1 / rms, so no block has to see a whole row before it can start.  What
//     passes between the stages without going through a product (hidden state, gate, readout) stays float32;
//   * the products stream the weights once, straight into the fragments of mma.sync (16 weight rows x 16 of the
//     contraction x 8 sequences): with at most 64 sequences they are far below the tensor-core ridge, and a lane
//     reads 8 consecutive weights of a row because the contraction order is free as long as both operands share
//     it.  The 8 warps of a block split the contraction of a 16-row tile, so even 768 output rows keep 48 blocks
//     of 8 warps busy;
//   * every kernel is launched with programmatic stream serialisation: it requests what no kernel of this call
//     writes (weights, the old state and convolution history) before it waits for its predecessor.
// Whole model call, 24 layers of hidden 768, 24 heads x 128 modes, vocabulary 50280, before and now: 13.6 and 0.66 ms
// at one sequence (0.48 ms on the device, the rest is the host's 97 launches and look at 336 parameters), 13.7 and
// 1.1 ms at 32.
#include <mutex>

#include "common.cuh"
#include "scan_tile.cuh"

namespace fracssm {
namespace {

constexpr int kThreads = 256, kWarps = 8, kTileRows = 16, kMaxSeq = 64;
constexpr int kPre = 6;              // 32-wide steps of the contraction a warp holds weights for
constexpr int kRedStride = 20;       // floats per sequence in the exchange buffer: 16 rows, bank-conflict free
constexpr int kPassTiles = 2;        // groups of 8 sequences exchanged at a time
constexpr int kMaxHidden = 8192;     // longest hidden state
enum { kIn = 0, kProj = 1, kOut = 2 };

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

struct LinArgs {
  const __nv_bfloat16 *w, *w2;   // [n][K]; kProj: w = rw_proj, w2 = dyn_proj
  int n, n2, K, B, blocks2;      // kProj: the first blocks2 blocks take one tile of w2 each
  const __nv_bfloat16 *act, *act2;   // [B][K]; kProj: x_conv and x; else the row times the norm's weight
  const float *ss;               // kIn, kOut: partial sums of squares of the rows [B][nss]
  int nss;
  float eps;
  // kIn outputs and the convolution
  __nv_bfloat16 *x, *x_conv, *new_conv;
  float *gate;
  const __nv_bfloat16 *old_conv, *conv_w, *conv_b;
  int di;
  // kProj outputs
  float *out, *out2;
  const __nv_bfloat16 *bias2;
  // kOut: dst = res + result, and for the next layer's norm (weight next_w or null) dst * next_w and a sum per tile
  const float *res;              // the hidden state stays float32 from layer to layer
  float *dst;                    // null in the last layer, which writes bfloat16 to dst_last
  __nv_bfloat16 *dst_last, *dst_w;
  float *dst_ss;
  const void *next_w; int next_dt;
};

// 16 bytes to shared memory, zeros where `on` is false
__device__ __forceinline__ void copy_async16(uint32_t dst, const void *src, bool on) {
  const int n = on ? 16 : 0;   // (0: nothing is read)
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// NT groups of 8 sequences.
template <int NT, int KIND>
__global__ void __launch_bounds__(kThreads, NT == 1 ? 3 : NT <= 4 ? 2 : 1) decode_linear_kernel(const LinArgs a) {
  extern __shared__ __align__(16) uint8_t lin_smem[];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, tig = lane & 3;
  grid_dep_launch();
  // rows of the activation tile lie 64 mod 128 bytes apart: a quarter-warp's 16-byte reads then cover all banks
  const uint32_t stride = a.K * 2 + ((a.K * 2) % 128 == 0 ? 64 : 128);
  float *red = reinterpret_cast<float *>(lin_smem + (NT == 1 ? 0 : 8 * NT * stride));
  const bool second = KIND == kProj && (int)blockIdx.x < a.blocks2;
  const __nv_bfloat16 *W = second ? a.w2 : a.w;
  const int N = second ? a.n2 : a.n;
  const int tile0 = KIND == kProj && !second ? blockIdx.x - a.blocks2 : blockIdx.x;
  const int tiles = (N + kTileRows - 1) / kTileRows;
  const int tile_step = second ? tiles : KIND == kProj ? gridDim.x - a.blocks2 : gridDim.x;
  const int steps = a.K / 32, share = (steps + kWarps - 1) / kWarps;
  const int k_lo = min(w * share, steps), k_hi = min(k_lo + share, steps);

  uint4 wr[kPre][2];
  auto request = [&](int tile, int k0) {
    const int r0 = min(tile * kTileRows + g, N - 1), r1 = min(tile * kTileRows + g + 8, N - 1);
    const __nv_bfloat16 *p0 = W + (int64_t)r0 * a.K + 8 * tig, *p1 = W + (int64_t)r1 * a.K + 8 * tig;
#pragma unroll
    for (int i = 0; i < kPre; ++i) {
      if (k0 + i < k_hi) {
        wr[i][0] = ldg_weights(p0 + (k0 + i) * 32);
        wr[i][1] = ldg_weights(p1 + (k0 + i) * 32);
      }
    }
  };
  request(tile0, k_lo);
  // what the epilogue of this thread's first value needs and no kernel of this call writes
  const int e_row = tid & 15, e_seq = tid >> 4;
  constexpr int kPasses = (NT + kPassTiles - 1) / kPassTiles;
  uint2 cw = make_uint2(0, 0);
  float cb = 0.f, nw = 0.f;
  __nv_bfloat16 ch[kPasses][3] = {};
  auto conv_inputs = [&](int n) {   // of row n, for all of this thread's sequences
    if (n >= a.di) return;
    cw = *reinterpret_cast<const uint2 *>(a.conv_w + (int64_t)n * 4);
    cb = a.conv_b ? __bfloat162float(a.conv_b[n]) : 0.f;
    if (a.old_conv) {
#pragma unroll
      for (int p = 0; p < kPasses; ++p) {
        const int b = 8 * kPassTiles * p + e_seq;
        if (b < a.B) {
          const __nv_bfloat16 *src = a.old_conv + ((int64_t)b * a.di + n) * 3;
          ch[p][0] = src[0]; ch[p][1] = src[1]; ch[p][2] = src[2];
        }
      }
    }
  };
  const int e_n = tile0 * kTileRows + e_row;
  if (KIND == kIn) conv_inputs(e_n);
  if (KIND == kOut && a.next_w && e_n < N) nw = ld_f32(a.next_w, e_n, a.next_dt);

  grid_dep_wait();

  // ---- activations (bf16, zeros beyond B): each warp its own share of the contraction.  Up to 8 sequences straight
  // into the fragments; beyond, every tile reads them again, so they go to shared memory once.
  const __nv_bfloat16 *act = second ? a.act2 : a.act;
  const uint32_t act_s = (uint32_t)__cvta_generic_to_shared(lin_smem);
  if (NT > 1) {
    const int pieces = (k_hi - k_lo) * 4;     // 16-byte pieces of this warp's share of a row
    for (int i = lane; i < pieces; i += 32) {
      const __nv_bfloat16 *src = act + (4 * k_lo + i) * 8;
      uint32_t dst = act_s + (4 * k_lo + i) * 16;
#pragma unroll 8
      for (int b = 0; b < 8 * NT; ++b, dst += stride) {
        copy_async16(dst, src, b < a.B);
        if (b + 1 < a.B) src += a.K;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // 1 / rms of this thread's sequences: 16 threads share one
  float rs[kPasses];
  if (KIND != kProj) {
#pragma unroll
    for (int p = 0; p < kPasses; ++p) {
      const int b = 8 * kPassTiles * p + e_seq;
      float t = 0.f;
      if (b < a.B)
        for (int i = e_row; i < a.nss; i += 16) t += __ldcg(a.ss + (int64_t)b * a.nss + i);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      rs[p] = rsqrtf(t / (float)a.K + a.eps);
    }
  }
  if (NT > 1) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
  }

  for (int tile = tile0; tile < tiles; tile += tile_step) {
    float acc[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
    for (int k0 = k_lo; k0 < k_hi; k0 += kPre) {
      if (k0 != k_lo) request(tile, k0);
      uint4 xs[NT == 1 ? kPre : 1];
      if (NT == 1) {
#pragma unroll
        for (int i = 0; i < kPre; ++i) {
          xs[i] = make_uint4(0, 0, 0, 0);
          if (k0 + i < k_hi && g < a.B)
            xs[i] = __ldcg(reinterpret_cast<const uint4 *>(act + (int64_t)g * a.K + (k0 + i) * 32 + 8 * tig));
        }
      }
#pragma unroll
      for (int i = 0; i < kPre; ++i) {
        if (k0 + i < k_hi) {
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            const uint4 x = NT == 1 ? xs[NT == 1 ? i : 0]
                                    : *reinterpret_cast<const uint4 *>(lin_smem + (8 * t + g) * stride +
                                                                       (k0 + i) * 64 + 16 * tig);
            mma_bf16(acc[t], wr[i][0].x, wr[i][1].x, wr[i][0].y, wr[i][1].y, x.x, x.y);
            mma_bf16(acc[t], wr[i][0].z, wr[i][1].z, wr[i][0].w, wr[i][1].w, x.z, x.w);
          }
        }
      }
    }
    if (tile + tile_step < tiles) request(tile + tile_step, k_lo);   // on their way during the epilogue
    if (KIND == kIn && tile != tile0) conv_inputs(tile * kTileRows + e_row);
    // ---- the warps' shares of the contraction are added, a value per thread
#pragma unroll
    for (int p = 0; p < NT; p += kPassTiles) {
#pragma unroll
      for (int t = p; t < p + kPassTiles && t < NT; ++t) {
        float *d = red + (w * 8 * kPassTiles + 8 * (t - p) + 2 * tig) * kRedStride + g;
        d[0] = acc[t][0];
        d[kRedStride] = acc[t][1];
        d[8] = acc[t][2];
        d[kRedStride + 8] = acc[t][3];
      }
      __syncthreads();
      const int b = 8 * p + e_seq, n = tile * kTileRows + e_row;
      const bool on = e_seq < 8 * (NT - p) && b < a.B && n < N;
      float sq = 0.f;
      if (on) {
        float v = 0.f;
#pragma unroll
        for (int i = 0; i < kWarps; ++i) v += red[(i * 8 * kPassTiles + e_seq) * kRedStride + e_row];
        if (KIND != kProj) v *= rs[p / kPassTiles];
        if (KIND == kIn) {
          const __nv_bfloat16 xb = __float2bfloat16_rn(v);
          if (n < a.di) {
            const float xv = __bfloat162float(xb);
            const __nv_bfloat16 *c3 = ch[p / kPassTiles];
            const float c0 = __bfloat162float(c3[0]), c1 = __bfloat162float(c3[1]), c2 = __bfloat162float(c3[2]);
            float y = cb;
            y = fmaf(bf(cw.x), c0, y);
            y = fmaf(bf_hi(cw.x), c1, y);
            y = fmaf(bf(cw.y), c2, y);
            y = fmaf(bf_hi(cw.y), xv, y);
            const int64_t at = (int64_t)b * a.di + n;
            a.x[at] = xb;
            a.x_conv[at] = __float2bfloat16_rn(y / (1.f + __expf(-y)));
            if (a.new_conv) {
              __nv_bfloat16 *q = a.new_conv + at * 3;
              q[0] = c3[1];
              q[1] = c3[2];
              q[2] = xb;
            }
          } else {
            a.gate[(int64_t)b * a.di + n - a.di] = v;
          }
        } else if (KIND == kProj) {
          if (second) a.out2[(int64_t)b * N + n] = v + (a.bias2 ? __bfloat162float(a.bias2[n]) : 0.f);
          else a.out[(int64_t)b * N + n] = v;
        } else {
          const int64_t at = (int64_t)b * N + n;
          const float hv = __ldcg(a.res + at) + v;
          if (a.dst) a.dst[at] = hv;
          else a.dst_last[at] = __float2bfloat16_rn(hv);
          if (a.next_w) {
            if (tile != tile0) nw = ld_f32(a.next_w, n, a.next_dt);
            a.dst_w[at] = __float2bfloat16_rn(hv * nw);
            sq = hv * hv;
          }
        }
      }
      if (KIND == kOut && a.next_w) {   // the tile's 16 rows of a sequence lie in 16 neighbouring lanes
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (on && e_row == 0) a.dst_ss[(int64_t)b * tiles + tile] = sq;
      }
      __syncthreads();
    }
  }
}

// The embedding times the first norm's weight, and its sums of squares (one part per row).
__global__ void __launch_bounds__(kThreads)
decode_first_kernel(const __nv_bfloat16 *h, const void *w, int w_dt, float *h_f32, __nv_bfloat16 *h_w, float *ss, int d) {
  __shared__ float red[kWarps];
  const int64_t b = blockIdx.x;
  grid_dep_launch();
  float sq = 0.f;
  for (int i = threadIdx.x; i < d; i += kThreads) {
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

struct MixArgs {
  const float *rw, *dyn;               // [B][2 H M], [B][3 H]
  const __nv_bfloat16 *x_conv;         // [B][H R]
  const float *gate;                   // [B][H R]
  const float *old_state;              // [B][H][M][R] or null (zeros)
  float *new_state;                    // or null
  const void *dt_bias, *read_logit, *write_logit, *log_tau, *D, *norm_w;
  int dt_bias_dt, read_dt, write_dt, log_tau_dt, D_dt, norm_dt;
  float inv_read_temp, dt_min, dt_max, a_min, a_max, l_min, l_max, gate_bias;
  __nv_bfloat16 *vals;                 // [B][H R]: the gated result times the output norm's weight
  float *ss;                           // [B][H splits]: sums of squares of the gated result
  int H, R, M, splits;
};

constexpr int kMixPre = 8;             // float4 pieces of the old state a thread requests ahead

// One block per (sequence, head, share of the head's columns).
__global__ void __launch_bounds__(kThreads) decode_mix_kernel(const MixArgs a) {
  extern __shared__ __align__(16) float mix_smem[];
  const int M = a.M, H = a.H, R = a.R, Mr = (M + 3) & ~3;
  float *cc = mix_smem, *kk = cc + Mr, *rr = kk + Mr, *part = rr + Mr;   // part [rows][cols], 16-byte aligned
  __shared__ float red[2][4][2], sums[kWarps];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int h = blockIdx.x / a.splits, sp = blockIdx.x % a.splits, b = blockIdx.y;
  const int cols = R / a.splits, quads = cols / 4, groups = kThreads / quads;
  const int q = tid % quads, mg = tid / quads;
  const bool on = mg < groups;
  // a warp holds several mode groups of the same columns when quads is a power of two: they are added by shuffles
  const bool fold = quads <= 32 && (quads & (quads - 1)) == 0;
  grid_dep_launch();
  // ---- requested before the wait: the old state, the parameters
  const int64_t sbase = ((int64_t)b * H + h) * M * R + sp * cols + 4 * q;
  float4 pre[kMixPre];
#pragma unroll
  for (int i = 0; i < kMixPre; ++i) {
    const int m = mg + i * groups;
    pre[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (on && m < M && a.old_state)
      pre[i] = __ldcs(reinterpret_cast<const float4 *>(a.old_state + sbase + (int64_t)m * R));
  }
  // threads 0..127: the read side of the parameters, 128..255 the write side
  const int side = tid >> 7, t128 = tid & 127;
  const float read_gate = sigmoid_(ld_f32(a.read_logit, 0, a.read_dt));
  const float write_gate = sigmoid_(ld_f32(a.write_logit, 0, a.write_dt));
  const float dtb = ld_f32(a.dt_bias, h, a.dt_bias_dt);
  const float lt0 = t128 < M ? ld_f32(a.log_tau, t128, a.log_tau_dt) : 0.f;
  const float tau0 = fmaxf(expf(lt0), 1e-6f);
  float Dv = 0.f, nwv = 0.f;
  if (tid < cols) {
    Dv = ld_f32(a.D, (int64_t)h * R + sp * cols + tid, a.D_dt);
    nwv = ld_f32(a.norm_w, (int64_t)h * R + sp * cols + tid, a.norm_dt);
  }
  grid_dep_wait();

  // ---- scan parameters (the formulas of compute_params_kernel)
  const float *dyn = a.dyn + (int64_t)b * 3 * H + h;
  const float *res = a.rw + (int64_t)b * 2 * H * M + (int64_t)side * H * M + (int64_t)h * M;
  const float r0 = t128 < M ? __ldcg(res + t128) : 0.f;
  const float y0 = __ldcg(dyn), y1 = __ldcg(dyn + H), y2 = __ldcg(dyn + 2 * H);
  const int64_t col = (int64_t)b * H * R + (int64_t)h * R + sp * cols;
  uint2 uw = make_uint2(0, 0);
  if (on) uw = __ldcg(reinterpret_cast<const uint2 *>(a.x_conv + col + 4 * q));
  float uc = 0.f, gc = 0.f;
  if (tid < cols) {
    uc = __bfloat162float(__ldcg(a.x_conv + col + tid));
    gc = __ldcg(a.gate + col + tid);
  }
  const float d0 = y0 + dtb;
  float dt = d0 > 20.f ? d0 : log1pf(expf(d0));
  dt = fminf(fmaxf(dt, a.dt_min), a.dt_max);
  const float alpha = a.a_min + sigmoid_(y1) * (a.a_max - a.a_min);
  const float lam = a.l_min + sigmoid_(y2) * (a.l_max - a.l_min);
  const float rate = powf(fmaxf(lam, 1e-4f), 1.f / fmaxf(alpha, 1e-4f));
  float *dst = side ? kk : cc;
  float mx = -INFINITY;
  for (int m = t128; m < M; m += 128) {
    const float prior = -alpha * (m == t128 ? lt0 : ld_f32(a.log_tau, m, a.log_tau_dt));
    const float rv = m == t128 ? r0 : __ldcg(res + m);
    const float l = side ? prior + write_gate * rv : (prior + read_gate * rv) * a.inv_read_temp;
    dst[m] = l;
    mx = fmaxf(mx, l);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) red[side][w & 3][0] = mx;
  __syncthreads();
  mx = fmaxf(fmaxf(red[side][0][0], red[side][1][0]), fmaxf(red[side][2][0], red[side][3][0]));
  float sum = 0.f;
  for (int m = t128; m < M; m += 128) {
    const float e = __expf(dst[m] - mx);
    dst[m] = e;
    sum += e;
  }
  sum = sum_warp(sum);
  if (lane == 0) red[side][w & 3][1] = sum;
  __syncthreads();
  const float inv = 1.f / (red[side][0][1] + red[side][1][1] + red[side][2][1] + red[side][3][1]);
  for (int m = t128; m < M; m += 128) {
    if (side) {
      float rho = expf(-dt * (rate / (m == t128 ? tau0 : fmaxf(expf(ld_f32(a.log_tau, m, a.log_tau_dt)), 1e-6f))));
      rho = fminf(fmaxf(rho, 1e-6f), 1.f - 1e-6f);
      kk[m] = (1.f - rho) * (kk[m] * inv);
      rr[m] = rho;
    } else {
      cc[m] *= inv;
    }
  }
  __syncthreads();

  // ---- the state one token further, and the readout
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (on) {
    const float u0 = bf(uw.x), u1 = bf_hi(uw.x), u2 = bf(uw.y), u3 = bf_hi(uw.y);
    auto step = [&](int m, float4 s) {
      const float rho = rr[m], kap = kk[m], c = cc[m];
      s.x = fmaf(rho, s.x, kap * u0);
      s.y = fmaf(rho, s.y, kap * u1);
      s.z = fmaf(rho, s.z, kap * u2);
      s.w = fmaf(rho, s.w, kap * u3);
      if (a.new_state) __stcs(reinterpret_cast<float4 *>(a.new_state + sbase + (int64_t)m * R), s);
      acc.x = fmaf(c, s.x, acc.x);
      acc.y = fmaf(c, s.y, acc.y);
      acc.z = fmaf(c, s.z, acc.z);
      acc.w = fmaf(c, s.w, acc.w);
    };
#pragma unroll
    for (int i = 0; i < kMixPre; ++i)
      if (mg + i * groups < M) step(mg + i * groups, pre[i]);
#pragma unroll 4
    for (int m = mg + kMixPre * groups; m < M; m += groups)
      step(m, a.old_state ? __ldcs(reinterpret_cast<const float4 *>(a.old_state + sbase + (int64_t)m * R))
                          : make_float4(0.f, 0.f, 0.f, 0.f));
  }
  if (fold) {
    for (int o = quads; o < 32; o *= 2) {
      acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
      acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
      acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
      acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
    }
    if (lane < quads) *reinterpret_cast<float4 *>(part + w * cols + 4 * q) = acc;
  } else if (on) {
    *reinterpret_cast<float4 *>(part + mg * cols + 4 * q) = acc;
  }
  __syncthreads();
  const int rows = fold ? kWarps : groups;
  float sq = 0.f;
  for (int c = tid; c < cols; c += kThreads) {
    if (c != tid) {   // (heads wider than the block)
      Dv = ld_f32(a.D, (int64_t)h * R + sp * cols + c, a.D_dt);
      nwv = ld_f32(a.norm_w, (int64_t)h * R + sp * cols + c, a.norm_dt);
      uc = __bfloat162float(__ldcg(a.x_conv + col + c));
      gc = __ldcg(a.gate + col + c);
    }
    float o = 0.f;
#pragma unroll 8
    for (int i = 0; i < rows; ++i) o += part[i * cols + c];
    const float z = gc + a.gate_bias;
    const float v = (o + uc * Dv) * (z * sigmoid_(z));
    a.vals[col + c] = __float2bfloat16_rn(v * nwv);
    sq = fmaf(v, v, sq);
  }
  sq = sum_warp(sq);
  if (lane == 0) sums[w] = sq;
  __syncthreads();
  if (tid == 0) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < kWarps; ++i) t += sums[i];
    a.ss[(int64_t)b * H * a.splits + h * a.splits + sp] = t;
  }
}

template <typename Arg>
cudaError_t launch_dep(void (*kernel)(const Arg), dim3 grid, size_t smem, cudaStream_t st, bool dependent, const Arg &arg) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, arg);
}

size_t lin_smem_bytes(int nt, int64_t K) {
  const size_t stride = K * 2 + ((K * 2) % 128 == 0 ? 64 : 128);
  const size_t red = (size_t)kWarps * 8 * kPassTiles * kRedStride * 4;
  return (nt == 1 ? 0 : 8 * nt * stride) + red;
}
size_t mix_smem_bytes(int64_t M) { return (size_t)(3 * ((M + 3) / 4 * 4) + kThreads * 4) * 4; }

template <int NT>
cudaError_t allow_smem() {
  constexpr int kMost = 227 * 1024;
  constexpr cudaFuncAttribute kAttr = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaFuncSetAttribute(decode_linear_kernel<NT, kIn>, kAttr, kMost);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(decode_linear_kernel<NT, kProj>, kAttr, kMost);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(decode_linear_kernel<NT, kOut>, kAttr, kMost);
  return e;
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// the columns of a (sequence, head) are spread over 1, 2 or 4 blocks while the launch has fewer blocks than SMs
int mix_splits(int64_t B, int64_t H, int64_t R) {
  int s = 1;
  while (s < 4 && B * H * s < 148 && R % (8 * s) == 0) s *= 2;
  return s;
}

struct Scratch {
  size_t x, gate, x_conv, rw, dyn, vals, ss, hid, hid_w, hid_ss, bytes;
};
Scratch scratch_layout(int64_t B, int64_t d, int64_t di, int64_t H, int64_t M) {
  Scratch s{};
  size_t off = 0;
  auto take = [&](size_t n) { const size_t at = off; off += align256(n); return at; };
  s.x = take((size_t)B * di * 2);
  s.gate = take((size_t)B * di * 4);
  s.x_conv = take((size_t)B * di * 2);
  s.rw = take((size_t)B * 2 * H * M * 4);
  s.dyn = take((size_t)B * 3 * H * 4);
  s.vals = take((size_t)B * di * 2);
  s.ss = take((size_t)B * H * 4 * 4);
  s.hid = take(2 * align256((size_t)B * d * 4));
  s.hid_w = take((size_t)B * d * 2);
  s.hid_ss = take((size_t)B * ((d + kTileRows - 1) / kTileRows) * 4);
  s.bytes = off;
  return s;
}

enum LayerPtr { kNormW, kInW, kConvW, kConvB, kDynW, kDynB, kRwW, kDtBias, kReadLogit, kWriteLogit, kLogTau, kD,
                kOutNormW, kOutW, kOldState, kOldConv, kNewState, kNewConv, kF32Mask, kLayerPtrs };
enum LayerNum { kEpsIn, kEpsOut, kReadTemp, kDtMin, kDtMax, kAMin, kAMax, kLMin, kLMax, kGateBias, kLayerNums };

template <int NT>
int run_layers(const uint64_t *ptrs, const float *nums, int64_t layers, const void *hidden_in, void *hidden_out,
               char *ws, int64_t B, int64_t d, int64_t H, int64_t R, int64_t M, cudaStream_t st) {
  static std::mutex mu;
  static bool ready[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
    return fail(FRACSSM_ERR_CUDA, "decode_layers: cannot identify the current device");
  {
    std::lock_guard<std::mutex> lock(mu);
    if (!ready[dev]) {
      const cudaError_t e = allow_smem<NT>();
      if (e != cudaSuccess) return fail(FRACSSM_ERR_CUDA, "decode_layers: %s", cudaGetErrorString(e));
      ready[dev] = true;
    }
  }
  const int64_t di = H * R;
  const Scratch s = scratch_layout(B, d, di, H, M);
  const int splits = mix_splits(B, H, R);
  const size_t smem_d = lin_smem_bytes(NT, d), smem_di = lin_smem_bytes(NT, di), mix_smem = mix_smem_bytes(M);
  auto at = [&](size_t off) { return ws + off; };
  const int64_t tiles_in = ceil_div(2 * di, kTileRows), tiles_rw = ceil_div(2 * H * M, kTileRows),
                tiles_dyn = ceil_div(3 * H, kTileRows), tiles_out = ceil_div(d, kTileRows);
  // Up to 8 sequences a block takes one tile (three blocks per SM: up to 444 tiles, 7104 output rows, are resident at
  // once, which the products of a model of hidden 768 are).  Beyond, filling the activation tile costs as much as a
  // tile's weights: one or two blocks per SM walk over the tiles.
  auto blocks = [&](int64_t tiles, size_t smem) -> int64_t {
    if (NT == 1) return tiles;
    const int64_t most = 148 * (smem <= 110 * 1024 ? 2 : 1);
    return ceil_div(tiles, ceil_div(tiles, most));
  };
  cudaError_t e = cudaSuccess;
  // the hidden state, float32, in two buffers in turn
  auto hid_at = [&](int64_t l) { return reinterpret_cast<float *>(at(s.hid) + (l & 1) * align256((size_t)B * d * 4)); };
  __nv_bfloat16 *hid_w = reinterpret_cast<__nv_bfloat16 *>(at(s.hid_w));
  float *hid_ss = reinterpret_cast<float *>(at(s.hid_ss));
  decode_first_kernel<<<(unsigned)B, kThreads, 0, st>>>(reinterpret_cast<const __nv_bfloat16 *>(hidden_in),
                                                       reinterpret_cast<const void *>(ptrs[kNormW]),
                                                       ptrs[kF32Mask] & 1 ? FRACSSM_F32 : FRACSSM_BF16, hid_at(0), hid_w,
                                                       hid_ss, (int)d);
  e = cudaGetLastError();
  for (int64_t l = 0; l < layers && e == cudaSuccess; ++l) {
    const uint64_t *p = ptrs + l * kLayerPtrs;
    const float *f = nums + l * kLayerNums;
    const uint64_t f32 = p[kF32Mask];
    auto bfp = [&](int i) { return reinterpret_cast<const __nv_bfloat16 *>(p[i]); };
    auto raw = [&](int i) { return reinterpret_cast<const void *>(p[i]); };
    auto dt = [&](int i) { return (f32 >> i) & 1 ? FRACSSM_F32 : FRACSSM_BF16; };
    LinArgs in{};
    in.w = bfp(kInW); in.n = (int)(2 * di); in.K = (int)d; in.B = (int)B;
    in.act = hid_w; in.ss = hid_ss; in.nss = l == 0 ? 1 : (int)tiles_out; in.eps = f[kEpsIn];
    in.x = reinterpret_cast<__nv_bfloat16 *>(at(s.x));
    in.gate = reinterpret_cast<float *>(at(s.gate));
    in.x_conv = reinterpret_cast<__nv_bfloat16 *>(at(s.x_conv));
    in.new_conv = reinterpret_cast<__nv_bfloat16 *>(p[kNewConv]);
    in.old_conv = bfp(kOldConv);
    in.conv_w = bfp(kConvW); in.conv_b = bfp(kConvB); in.di = (int)di;
    e = launch_dep(decode_linear_kernel<NT, kIn>, dim3((unsigned)blocks(tiles_in, smem_d)), smem_d, st, true, in);
    if (e != cudaSuccess) break;

    LinArgs pr{};
    pr.w = bfp(kRwW); pr.n = (int)(2 * H * M); pr.w2 = bfp(kDynW); pr.n2 = (int)(3 * H); pr.K = (int)di; pr.B = (int)B;
    pr.blocks2 = (int)tiles_dyn;
    pr.act = in.x_conv; pr.act2 = in.x;
    pr.out = reinterpret_cast<float *>(at(s.rw)); pr.out2 = reinterpret_cast<float *>(at(s.dyn));
    pr.bias2 = bfp(kDynB);
    const dim3 pr_grid((unsigned)(tiles_dyn + blocks(tiles_rw, smem_di)));
    e = launch_dep(decode_linear_kernel<NT, kProj>, pr_grid, smem_di, st, true, pr);
    if (e != cudaSuccess) break;

    MixArgs m{};
    m.rw = pr.out; m.dyn = pr.out2; m.x_conv = in.x_conv; m.gate = in.gate;
    m.old_state = reinterpret_cast<const float *>(p[kOldState]);
    m.new_state = reinterpret_cast<float *>(p[kNewState]);
    m.dt_bias = raw(kDtBias); m.dt_bias_dt = dt(kDtBias);
    m.read_logit = raw(kReadLogit); m.read_dt = dt(kReadLogit);
    m.write_logit = raw(kWriteLogit); m.write_dt = dt(kWriteLogit);
    m.log_tau = raw(kLogTau); m.log_tau_dt = dt(kLogTau);
    m.D = raw(kD); m.D_dt = dt(kD);
    m.inv_read_temp = 1.f / f[kReadTemp];
    m.dt_min = f[kDtMin]; m.dt_max = f[kDtMax]; m.a_min = f[kAMin]; m.a_max = f[kAMax];
    m.l_min = f[kLMin]; m.l_max = f[kLMax]; m.gate_bias = f[kGateBias];
    m.norm_w = raw(kOutNormW); m.norm_dt = dt(kOutNormW);
    m.vals = reinterpret_cast<__nv_bfloat16 *>(at(s.vals)); m.ss = reinterpret_cast<float *>(at(s.ss));
    m.H = (int)H; m.R = (int)R; m.M = (int)M; m.splits = splits;
    e = launch_dep(decode_mix_kernel, dim3((unsigned)(H * splits), (unsigned)B), mix_smem, st, true, m);
    if (e != cudaSuccess) break;

    LinArgs o{};
    o.w = bfp(kOutW); o.n = (int)d; o.K = (int)di; o.B = (int)B;
    o.act = m.vals; o.ss = m.ss; o.nss = (int)(H * splits); o.eps = f[kEpsOut];
    o.res = hid_at(l);
    if (l + 1 < layers) o.dst = hid_at(l + 1);
    else o.dst_last = reinterpret_cast<__nv_bfloat16 *>(hidden_out);
    if (l + 1 < layers) {
      o.dst_w = hid_w; o.dst_ss = hid_ss;
      o.next_w = reinterpret_cast<const void *>(p[kLayerPtrs + kNormW]);
      o.next_dt = p[kLayerPtrs + kF32Mask] & 1 ? FRACSSM_F32 : FRACSSM_BF16;
    }
    e = launch_dep(decode_linear_kernel<NT, kOut>, dim3((unsigned)blocks(tiles_out, smem_di)), smem_di, st, true, o);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(FRACSSM_ERR_CUDA, "decode_layers: %s", cudaGetErrorString(e));
  }
  return check_launch("decode_layers");
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
  return lin_smem_bytes(nt, di) <= 227 * 1024 && lin_smem_bytes(nt, hidden) <= 227 * 1024 &&
         mix_smem_bytes(M) <= 47 * 1024;
}

extern "C" size_t fracssm_decode_layers_workspace_bytes(int64_t B, int64_t hidden, int64_t H, int64_t R, int64_t M) {
  if (B < 1 || hidden < 1 || H < 1 || R < 1 || M < 1) return 0;
  return fracssm::scratch_layout(B, hidden, H * R, H, M).bytes;
}

extern "C" int fracssm_decode_layers(const uint64_t *layer_ptrs, const float *layer_nums, int64_t layers,
                                     const void *hidden_in, void *hidden_out, void *workspace, size_t workspace_bytes,
                                     int64_t B, int64_t hidden, int64_t H, int64_t R, int64_t M, int64_t K, void *stream) {
  using namespace fracssm;
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
  if (B <= 8) return run_layers<1>(layer_ptrs, layer_nums, layers, hidden_in, hidden_out, ws, B, hidden, H, R, M, st);
  if (B <= 16) return run_layers<2>(layer_ptrs, layer_nums, layers, hidden_in, hidden_out, ws, B, hidden, H, R, M, st);
  if (B <= 32) return run_layers<4>(layer_ptrs, layer_nums, layers, hidden_in, hidden_out, ws, B, hidden, H, R, M, st);
  return run_layers<8>(layer_ptrs, layer_nums, layers, hidden_in, hidden_out, ws, B, hidden, H, R, M, st);
}
