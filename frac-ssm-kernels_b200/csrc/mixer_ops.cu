// The two mixer steps next to the scan path that the reference runs in PyTorch:
//   * the causal depthwise convolution + SiLU that produces x_conv
//     (frac_ssm/models/modeling_frac.py:116-140, `_causal_conv_full`);
//   * the single-token state update of the decode loop
//     (frac_ssm/models/modeling_frac.py:159-179, `_update_state`, and the D skip of :236).
// Both are bandwidth kernels: every input element is read once, every output written once.
#include "common.cuh"
#include "prefill_dyn.cuh"
#include "scan_tile.cuh"

namespace fracssm {
namespace {

__device__ __forceinline__ float silu_(float x) { return x / (1.f + __expf(-x)); }

constexpr int kConvMaxK = 8;     // kernel widths 1..8
constexpr int kConvTokens = 32;  // tokens per thread: the window slides in registers

// General path: one channel per thread, any dtype.  grid (ceil(C/128), ceil(L/kConvTokens), B).
__global__ void __launch_bounds__(128)
causal_conv_silu_kernel(const void *__restrict__ x, int x_dt, int64_t x_sb, int64_t x_sl,
                        const float *__restrict__ mask, int64_t m_sb, int64_t m_sl,
                        const void *__restrict__ w, int w_dt, const void *__restrict__ bias, int K,
                        void *__restrict__ y, int y_dt, void *__restrict__ u_heads, int64_t R, int64_t L,
                        int64_t C) {
  const int64_t ch = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (ch >= C) return;
  const int64_t H = u_heads ? C / R : 0, hh = u_heads ? ch / R : 0, rr = u_heads ? ch % R : 0;
  const int64_t b = blockIdx.z, l0 = (int64_t)blockIdx.y * kConvTokens;
  float wk[kConvMaxK], win[kConvMaxK];
#pragma unroll
  for (int k = 0; k < kConvMaxK; ++k) wk[k] = k < K ? ld_f32(w, ch * K + k, w_dt) : 0.f;
  const float bv = bias ? ld_f32(bias, ch, w_dt) : 0.f;
  auto in = [&](int64_t l) -> float {
    if (l < 0) return 0.f;
    float v = ld_f32(x, b * x_sb + l * x_sl + ch, x_dt);
    if (mask) v *= mask[b * m_sb + l * m_sl];
    return v;
  };
  // win[k] pairs with wk[k]: win[K-1] is the current token, win[0] the oldest one
#pragma unroll
  for (int k = 0; k < kConvMaxK; ++k) win[k] = (k < K - 1) ? in(l0 - (K - 1) + k) : 0.f;
  const int64_t l1 = min(l0 + kConvTokens, L);
  for (int64_t l = l0; l < l1; ++l) {
    const float cur = in(l);
    float acc = bv;
#pragma unroll
    for (int k = 0; k < kConvMaxK; ++k) {
      if (k < K - 1) acc = fmaf(wk[k], win[k], acc);
      else if (k == K - 1) acc = fmaf(wk[k], cur, acc);
    }
    const float out = silu_(acc);
    st_f32(y, (b * L + l) * C + ch, y_dt, out);
    if (u_heads) st_f32(u_heads, ((b * H + hh) * L + l) * R + rr, y_dt, out);
#pragma unroll
    for (int k = 0; k < kConvMaxK - 1; ++k) {
      if (k < K - 2) win[k] = win[k + 1];
      else if (k == K - 2) win[k] = cur;
    }
  }
}

using tile::f2;
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// bf16 path for the usual width 4.
__device__ __forceinline__ void unpack8(const uint4 &p, float (&f)[8]) {
  const uint32_t wds[4] = {p.x, p.y, p.z, p.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(wds[i] << 16);
    f[2 * i + 1] = __uint_as_float(wds[i] & 0xFFFF0000u);
  }
}

// What the convolution of the next token needs: tail[b, ch, k] = the last K - 1 inputs times their mask (rounded to
// the input's type, like the product), zero before the first token.
struct ConvTail {
  __nv_bfloat16 *out;   // [B, C, K - 1], or null
  int K;
};
__device__ __forceinline__ void conv_tail(const __nv_bfloat16 *x, int64_t x_sb, int64_t x_sl, const float *mask, int64_t m_sb,
                                          int64_t m_sl, const ConvTail &tail, int64_t b, int64_t ch, int64_t L, int64_t C) {
  for (int k = 0; k < tail.K - 1; ++k) {
    const int64_t l = L - (tail.K - 1) + k;
    __nv_bfloat16 v = __float2bfloat16_rn(0.f);
    if (l >= 0) {
      v = x[b * x_sb + l * x_sl + ch];
      if (mask)
        v = __float2bfloat16_rn(__bfloat162float(v) * __bfloat162float(__float2bfloat16_rn(mask[b * m_sb + l * m_sl])));
    }
    tail.out[(b * C + ch) * (tail.K - 1) + k] = v;
  }
}
__global__ void __launch_bounds__(128)
conv_tail_kernel(const __nv_bfloat16 *__restrict__ x, int64_t x_sb, int64_t x_sl, const float *__restrict__ mask,
                 int64_t m_sb, int64_t m_sl, const ConvTail tail, int64_t L, int64_t C) {
  const int64_t ch = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (ch < C) conv_tail(x, x_sb, x_sl, mask, m_sb, m_sl, tail, blockIdx.y, ch, L, C);
}

// Four channels (8 bytes) per thread, TOKENS (32 at full size) tokens walked with the window in registers, the next
// four tokens requested before the current four are worked on.  Bound by the instructions a thread issues until its next
// request as much as by memory: with the channels as packed pairs and running addresses 16 x 4096 tokens x 1536
// channels take 109 us (125 with an fma per channel and 64-bit index products a token; 8 blocks of 128 threads per SM,
// 114 with 6), 4 x 1000 10.0 (11.6), 397 3.9 (4.4; 6 blocks, 8 are 12 % slower there).  Before: 0.154 ms with 16 tokens per
// thread and the loads of a group issued right before their use, 0.143 with 32 tokens (the three window tokens and the
// weights are read once per 32).  A short sequence is cut into runs of 16 or 8 tokens so that the grid covers the GPU.
// With TAIL, the last row of blocks writes it; at full size a launch of its own does, since that branch costs the kernel
// registers and 6 % of its time.
template <int TOKENS, bool TAIL>
__global__ void __launch_bounds__(128, TOKENS == kConvTokens ? 8 : 6)
causal_conv4_silu_bf16_kernel(const __nv_bfloat16 *__restrict__ x, int64_t x_sb, int64_t x_sl,
                              const float *__restrict__ mask, int64_t m_sb, int64_t m_sl,
                              const void *__restrict__ w, int w_dt, const void *__restrict__ bias,
                              __nv_bfloat16 *__restrict__ y, __nv_bfloat16 *__restrict__ u_heads, int64_t R,
                              int64_t L, int64_t C, const ConvTail tail) {
  const int64_t ch = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (ch >= C) return;
  if (TAIL && blockIdx.y == gridDim.y - 1) {
    for (int i = 0; i < 4; ++i) conv_tail(x, x_sb, x_sl, mask, m_sb, m_sl, tail, blockIdx.z, ch + i, L, C);
    return;
  }
  // the same four values also go to the head-major copy [Bt * H, L, R] (R a multiple of 4)
  __nv_bfloat16 *u_row = nullptr;
  if (u_heads) u_row = u_heads + ((int64_t)blockIdx.z * (C / R) + ch / R) * L * R + ch % R;
  const int64_t b = blockIdx.z, l0 = (int64_t)blockIdx.y * TOKENS;
  f2 wk[4][2], bv[2], w0[2], w1[2], w2[2];      // pairs of channels: half the multiply-adds
  if (w_dt == FRACSSM_BF16) {   // 4 channels x 4 taps = 32 contiguous bytes (ch is a multiple of 4)
    const uint4 *wp = reinterpret_cast<const uint4 *>(reinterpret_cast<const __nv_bfloat16 *>(w) + ch * 4);
#pragma unroll
    for (int q = 0; q < 2; ++q) {   // piece q holds channels 2q, 2q + 1
      float f[8];
      unpack8(__ldg(wp + q), f);
#pragma unroll
      for (int k = 0; k < 4; ++k) wk[k][q] = tile::mk2(f[k], f[4 + k]);
    }
  } else {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        wk[k][q] = tile::mk2(ld_f32(w, (ch + 2 * q) * 4 + k, w_dt), ld_f32(w, (ch + 2 * q + 1) * 4 + k, w_dt));
    }
  }
#pragma unroll
  for (int q = 0; q < 2; ++q)
    bv[q] = bias ? tile::mk2(ld_f32(bias, ch + 2 * q, w_dt), ld_f32(bias, ch + 2 * q + 1, w_dt)) : tile::mk2(0.f, 0.f);
  const __nv_bfloat16 *xp = x + b * x_sb + ch;
  const float *mp = mask ? mask + b * m_sb : nullptr;
  auto widen = [&](const uint2 &p, float m, f2 (&f)[2]) {
    f[0] = tile::mk2(__uint_as_float(p.x << 16), __uint_as_float(p.x & 0xFFFF0000u));
    f[1] = tile::mk2(__uint_as_float(p.y << 16), __uint_as_float(p.y & 0xFFFF0000u));
    if (mask) {
      f[0] = tile::mul2(f[0], tile::mk2(m, m));
      f[1] = tile::mul2(f[1], tile::mk2(m, m));
    }
  };
  auto in = [&](int64_t l, f2 (&f)[2]) {
    if (l < 0) {
      f[0] = f[1] = tile::mk2(0.f, 0.f);
      return;
    }
    widen(__ldcs(reinterpret_cast<const uint2 *>(xp + l * x_sl)), mask ? mp[l * m_sl] : 1.f, f);
  };
  in(l0 - 3, w0);
  in(l0 - 2, w1);
  in(l0 - 1, w2);
  const int n = (int)(min(l0 + TOKENS, L) - l0);
  xp += l0 * x_sl;
  if (mask) mp += l0 * m_sl;
  __nv_bfloat16 *yp = y + (b * L + l0) * C + ch;
  if (u_row) u_row += l0 * R;
  // the next four tokens are requested before the current four are worked on
  uint2 nraw[4];
  float nmk[4];
  auto request = [&](int g) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      nraw[j] = make_uint2(0u, 0u);
      nmk[j] = 1.f;
      if (g + j < n) {
        nraw[j] = __ldcs(reinterpret_cast<const uint2 *>(xp + j * x_sl));
        if (mask) nmk[j] = mp[j * m_sl];
      }
    }
    xp += 4 * x_sl;
    if (mask) mp += 4 * m_sl;
  };
  request(0);
  for (int g = 0; g < n; g += 4) {
    uint2 raw[4];
    float mk[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) { raw[j] = nraw[j]; mk[j] = nmk[j]; }
    if (g + 4 < n) request(g + 4);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (g + j < n) {
        f2 cur[2];
        widen(raw[j], mk[j], cur);
        uint32_t o[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          f2 acc = fma2(wk[0][i], w0[i], bv[i]);
          acc = fma2(wk[1][i], w1[i], acc);
          acc = fma2(wk[2][i], w2[i], acc);
          acc = fma2(wk[3][i], cur[i], acc);
          float r0, r1;
          tile::un2(acc, r0, r1);
          r0 = __fdividef(r0, 1.f + __expf(-r0));   // silu, about 2 ulp: the output is bf16
          r1 = __fdividef(r1, 1.f + __expf(-r1));
          const __nv_bfloat162 t = __floats2bfloat162_rn(r0, r1);
          o[i] = *reinterpret_cast<const uint32_t *>(&t);
          w0[i] = w1[i];
          w1[i] = w2[i];
          w2[i] = cur[i];
        }
        __stcs(reinterpret_cast<uint2 *>(yp), make_uint2(o[0], o[1]));
        if (u_row) {
          __stcs(reinterpret_cast<uint2 *>(u_row), make_uint2(o[0], o[1]));
          u_row += R;
        }
        yp += C;
      }
    }
  }
  // a grid that this one was started beside ends before this one does (else nothing to wait for)
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

// One token of the recurrence for every (batch, head): state [M, R] float32 updated in place,
//   state[m, r] = rho[m] * state[m, r] + kappa[m] * u[r];  out[r] = sum_m c[m] * state[m, r] + u[r] * D[r].
// One block per (batch, head); thread r-lane strides over R, the modes are walked in the block's
// y dimension and reduced through shared memory.
__global__ void __launch_bounds__(256)
decode_step_kernel(const void *__restrict__ u, int u_dt, const float *__restrict__ c,
                   const float *__restrict__ kappa, const float *__restrict__ rho,
                   const float *__restrict__ Dp, float *__restrict__ state, float *__restrict__ out,
                   int64_t H, int64_t R, int64_t M) {
  extern __shared__ float part[];  // [blockDim.y][R]
  const int64_t bh = blockIdx.x, h = bh % H;
  const int ty = threadIdx.y, ny = blockDim.y;
  float *st = state + bh * M * R;
  for (int64_t r = threadIdx.x; r < R; r += blockDim.x) {
    const float ur = ld_f32(u, bh * R + r, u_dt);
    float acc = 0.f;
    for (int64_t m = ty; m < M; m += ny) {
      const float s = fmaf(rho[bh * M + m], st[m * R + r], kappa[bh * M + m] * ur);
      st[m * R + r] = s;
      acc = fmaf(c[bh * M + m], s, acc);
    }
    part[ty * R + r] = acc;
  }
  __syncthreads();
  if (ty == 0) {
    for (int64_t r = threadIdx.x; r < R; r += blockDim.x) {
      float acc = 0.f;
      for (int y = 0; y < ny; ++y) acc += part[y * R + r];
      out[bh * R + r] = acc + ld_f32(u, bh * R + r, u_dt) * Dp[h * R + r];
    }
  }
}

}  // namespace
}  // namespace fracssm

extern "C" int fracssm_causal_conv_silu(const void *x, int x_dtype, int64_t x_sb, int64_t x_sl,
                                        const float *mask, int64_t m_sb, int64_t m_sl,
                                        const void *weight, const void *bias, int w_dtype, void *y,
                                        int y_dtype, int64_t Bt, int64_t L, int64_t C, int64_t K,
                                        void *stream) {
  return fracssm_causal_conv_silu_heads(x, x_dtype, x_sb, x_sl, mask, m_sb, m_sl, weight, bias, w_dtype, y, y_dtype,
                                        nullptr, 0, Bt, L, C, K, stream);
}

static int conv_silu_heads(const void *x, int x_dtype, int64_t x_sb, int64_t x_sl,
                                              const float *mask, int64_t m_sb, int64_t m_sl,
                                              const void *weight, const void *bias, int w_dtype, void *y,
                                              int y_dtype, void *u_heads, int64_t R, int64_t Bt, int64_t L,
                                              int64_t C, int64_t K, void *stream, const fracssm::ConvTail &tail,
                                              bool beside) {
  using namespace fracssm;
  if (u_heads && (R <= 0 || C % R != 0))
    return fail(FRACSSM_ERR_ARG, "causal_conv_silu: the head width must divide the channel count");
  if (Bt < 0 || L < 0 || C <= 0 || K < 1 || K > kConvMaxK) return fail(FRACSSM_ERR_ARG, "causal_conv_silu: bad sizes (kernel width 1..8)");
  if (!known_dtype(x_dtype) || !known_dtype(w_dtype) || !known_dtype(y_dtype))
    return fail(FRACSSM_ERR_ARG, "causal_conv_silu: unsupported dtype");
  if (Bt == 0 || L == 0) return FRACSSM_OK;
  if (!x || !weight || !y) return fail(FRACSSM_ERR_ARG, "causal_conv_silu: null pointer");
  if (Bt > 65535 || ceil_div(L, kConvTokens) > 65535)
    return fail(FRACSSM_ERR_UNSUPPORTED, "causal_conv_silu: batch or sequence too large for one launch");
  auto al16 = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  const dim3 block(128);
  if (K == 4 && x_dtype == FRACSSM_BF16 && y_dtype == FRACSSM_BF16 && C % 8 == 0 && al16(x) && al16(y) &&
      x_sb % 8 == 0 && x_sl % 8 == 0 && (!u_heads || (R % 8 == 0 && al16(u_heads))) &&
      (w_dtype != FRACSSM_BF16 || al16(weight))) {
    int tokens = kConvTokens;
    while (tokens > 8 && ceil_div(C / 4, 128) * ceil_div(L, tokens) * Bt < 148 * 4) tokens /= 2;
    if (ceil_div(L, tokens) > 65535) tokens = kConvTokens;
    const bool same_launch = tail.out && tokens < kConvTokens && ceil_div(L, tokens) < 65535;
    const dim3 grid((unsigned)ceil_div(C / 4, 128), (unsigned)(ceil_div(L, tokens) + (same_launch ? 1 : 0)), (unsigned)Bt);
    auto kernel = causal_conv4_silu_bf16_kernel<kConvTokens, false>;
    if (tokens == 16) kernel = same_launch ? causal_conv4_silu_bf16_kernel<16, true> : causal_conv4_silu_bf16_kernel<16, false>;
    if (tokens == 8) kernel = same_launch ? causal_conv4_silu_bf16_kernel<8, true> : causal_conv4_silu_bf16_kernel<8, false>;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = (cudaStream_t)stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = beside ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(
        &cfg, kernel, reinterpret_cast<const __nv_bfloat16 *>(x), x_sb, x_sl, mask, m_sb, m_sl, weight, w_dtype, bias,
        reinterpret_cast<__nv_bfloat16 *>(y), reinterpret_cast<__nv_bfloat16 *>(u_heads), R, L, C, tail);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(FRACSSM_ERR_CUDA, "causal_conv_silu: %s", cudaGetErrorString(e));
    }
    if (tail.out && !same_launch)
      conv_tail_kernel<<<dim3((unsigned)ceil_div(C, 128), (unsigned)Bt), 128, 0, (cudaStream_t)stream>>>(
          reinterpret_cast<const __nv_bfloat16 *>(x), x_sb, x_sl, mask, m_sb, m_sl, tail, L, C);
    return check_launch("causal_conv_silu");
  }
  const dim3 grid((unsigned)ceil_div(C, 128), (unsigned)ceil_div(L, kConvTokens), (unsigned)Bt);
  causal_conv_silu_kernel<<<grid, block, 0, (cudaStream_t)stream>>>(x, x_dtype, x_sb, x_sl, mask, m_sb, m_sl, weight,
                                                                 w_dtype, bias, (int)K, y, y_dtype, u_heads, R, L, C);
  if (tail.out)
    conv_tail_kernel<<<dim3((unsigned)ceil_div(C, 128), (unsigned)Bt), 128, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const __nv_bfloat16 *>(x), x_sb, x_sl, mask, m_sb, m_sl, tail, L, C);
  return check_launch("causal_conv_silu");
}

extern "C" int fracssm_causal_conv_silu_heads(const void *x, int x_dtype, int64_t x_sb, int64_t x_sl,
                                              const float *mask, int64_t m_sb, int64_t m_sl,
                                              const void *weight, const void *bias, int w_dtype, void *y,
                                              int y_dtype, void *u_heads, int64_t R, int64_t Bt, int64_t L,
                                              int64_t C, int64_t K, void *stream) {
  return conv_silu_heads(x, x_dtype, x_sb, x_sl, mask, m_sb, m_sl, weight, bias, w_dtype, y, y_dtype, u_heads, R, Bt, L, C, K,
                         stream, fracssm::ConvTail{nullptr, 0}, false);
}

extern "C" int fracssm_decode_step(const void *u, int u_dtype, const float *c, const float *kappa,
                                   const float *rho, const float *D, float *state, float *out,
                                   int64_t Bt, int64_t H, int64_t R, int64_t M, void *stream) {
  using namespace fracssm;
  if (Bt < 0 || H <= 0 || R <= 0 || M <= 0) return fail(FRACSSM_ERR_ARG, "decode_step: bad sizes");
  if (!known_dtype(u_dtype)) return fail(FRACSSM_ERR_ARG, "decode_step: unsupported dtype");
  if (Bt == 0) return FRACSSM_OK;
  if (!u || !c || !kappa || !rho || !D || !state || !out) return fail(FRACSSM_ERR_ARG, "decode_step: null pointer");
  int tx = 32;
  while (tx < R && tx < 256) tx *= 2;
  int ty = 256 / tx;
  if (ty > M) ty = (int)M;
  if (ty < 1) ty = 1;
  const size_t smem = (size_t)ty * R * sizeof(float);
  if (smem > 48 * 1024) return fail(FRACSSM_ERR_UNSUPPORTED, "decode_step: head_dim too large");
  decode_step_kernel<<<(unsigned)(Bt * H), dim3(tx, ty), smem, (cudaStream_t)stream>>>(u, u_dtype, c, kappa, rho, D,
                                                                                     state, out, H, R, M);
  return check_launch("decode_step");
}

extern "C" int fracssm_prefill_conv(const void *x, int64_t x_sl, const float *mask, const void *weight, const void *bias,
                                    void *y, void *u_heads, void *tail, int64_t R, int64_t Bt, int64_t L, int64_t C,
                                    int64_t K, void *stream) {
  // bf16 in and out
  const fracssm::ConvTail next{K >= 2 ? reinterpret_cast<__nv_bfloat16 *>(tail) : nullptr, (int)K};
  return conv_silu_heads(x, FRACSSM_BF16, L * x_sl, x_sl, mask, L, 1, weight, bias, FRACSSM_BF16, y, FRACSSM_BF16, u_heads, R,
                         Bt, L, C, K, stream, next, false);
}

extern "C" int fracssm_prefill_conv_dyn(const void *x, int64_t x_sl, const float *mask, const void *weight, const void *bias,
                                        void *y, void *u_heads, void *tail, const void *dyn_weight, void *dyn,
                                        int64_t dyn_cols, int64_t R, int64_t Bt, int64_t L, int64_t C, int64_t K,
                                        void *stream) {
  const int rc = fracssm::prefill_dyn_launch(x, x_sl, dyn_weight, dyn, Bt * L, C, dyn_cols, (cudaStream_t)stream);
  if (rc) return rc;
  const fracssm::ConvTail next{K >= 2 ? reinterpret_cast<__nv_bfloat16 *>(tail) : nullptr, (int)K};
  return conv_silu_heads(x, FRACSSM_BF16, L * x_sl, x_sl, mask, L, 1, weight, bias, FRACSSM_BF16, y, FRACSSM_BF16, u_heads, R,
                         Bt, L, C, K, stream, next, true);
}
