// The scan for shapes the single-pass tcgen05 kernel does not cover (up to 128 modes, any head width,
// any of the three dtypes, strided rows): the token recurrence itself, in float32,
//   S = rho (.) S + u kappa^T,   h = S c,
// with every row cut into segments so that few long rows fill the GPU too.
//
//   1. few_scan_kernel<.., false>: per segment but the last, the state it reaches from zero and the
//      product of its decays;
//   2. few_carry_kernel: the state that enters every segment (in place of the states of step 1);
//   3. few_scan_kernel<.., true>: every segment again from its true incoming state, writing h.
// Rows that are enough by themselves (see few_plan) take step 3 alone.
//
// What bounds it: the FMA pipe.  A state element costs a multiply and two fused multiply-adds per token
// (two instructions without the readout), so R * M = 2048 takes 48 cycles per token and SM in step 3.  The
// chunked stages this replaces spend an exponential per (t, k, m) of a chunk on top and keep the running
// log-decay, the chunk states and their prefix in memory.  A thread owns 4 columns of u and 8 or 16 modes
// (32 or 64 state elements in registers, worked on as packed pairs), which spreads the shared-memory
// reads of rho / kappa / c over four columns and leaves the other pipes to the conversions.  The inputs
// of the next two or three groups of 8 tokens are on their way into shared memory (cp.async) while a
// group is worked on.  Whole call, 2 rows x 32768 tokens, 128 columns, 16 modes, bfloat16: 328 us with the
// chunked stages, 80 us here.
#include "common.cuh"
#include "scan_tile.cuh"

namespace fracssm {
namespace {

using tile::f2;
using tile::mk2;
using tile::mul2;
using tile::un2;
using tile::widen_bf2;

__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

constexpr int kGroup = 8;      // tokens per stage
constexpr int kCols = 4;       // columns of u per thread
constexpr int kMaxBlockCols = 128;

struct Rows {                  // one input: base, strides in bytes, bytes of a row, bytes per copy (16, 8, 4 or 2)
  const char *p;
  int64_t sb, sl;
  int bytes, vec, shift;       // shift: log2 of the copies per row, or -1 when that is no power of two
};

struct FewArgs {
  Rows u, c, kappa, rho;
  int u_dt;
  const float *init;           // [B, R, M] or null
  void *h;                     // [B, L, R]
  int h_vec;                   // a thread's four columns go out in one store
  void *fin;                   // [B, R, M] or null
  int fin_dt;
  float *states;               // [B][nseg][R][Mp]
  float *decay;                // [B][nseg][Mp]
  int64_t L;
  int B, R, M, nseg, seg, block_cols;
};

__device__ __forceinline__ void copy_async(uint32_t dst, const char *src, int vec) {
  if (vec == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  else if (vec == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
  else if (vec == 4) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
  else {
    const unsigned short v = *reinterpret_cast<const unsigned short *>(src);
    asm volatile("st.shared.u16 [%0], %1;" ::"r"(dst), "h"(v) : "memory");
  }
}

// n tokens of one input (rows of `bytes` bytes starting at src, sl bytes apart) to shared memory
__device__ __forceinline__ void stage_rows(uint32_t dst, uint32_t tok_bytes, const char *src, int64_t sl, int bytes,
                                           int vec, int shift, int n) {
  const int per_row = bytes / vec;
  for (int i = threadIdx.x; i < n * per_row; i += blockDim.x) {
    const int t = shift >= 0 ? i >> shift : i / per_row, q = i - t * per_row;
    copy_async(dst + t * tok_bytes + q * vec, src + t * sl + q * vec, vec);
  }
}

// eight coefficients of one token as packed pairs
template <int CK>
__device__ __forceinline__ void ld8(const uint8_t *p, f2 (&v)[4]) {
  if constexpr (CK == FRACSSM_F32) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(p), b = *reinterpret_cast<const ulonglong2 *>(p + 16);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  } else {
    const uint4 a = *reinterpret_cast<const uint4 *>(p);
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if constexpr (CK == FRACSSM_BF16) {
        v[i] = widen_bf2(w[i]);
      } else {
        const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
        v[i] = mk2(f.x, f.y);
      }
    }
  }
}

// A block owns one segment of one row and block_cols columns of u.  Thread = (column lane, mode group):
// columns 4 cl .. 4 cl + 3, modes in blocks of 8: block j * G + g for j < MT / 8 (Mp = MT * G modes,
// zero-filled beyond M).
template <int MT, int G, int CK, bool READOUT>
__global__ void __launch_bounds__(32 * G) few_scan_kernel(const FewArgs a) {
  constexpr int Mp = MT * G, NB = MT / 8, kStages = Mp <= 32 ? 4 : 3;
  constexpr int kCk = CK == FRACSSM_F32 ? 4 : 2;
  constexpr uint32_t kOffK = Mp * 4, kOffC = kOffK + Mp * kCk, kOffU = kOffC + (READOUT ? Mp * kCk : 0);
  extern __shared__ __align__(16) uint8_t few_smem[];
  const int us = a.u_dt == FRACSSM_F32 ? 4 : 2;
  const uint32_t tok_bytes = kOffU + a.block_cols * us;   // a multiple of 16: block_cols is one of 8
  const uint32_t stage_bytes = kGroup * tok_bytes;
  const int64_t item = blockIdx.x;
  const int segs = READOUT ? a.nseg : a.nseg - 1;
  const int64_t b = item / segs;
  const int s = (int)(item - b * segs);
  const int col0 = blockIdx.y * a.block_cols, cols = min(a.block_cols, a.R - col0);
  const int64_t t0 = (int64_t)s * a.seg;
  const int ntok = (int)min((int64_t)a.seg, a.L - t0);
  const int g = threadIdx.x % G, cl = threadIdx.x / G;
  const bool live = cl * kCols < cols;
  const int my = live ? cl * kCols : 0;    // idle lanes compute along on column 0 and store nothing
  const uint32_t smem_base = (uint32_t)__cvta_generic_to_shared(few_smem);

  if (a.M < Mp || cols % kCols != 0) {   // modes and columns beyond the end count as zeros
    for (uint32_t i = threadIdx.x * 4; i < kStages * stage_bytes; i += blockDim.x * 4)
      *reinterpret_cast<uint32_t *>(few_smem + i) = 0u;
    __syncthreads();
  }
  const char *rho_p = a.rho.p + b * a.rho.sb + t0 * a.rho.sl, *kap_p = a.kappa.p + b * a.kappa.sb + t0 * a.kappa.sl;
  const char *c_p = a.c.p + b * a.c.sb + t0 * a.c.sl, *u_p = a.u.p + b * a.u.sb + t0 * a.u.sl + (int64_t)col0 * us;
  const int u_bytes = cols * us;
  const int u_shift = cols == a.block_cols ? a.u.shift : -1;
  const int groups = (ntok + kGroup - 1) / kGroup;
  auto request = [&](int ib) {
    if (ib < groups) {
      const int64_t t = (int64_t)ib * kGroup;
      const int n = min(kGroup, ntok - ib * kGroup);
      const uint32_t dst = smem_base + (ib % kStages) * stage_bytes;
      stage_rows(dst, tok_bytes, rho_p + t * a.rho.sl, a.rho.sl, a.rho.bytes, a.rho.vec, a.rho.shift, n);
      stage_rows(dst + kOffK, tok_bytes, kap_p + t * a.kappa.sl, a.kappa.sl, a.kappa.bytes, a.kappa.vec, a.kappa.shift, n);
      if (READOUT)
        stage_rows(dst + kOffC, tok_bytes, c_p + t * a.c.sl, a.c.sl, a.c.bytes, a.c.vec, a.c.shift, n);
      stage_rows(dst + kOffU, tok_bytes, u_p + t * a.u.sl, a.u.sl, u_bytes, a.u.vec, u_shift, n);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) request(i);

  f2 st[kCols][NB * 4];
  f2 prod[NB * 4];
#pragma unroll
  for (int r = 0; r < kCols; ++r)
#pragma unroll
    for (int p = 0; p < NB * 4; ++p) st[r][p] = mk2(0.f, 0.f);
#pragma unroll
  for (int p = 0; p < NB * 4; ++p) prod[p] = mk2(1.f, 1.f);
  const int nr = live ? min(kCols, cols - my) : 0;   // columns this thread really owns
  if (READOUT && (s > 0 || a.init)) {
    // (compile-time indexes into the state: it lives in registers)
#pragma unroll
    for (int r = 0; r < kCols; ++r) {
      if (r < nr) {
        if (s > 0) {
          const float *src = a.states + (((int64_t)b * a.nseg + s) * a.R + col0 + my + r) * Mp;
#pragma unroll
          for (int j = 0; j < NB; ++j) {
            const ulonglong2 x = __ldcg(reinterpret_cast<const ulonglong2 *>(src + 8 * (j * G + g)));
            const ulonglong2 y = __ldcg(reinterpret_cast<const ulonglong2 *>(src + 8 * (j * G + g) + 4));
            st[r][4 * j] = x.x; st[r][4 * j + 1] = x.y; st[r][4 * j + 2] = y.x; st[r][4 * j + 3] = y.y;
          }
        } else {
          const float *src = a.init + ((int64_t)b * a.R + col0 + my + r) * a.M;
#pragma unroll
          for (int p = 0; p < NB * 4; ++p) {
            const int m = 8 * ((p / 4) * G + g) + 2 * (p % 4);
            st[r][p] = mk2(m < a.M ? src[m] : 0.f, m + 1 < a.M ? src[m + 1] : 0.f);
          }
        }
      }
    }
  }

  for (int ib = 0; ib < groups; ++ib) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();
    request(ib + kStages - 1);   // into the stage that was used up before this barrier
    const uint8_t *stage = few_smem + (ib % kStages) * stage_bytes;
    const int n = min(kGroup, ntok - ib * kGroup);
#pragma unroll 2
    for (int t = 0; t < n; ++t) {
      const uint8_t *tok = stage + t * tok_bytes;
      f2 uu[kCols], acc[kCols];
      {
        float uf[kCols];
        if (a.u_dt == FRACSSM_F32) {
          const float2 lo = *reinterpret_cast<const float2 *>(tok + kOffU + my * 4);
          const float2 hi = *reinterpret_cast<const float2 *>(tok + kOffU + my * 4 + 8);
          uf[0] = lo.x; uf[1] = lo.y; uf[2] = hi.x; uf[3] = hi.y;
        } else {
          const uint2 w = *reinterpret_cast<const uint2 *>(tok + kOffU + my * 2);
          if (a.u_dt == FRACSSM_BF16) {
            un2(widen_bf2(w.x), uf[0], uf[1]);
            un2(widen_bf2(w.y), uf[2], uf[3]);
          } else {
            const float2 lo = __half22float2(*reinterpret_cast<const __half2 *>(&w.x));
            const float2 hi = __half22float2(*reinterpret_cast<const __half2 *>(&w.y));
            uf[0] = lo.x; uf[1] = lo.y; uf[2] = hi.x; uf[3] = hi.y;
          }
        }
#pragma unroll
        for (int r = 0; r < kCols; ++r) { uu[r] = mk2(uf[r], uf[r]); acc[r] = mk2(0.f, 0.f); }
      }
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const int blk = j * G + g;
        f2 rh[4], ka[4], cc[4];
        ld8<FRACSSM_F32>(tok + blk * 32, rh);
        ld8<CK>(tok + kOffK + blk * 8 * kCk, ka);
        if (READOUT) ld8<CK>(tok + kOffC + blk * 8 * kCk, cc);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          float lo, hi;
          un2(rh[p], lo, hi);
          const f2 rr = mk2(fmaxf(lo, kRhoFloor), fmaxf(hi, kRhoFloor));
          if (!READOUT) prod[4 * j + p] = mul2(prod[4 * j + p], rr);
#pragma unroll
          for (int r = 0; r < kCols; ++r) {
            st[r][4 * j + p] = fma2(rr, st[r][4 * j + p], mul2(ka[p], uu[r]));
            if (READOUT) acc[r] = fma2(cc[p], st[r][4 * j + p], acc[r]);
          }
        }
      }
      if (READOUT) {
        float o[kCols];
#pragma unroll
        for (int r = 0; r < kCols; ++r) {
          float lo, hi;
          un2(acc[r], lo, hi);
          o[r] = lo + hi;
        }
        const int64_t row = ((int64_t)b * a.L + t0 + (int64_t)ib * kGroup + t) * a.R + col0 + my;
        if constexpr (G == 1) {
          if (a.h_vec && nr == kCols) {
            if (a.u_dt == FRACSSM_F32) {
              *reinterpret_cast<float4 *>(reinterpret_cast<float *>(a.h) + row) = make_float4(o[0], o[1], o[2], o[3]);
            } else if (a.u_dt == FRACSSM_BF16) {
              *reinterpret_cast<uint2 *>(reinterpret_cast<__nv_bfloat16 *>(a.h) + row) =
                  make_uint2(tile::pack2(o[0], o[1]), tile::pack2(o[2], o[3]));
            } else {
              const __half2 p0 = __floats2half2_rn(o[0], o[1]), p1 = __floats2half2_rn(o[2], o[3]);
              *reinterpret_cast<uint2 *>(reinterpret_cast<__half *>(a.h) + row) =
                  make_uint2(*reinterpret_cast<const uint32_t *>(&p0), *reinterpret_cast<const uint32_t *>(&p1));
            }
          } else {
#pragma unroll
            for (int r = 0; r < kCols; ++r)
              if (r < nr) st_f32(a.h, row + r, a.u_dt, o[r]);
          }
        } else {
          // sum over the mode groups; each step halves the columns a lane answers for
          const bool odd = g & 1;
          float x0 = __shfl_xor_sync(0xffffffffu, odd ? o[0] : o[2], 1);
          float x1 = __shfl_xor_sync(0xffffffffu, odd ? o[1] : o[3], 1);
          x0 += odd ? o[2] : o[0];
          x1 += odd ? o[3] : o[1];
          const int r0 = odd ? 2 : 0;
          if constexpr (G == 2) {
            if (r0 < nr) st_f32(a.h, row + r0, a.u_dt, x0);
            if (r0 + 1 < nr) st_f32(a.h, row + r0 + 1, a.u_dt, x1);
          } else {
            const bool up = g & 2;
            float y = __shfl_xor_sync(0xffffffffu, up ? x0 : x1, 2);
            y += up ? x1 : x0;
            if constexpr (G == 8) y += __shfl_xor_sync(0xffffffffu, y, 4);
            const int r = r0 + (up ? 1 : 0);
            if (g < 4 && r < nr) st_f32(a.h, row + r, a.u_dt, y);
          }
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");

  if (!READOUT) {
#pragma unroll
    for (int r = 0; r < kCols; ++r) {
      if (r < nr) {
        float *dst = a.states + (((int64_t)b * a.nseg + s) * a.R + col0 + my + r) * Mp;
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          __stcg(reinterpret_cast<ulonglong2 *>(dst + 8 * (j * G + g)), make_ulonglong2(st[r][4 * j], st[r][4 * j + 1]));
          __stcg(reinterpret_cast<ulonglong2 *>(dst + 8 * (j * G + g) + 4),
                 make_ulonglong2(st[r][4 * j + 2], st[r][4 * j + 3]));
        }
      }
    }
    if (cl == 0 && blockIdx.y == 0) {
      float *dst = a.decay + ((int64_t)b * a.nseg + s) * Mp;
#pragma unroll
      for (int p = 0; p < NB * 4; ++p)
        *reinterpret_cast<f2 *>(dst + 8 * ((p / 4) * G + g) + 2 * (p % 4)) = prod[p];
    }
  } else if (a.fin && s == a.nseg - 1) {
#pragma unroll
    for (int r = 0; r < kCols; ++r) {
      if (r < nr) {
        const int64_t dst = ((int64_t)b * a.R + col0 + my + r) * a.M;
#pragma unroll
        for (int p = 0; p < NB * 4; ++p) {
          const int m = 8 * ((p / 4) * G + g) + 2 * (p % 4);
          float lo, hi;
          un2(st[r][p], lo, hi);
          if (m < a.M) st_f32(a.fin, dst + m, a.fin_dt, lo);
          if (m + 1 < a.M) st_f32(a.fin, dst + m + 1, a.fin_dt, hi);
        }
      }
    }
  }
}

// states[b][s] := the state entering segment s.  A block owns 32 elements of a row's state; its 16 warps
// split the segments (each first composes its own share, so the serial chain is nseg / 16 long twice).
constexpr int kCarryWarps = 16, kCarryBatch = 8;
__global__ void __launch_bounds__(32 * kCarryWarps)
few_carry_kernel(float *__restrict__ states, const float *__restrict__ decay, const float *__restrict__ init,
                 int nseg, int R, int M, int Mp) {
  __shared__ float ps[kCarryWarps][32], ss[kCarryWarps][32];
  const int lane = threadIdx.x % 32, w = threadIdx.x / 32;
  const int64_t b = blockIdx.y, RM = (int64_t)R * Mp;
  const int64_t e = (int64_t)blockIdx.x * 32 + lane;
  const bool live = e < RM;
  const int r = live ? (int)(e / Mp) : 0, m = live ? (int)(e % Mp) : 0;
  float *sp = states + b * nseg * RM + (live ? e : 0);
  const float *dp = decay + b * nseg * Mp + m;
  const int share = (nseg + kCarryWarps - 1) / kCarryWarps;
  const int lo = min(w * share, nseg), hi = min(lo + share, nseg), last = nseg - 1;   // segment `last` has no summary
  float p = 1.f, v = 0.f;
  for (int s0 = lo; s0 < hi; s0 += kCarryBatch) {
    float x[kCarryBatch], d[kCarryBatch];
#pragma unroll
    for (int i = 0; i < kCarryBatch; ++i) {
      const bool on = s0 + i < hi && s0 + i < last;
      x[i] = on ? __ldcg(sp + (s0 + i) * RM) : 0.f;
      d[i] = on ? __ldcg(dp + (int64_t)(s0 + i) * Mp) : 1.f;
    }
#pragma unroll
    for (int i = 0; i < kCarryBatch; ++i) {
      v = fmaf(d[i], v, x[i]);
      p *= d[i];
    }
  }
  ps[w][lane] = p;
  ss[w][lane] = v;
  __syncthreads();
  if (!live) return;
  float run = init && m < M ? init[(b * R + r) * M + m] : 0.f;
  for (int i = 0; i < w; ++i) run = fmaf(ps[i][lane], run, ss[i][lane]);
  for (int s0 = lo; s0 < hi; s0 += kCarryBatch) {
    float x[kCarryBatch], d[kCarryBatch];
#pragma unroll
    for (int i = 0; i < kCarryBatch; ++i) {
      const bool on = s0 + i < hi && s0 + i < last;
      x[i] = on ? __ldcg(sp + (s0 + i) * RM) : 0.f;
      d[i] = on ? __ldcg(dp + (int64_t)(s0 + i) * Mp) : 1.f;
    }
#pragma unroll
    for (int i = 0; i < kCarryBatch; ++i) {
      if (s0 + i < hi) __stcg(sp + (s0 + i) * RM, run);
      run = fmaf(d[i], run, x[i]);
    }
  }
}

struct FewPlan {
  int MT, G, Mp, block_cols, col_blocks, seg, nseg;
  size_t bytes;
};

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

FewPlan few_plan(int64_t B, int64_t L, int64_t R, int64_t M) {
  FewPlan p{};
  p.MT = M <= 32 ? 8 : 16;
  p.G = M <= 8 ? 1 : M <= 16 ? 2 : M <= 64 ? 4 : 8;
  p.Mp = p.MT * p.G;
  p.col_blocks = (int)ceil_div(R, kMaxBlockCols);
  p.block_cols = (int)ceil_div(ceil_div(R, p.col_blocks), 8) * 8;
  // Warps a row keeps busy by itself.  From 8 warps per SM on the rows alone are enough (the cut costs a
  // second read of u, kappa and rho and two thirds more arithmetic); below, segments of at least 32
  // tokens such that about 16 warps per SM run.
  const int64_t row_warps = p.col_blocks * ceil_div(ceil_div(p.block_cols, kCols) * p.G, 32);
  int64_t nseg = 1;
  if (B * row_warps < 148 * 8) nseg = ceil_div(148 * 16, B * row_warps);
  int64_t seg = ceil_div(ceil_div(L, nseg), kGroup) * kGroup;
  if (seg < 32) seg = 32;
  p.seg = (int)(seg < L ? seg : L);
  p.nseg = (int)ceil_div(L, p.seg);
  if (p.nseg > 1)
    p.bytes = align256((size_t)B * p.nseg * R * p.Mp * 4) + align256((size_t)B * p.nseg * p.Mp * 4);
  return p;
}

Rows make_rows(const void *p, int64_t sb, int64_t sl, int64_t n, int esize, int64_t block_cols) {
  Rows r{};
  r.p = reinterpret_cast<const char *>(p);
  r.sb = sb * esize;
  r.sl = sl * esize;
  r.bytes = (int)(n * esize);
  // the widest copy that the base, both strides, the row and a block's share of it allow
  const uint64_t bits = (uint64_t)(uintptr_t)p | (uint64_t)r.sb | (uint64_t)r.sl | (uint64_t)r.bytes |
                        (uint64_t)(block_cols * esize);
  r.vec = bits % 16 == 0 ? 16 : bits % 8 == 0 ? 8 : bits % 4 == 0 ? 4 : 2;
  const int64_t per = (block_cols < n ? block_cols : n) * esize / r.vec;
  r.shift = -1;
  for (int s = 0; s < 16; ++s)
    if ((int64_t(1) << s) == per) r.shift = s;
  return r;
}

template <int MT, int G, int CK>
int few_launch(const FewArgs &a, const FewPlan &p, cudaStream_t st) {
  const int us = a.u_dt == FRACSSM_F32 ? 4 : 2;
  constexpr int kCk = CK == FRACSSM_F32 ? 4 : 2, Mp = MT * G, kStages = Mp <= 32 ? 4 : 3;
  const int threads = (int)(ceil_div(ceil_div(p.block_cols, kCols) * G, 32) * 32);
  const size_t sum_smem = (size_t)kStages * kGroup * (Mp * 4 + Mp * kCk + p.block_cols * us);
  const size_t out_smem = sum_smem + (size_t)kStages * kGroup * Mp * kCk;
  if (out_smem > 48 * 1024) return fail(FRACSSM_ERR_UNSUPPORTED, "frac_scan: shared memory of the segment kernel");
  if (p.nseg > 1) {
    few_scan_kernel<MT, G, CK, false>
        <<<dim3((unsigned)((int64_t)a.B * (p.nseg - 1)), p.col_blocks), threads, sum_smem, st>>>(a);
    few_carry_kernel<<<dim3((unsigned)ceil_div((int64_t)a.R * Mp, 32), (unsigned)a.B), 32 * kCarryWarps, 0, st>>>(
        a.states, a.decay, a.init, p.nseg, a.R, a.M, Mp);
  }
  few_scan_kernel<MT, G, CK, true><<<dim3((unsigned)((int64_t)a.B * p.nseg), p.col_blocks), threads, out_smem, st>>>(a);
  return check_launch("frac_scan (segment kernels)");
}

template <int CK>
int few_launch_modes(const FewArgs &a, const FewPlan &p, cudaStream_t st) {
  if (p.Mp == 8) return few_launch<8, 1, CK>(a, p, st);
  if (p.Mp == 16) return few_launch<8, 2, CK>(a, p, st);
  if (p.Mp == 32) return few_launch<8, 4, CK>(a, p, st);
  if (p.Mp == 64) return few_launch<16, 4, CK>(a, p, st);
  return few_launch<16, 8, CK>(a, p, st);
}

}  // namespace

// Up to 128 modes the state of 4 columns fits the registers of at most 8 threads; beyond, the chunked
// stages stay.  The other limits are those of the chunked stages (a launch's grid).
bool scan_few_supported(int64_t B, int64_t L, int64_t R, int64_t M, int64_t T) {
  if (B < 1 || L < 1 || R < 1 || M < 1 || M > 128 || R > 65535 || B > 65535 || L >= (int64_t(1) << 30)) return false;
  if (ceil_div(L, T) > 65535) return false;
  const FewPlan p = few_plan(B, L, R, M);
  return B * p.nseg < (int64_t(1) << 31);
}

size_t scan_few_workspace_bytes(int64_t B, int64_t L, int64_t R, int64_t M) { return few_plan(B, L, R, M).bytes; }

int scan_few_launch(const void *u, int u_dtype, int64_t u_sb, int64_t u_sl, const void *c, const void *kappa,
                    int ck_dtype, int64_t c_sb, int64_t c_sl, int64_t k_sb, int64_t k_sl, const float *rho,
                    int64_t r_sb, int64_t r_sl, const float *initial_state, void *h, void *final_state,
                    int final_dtype, void *workspace, int64_t B, int64_t L, int64_t R, int64_t M, void *stream) {
  const FewPlan p = few_plan(B, L, R, M);
  FewArgs a{};
  const int us = (int)dtype_size(u_dtype), ks = (int)dtype_size(ck_dtype);
  a.u = make_rows(u, u_sb, u_sl, R, us, p.block_cols);
  a.c = make_rows(c, c_sb, c_sl, M, ks, M);
  a.kappa = make_rows(kappa, k_sb, k_sl, M, ks, M);
  a.rho = make_rows(rho, r_sb, r_sl, M, 4, M);
  a.u_dt = u_dtype;
  a.init = initial_state;
  a.h = h;
  a.h_vec = R % 4 == 0 && (reinterpret_cast<uintptr_t>(h) & 15) == 0;
  a.fin = final_state;
  a.fin_dt = final_dtype;
  a.states = reinterpret_cast<float *>(workspace);
  a.decay = reinterpret_cast<float *>(reinterpret_cast<char *>(workspace) + align256((size_t)B * p.nseg * R * p.Mp * 4));
  a.L = L;
  a.B = (int)B;
  a.R = (int)R;
  a.M = (int)M;
  a.nseg = p.nseg;
  a.seg = p.seg;
  a.block_cols = p.block_cols;
  const cudaStream_t st = (cudaStream_t)stream;
  if (ck_dtype == FRACSSM_F32) return few_launch_modes<FRACSSM_F32>(a, p, st);
  if (ck_dtype == FRACSSM_BF16) return few_launch_modes<FRACSSM_BF16>(a, p, st);
  return few_launch_modes<FRACSSM_F16>(a, p, st);
}

}  // namespace fracssm
