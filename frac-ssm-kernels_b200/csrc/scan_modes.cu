// The scan for shapes the single-pass tcgen05 kernel does not cover (up to 128 modes, any head width,
// any of the three dtypes, strided rows): the token recurrence itself, in float32,
//   S = rho (.) S + u kappa^T,   h = S c,
// with every row cut into segments so that few long rows fill the GPU too.
//
//   1. few_scan_kernel<.., false, ..>: per segment but the last, the state it reaches from zero and the
//      product of its decays;
//   2. few_carry_kernel: the state that enters every segment (in place of the states of step 1);
//   3. few_scan_kernel<.., true, ..>:  every segment again from its true incoming state, writing h.
// Rows that are enough by themselves (see few_plan) take step 3 alone.
//
// What bounds it: instruction issue, half of it the FMA pipe.  A state element costs a multiply and two
// fused multiply-adds per token in step 3, one fused multiply-add and an eighth of a multiply in step 1: there kappa is
// multiplied with the decay behind its token within a group of 8 first, once for all columns (22 us as the recurrence, 16
// so).  Elements are worked on as packed pairs; a thread
// owns 4 columns of u and 8 modes (32 elements), so that registers leave room for 16 warps per SM.  (8 columns
// need fewer instructions in all, but 160 registers: 2.5 warps per scheduler, and the whole was slower.)
// What is not arithmetic is kept small: a group of 8 tokens is requested a group ahead into registers, widened
// to float32 once per block and read from shared memory by all its threads; with cp.async and the conversions in every
// thread a token took 188 instructions a warp.  (Calls whose rows do not load in 16-byte pieces request a group when it
// is due; large ones among them are left to the chunked stages, see few_narrow_limit.)
// Whole call, 2 rows x 32768 tokens, 128 columns, 16 modes, bfloat16: 328 us with the chunked stages, 80 us
// with the first form of these kernels, 62 us with a recurrence in step 1 too, 52 us here.
#include <type_traits>

#include "common.cuh"
#include "scan_tile.cuh"

namespace fracssm {
namespace {

using tile::f2;
using tile::mk2;
using tile::mul2;
using tile::un2;

__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

constexpr int kGroup = 8;      // tokens per group
constexpr int kCols = 4;       // columns of u per thread
constexpr int kModes = 8;      // modes per thread
constexpr int kMaxBlockCols = 128;
constexpr int kTokPad = 4;     // floats between a token's values and the next token's in the summary
// Least decay over several tokens, of a group, a segment or a share of the carry: a product of 7 decays of 1e-6 underflows, and
// zero times an infinity (of u, or of the state) would be NaN where the recurrence, whose single decays are no less than 1e-6,
// keeps the infinity.  What has decayed further stays at 1e-37 of its size.  Behind a token within its group the least is larger,
// so that a kappa down to 2e-15 times it is not zero either: 1e-30 |kappa u| too much in a state.
constexpr float kLeastDecay = 1e-37f, kLeastBehind = 1e-30f;

struct Rows {                  // one input: base and strides in bytes
  const char *p;
  int64_t sb, sl;
};

Rows few_rows(const void *p, int64_t sb, int64_t sl, int size) {
  return Rows{reinterpret_cast<const char *>(p), sb * size, sl * size};
}

struct FewArgs {
  Rows u, c, kappa, rho;
  const float *init;           // [B, R, M] or null
  void *h;                     // [B, L, R]
  int h_vec;                   // R a multiple of 4 and h 16-byte aligned: a lane's columns go out in one store
  void *fin;                   // [B, R, M] (or [B, M, R], by the strides) or null
  int fin_dt, fin_sr, fin_sm;
  float *states;               // [B][nseg][R][Mp]
  float *decay;                // [B][nseg][Mp]
  int64_t L;
  int B, R, M, nseg, seg, block_cols, lanes, per_block;   // lanes: threads of a segment; per_block: segments of a block
  int wide_loads, u_shift;     // 16-byte loads apply (see few_launch); log2 of u's 16-byte pieces per token
};

__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <int DT>
__device__ __forceinline__ void widen(const uint4 &raw, float (&f)[DT == FRACSSM_F32 ? 4 : 8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (DT == FRACSSM_F32) {
      f[i] = __uint_as_float(w[i]);
    } else if constexpr (DT == FRACSSM_BF16) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    } else {
      const float2 v = __half22float2(*reinterpret_cast<const __half2 *>(&w[i]));
      f[2 * i] = v.x;
      f[2 * i + 1] = v.y;
    }
  }
}

// four coefficients of a token: 16 bytes of float32, 8 of the 16-bit types
template <int DT>
__device__ __forceinline__ void widen4(const uint4 &raw, float (&f)[4]) {
  widen<FRACSSM_F32>(raw, f);
}
template <int DT>
__device__ __forceinline__ void widen4(const uint2 &raw, float (&f)[4]) {
  float g[8];
  widen<DT == FRACSSM_F16 ? FRACSSM_F16 : FRACSSM_BF16>(make_uint4(raw.x, raw.y, 0u, 0u), g);
#pragma unroll
  for (int i = 0; i < 4; ++i) f[i] = g[i];
}

__device__ __forceinline__ void ld_pairs(const float *p, f2 (&v)[4]) {   // eight floats
  const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(p), b = *reinterpret_cast<const ulonglong2 *>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// Room for two groups lets one be stored while the slower warps still read the one before.  A readout of 4 and more warps a
// segment is faster with one (400 rows x 2000 tokens, 64 columns x 64 modes, float32: 0.85 ms against 0.95; 400 x 2000,
// 128 x 16, bfloat16: 0.52 against 0.51 with two), and so is one of a warp or less, which needs no barrier to speak of (12 x
// 400, 128 x 8: 12.5 against 18.3 us for the three launches).
__host__ __device__ constexpr int few_buffers(int G, bool readout) { return readout && (G == 1 || G >= 8) ? 1 : 2; }

// `lanes` threads work on one segment of one row and block_cols columns of u: thread = (column lane, mode group),
// columns 4 cl .. 4 cl + 3, modes 8 g .. 8 g + 7 (Mp = 8 G modes, zeros beyond M).  Segments that need less than a
// warp share one.
// PADDED: M < Mp (as a branch of one kernel the care for the padding modes cost the others 2 %).
template <int G, int UD, int CK, bool READOUT, bool PADDED>
__global__ void __launch_bounds__(32 * G, G == 1 ? 16 : G == 2 ? 8 : G == 4 ? 4 : G == 8 ? 2 : 1)
few_scan_kernel(const FewArgs a) {
  constexpr int Mp = kModes * G;
  constexpr int kUs = UD == FRACSSM_F32 ? 4 : 2, kCk = CK == FRACSSM_F32 ? 4 : 2;
  constexpr int kOffK = Mp, kOffC = 2 * Mp, kOffU = READOUT ? 3 * Mp : 2 * Mp;   // a widened token, in floats
  constexpr int kBuffers = few_buffers(G, READOUT);
  constexpr int kPieces = kGroup * Mp / 4;                   // of four modes, of a group of tokens
  constexpr int kUMax = (2 * kUs + G - 1) / G;               // pieces of u per thread and group
  extern __shared__ __align__(16) float few_smem[];
  const int lanes = a.lanes, sub = threadIdx.x / lanes, lane = threadIdx.x - sub * lanes;
  const int tok_floats = kOffU + a.block_cols + (READOUT ? 0 : kTokPad), buf_floats = a.per_block * kGroup * tok_floats;
  // (threads beyond the last segment idle along)
  float *wide = few_smem + min(sub, a.per_block - 1) * kGroup * tok_floats;
  const int segs = READOUT ? a.nseg : a.nseg - 1;
  const int64_t items = (int64_t)a.B * segs, item = (int64_t)blockIdx.x * a.per_block + sub;
  const bool owner = sub < a.per_block && item < items;
  const int64_t b = owner ? item / segs : 0;
  const int s = owner ? (int)(item - b * segs) : 0;
  const int col0 = blockIdx.y * a.block_cols, cols = min(a.block_cols, a.R - col0);
  const int64_t t0 = (int64_t)s * a.seg;
  const int ntok = owner ? (int)min((int64_t)a.seg, a.L - t0) : 0;
  // Tokens of the block's longest segment: all its threads take this many steps, those without a token idle along
  // (the shuffles and barriers below are for whole warps and the whole block).
  const int all_tok = a.per_block > 1 ? a.seg
                                      : (int)min((int64_t)a.seg, a.L - (int64_t)(blockIdx.x % (unsigned)segs) * a.seg);
  const int g = lane % G, cl = lane / G;
  const bool live = owner && cl * kCols < cols;
  const int my = cl * kCols < cols ? cl * kCols : 0;   // idle lanes compute along on column 0 and store nothing
  const int nr = live ? min(kCols, cols - my) : 0;     // columns this thread really owns
  grid_dep_launch();

  const char *rho_p = a.rho.p + b * a.rho.sb + t0 * a.rho.sl, *kap_p = a.kappa.p + b * a.kappa.sb + t0 * a.kappa.sl;
  const char *c_p = a.c.p + b * a.c.sb + t0 * a.c.sl, *u_p = a.u.p + b * a.u.sb + t0 * a.u.sl + (int64_t)col0 * kUs;

  // ---- a group's raw inputs in registers: four modes of rho, kappa and c of a token per thread, and some pieces of u.  In the
  // summary the 8 tokens of a piece lie in neighbouring lanes (kTokPad keeps their stores apart), in the readout the pieces of a
  // token.
  using CkRaw = typename std::conditional<kCk == 4, uint4, uint2>::type;
  uint4 q_rho, q_u[kUMax];
  CkRaw q_kap, q_c;
  const int rt = READOUT ? lane / (Mp / 4) : lane % kGroup, rq = READOUT ? lane % (Mp / 4) : lane / kGroup;
  const bool owns = lane < kPieces;
  auto request = [&](int ib) {
    const int n = min(kGroup, ntok - ib * kGroup);
    const int64_t t = (int64_t)ib * kGroup;
    if (owns && rt < n) {
      q_rho = __ldg(reinterpret_cast<const uint4 *>(rho_p + (t + rt) * a.rho.sl) + rq);
      q_kap = __ldg(reinterpret_cast<const CkRaw *>(kap_p + (t + rt) * a.kappa.sl) + rq);
      if (READOUT) q_c = __ldg(reinterpret_cast<const CkRaw *>(c_p + (t + rt) * a.c.sl) + rq);
    }
#pragma unroll
    for (int i = 0; i < kUMax; ++i) {
      const int at = lane + i * lanes, ut = at >> a.u_shift, uq = at - (ut << a.u_shift);
      if (ut < n) q_u[i] = __ldg(reinterpret_cast<const uint4 *>(u_p + (t + ut) * a.u.sl) + uq);
    }
  };
  auto store_group = [&](int ib, float *to) {
    const int n = min(kGroup, ntok - ib * kGroup);
    const bool mine = owns && rt < n;
    float *d = to + rt * tok_floats + 4 * rq;
    if (READOUT) {
      if (mine) {
        float r[4], f[4];
        widen<FRACSSM_F32>(q_rho, r);
        *reinterpret_cast<float4 *>(d) = make_float4(fmaxf(r[0], kRhoFloor), fmaxf(r[1], kRhoFloor), fmaxf(r[2], kRhoFloor), fmaxf(r[3], kRhoFloor));
        widen4<CK>(q_kap, f);
        *reinterpret_cast<float4 *>(d + kOffK) = make_float4(f[0], f[1], f[2], f[3]);
        widen4<CK>(q_c, f);
        *reinterpret_cast<float4 *>(d + kOffC) = make_float4(f[0], f[1], f[2], f[3]);
      }
    } else {
      // the decay behind each of the 8 tokens, by three exchanges within 8 lanes (see suffix_kappa)
      float r[4] = {1.f, 1.f, 1.f, 1.f}, k[4] = {0.f, 0.f, 0.f, 0.f};
      if (mine) {
        widen<FRACSSM_F32>(q_rho, r);
        widen4<CK>(q_kap, k);
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        float v = mine ? fmaxf(r[x], kRhoFloor) : 1.f;
#pragma unroll
        for (int o = 1; o < kGroup; o *= 2) {
          const float y = __shfl_down_sync(0xffffffffu, v, o, kGroup);
          if (rt + o < kGroup) v *= y;
        }
        const float behind = __shfl_down_sync(0xffffffffu, v, 1, kGroup);
        k[x] *= rt + 1 < kGroup ? fmaxf(behind, kLeastBehind) : 1.f;
        r[x] = fmaxf(v, kLeastDecay);
      }
      if (owns) {
        *reinterpret_cast<float4 *>(d + kOffK) = make_float4(k[0], k[1], k[2], k[3]);
        if (rt == 0) *reinterpret_cast<float4 *>(d) = make_float4(r[0], r[1], r[2], r[3]);
      }
    }
#pragma unroll
    for (int i = 0; i < kUMax; ++i) {
      const int at = lane + i * lanes, ut = at >> a.u_shift, uq = at - (ut << a.u_shift);
      if (ut < n) {
        constexpr int kN = 16 / kUs;
        float f[kN];
        widen<UD>(q_u[i], f);
        float *du = to + ut * tok_floats + kOffU + kN * uq;
#pragma unroll
        for (int e = 0; e < kN; e += 4)
          *reinterpret_cast<float4 *>(du + e) = make_float4(f[e], f[e + 1], f[e + 2], f[e + 3]);
      }
    }
  };
  // any stride, alignment and size: element by element, when the group is due.  True where an infinity or NaN of u meets
  // padding modes: their zero coefficients would make NaN of it.
  auto copy_group = [&](int ib) {
    bool meets = false;
    const int n = min(kGroup, ntok - ib * kGroup);
    for (int i = lane; i < n * Mp; i += lanes) {
      const int t = i / Mp, m = i % Mp;
      const int64_t tt = (int64_t)ib * kGroup + t;
      float *d = wide + t * tok_floats + m;
      const bool on = m < a.M;
      d[0] = on ? fmaxf(reinterpret_cast<const float *>(rho_p + tt * a.rho.sl)[m], kRhoFloor) : kRhoFloor;
      d[kOffK] = on ? ld_f32(kap_p + tt * a.kappa.sl, m, CK) : 0.f;
      if (READOUT) d[kOffC] = on ? ld_f32(c_p + tt * a.c.sl, m, CK) : 0.f;
    }
    for (int i = lane; i < n * a.block_cols; i += lanes) {
      const int t = i / a.block_cols, r = i - t * a.block_cols;
      const float v = r < cols ? ld_f32(u_p + ((int64_t)ib * kGroup + t) * a.u.sl, r, UD) : 0.f;
      wide[t * tok_floats + kOffU + r] = v;
      if (PADDED) meets |= !isfinite(v);
    }
    return meets;
  };
  // kappa times the decay behind its token within the group, in place, and the group's decay in place of token 0's rho: the
  // same products in the same order as in store_group
  auto suffix_kappa = [&](int n) {
    for (int m = lane; n > 0 && m < Mp; m += lanes) {   // (n is 0 for threads beyond the last segment)
      float r[kGroup];
#pragma unroll
      for (int t = 0; t < kGroup; ++t) r[t] = t < n ? wide[t * tok_floats + m] : 1.f;
#pragma unroll
      for (int o = 1; o < kGroup; o *= 2) {
#pragma unroll
        for (int t = 0; t + o < kGroup; ++t) r[t] *= r[t + o];
      }
#pragma unroll
      for (int t = 0; t + 1 < kGroup; ++t)
        if (t < n) wide[t * tok_floats + kOffK + m] *= fmaxf(r[t + 1], kLeastBehind);
      wide[m] = fmaxf(r[0], kLeastDecay);
    }
  };
  if (a.wide_loads) request(0);
  grid_dep_wait();

  f2 st[kCols][4], prod[4];
#pragma unroll
  for (int r = 0; r < kCols; ++r)
#pragma unroll
    for (int p = 0; p < 4; ++p) st[r][p] = mk2(0.f, 0.f);
#pragma unroll
  for (int p = 0; p < 4; ++p) prod[p] = mk2(1.f, 1.f);
  if (READOUT && (s > 0 || a.init)) {
    // (compile-time indexes into the state: it lives in registers)
#pragma unroll
    for (int r = 0; r < kCols; ++r) {
      if (r < nr) {
        if (s > 0) {
          const float *src = a.states + (((int64_t)b * a.nseg + s) * a.R + col0 + my + r) * Mp + kModes * g;
          const ulonglong2 x = __ldcg(reinterpret_cast<const ulonglong2 *>(src));
          const ulonglong2 y = __ldcg(reinterpret_cast<const ulonglong2 *>(src + 4));
          st[r][0] = x.x; st[r][1] = x.y; st[r][2] = y.x; st[r][3] = y.y;
        } else {
          const float *src = a.init + ((int64_t)b * a.R + col0 + my + r) * a.M;
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const int m = kModes * g + 2 * p;
            st[r][p] = mk2(m < a.M ? src[m] : 0.f, m + 1 < a.M ? src[m + 1] : 0.f);
          }
        }
      }
    }
  }

  int64_t row = ((int64_t)b * a.L + t0) * a.R + col0 + my;
  // the sums over the modes of this thread's columns, and the nw first of them to row `row` of h
  auto read_state = [&](const f2 (&cc)[4], int64_t row, int nw) {
    float o[kCols];
#pragma unroll
    for (int r = 0; r < kCols; ++r) {
      f2 acc = mul2(cc[0], st[r][0]);
#pragma unroll
      for (int p = 1; p < 4; ++p) acc = fma2(cc[p], st[r][p], acc);
      float lo, hi;
      un2(acc, lo, hi);
      o[r] = lo + hi;
    }
    if constexpr (G == 1) {
      if (a.h_vec && nw == kCols) {
        if constexpr (UD == FRACSSM_F32) {
          *reinterpret_cast<float4 *>(reinterpret_cast<float *>(a.h) + row) = make_float4(o[0], o[1], o[2], o[3]);
        } else if constexpr (UD == FRACSSM_BF16) {
          *reinterpret_cast<uint2 *>(reinterpret_cast<__nv_bfloat16 *>(a.h) + row) =
              make_uint2(tile::pack2(o[0], o[1]), tile::pack2(o[2], o[3]));
        } else {
          const __half2 v0 = __floats2half2_rn(o[0], o[1]), v1 = __floats2half2_rn(o[2], o[3]);
          *reinterpret_cast<uint2 *>(reinterpret_cast<__half *>(a.h) + row) =
              make_uint2(*reinterpret_cast<const uint32_t *>(&v0), *reinterpret_cast<const uint32_t *>(&v1));
        }
      } else {
#pragma unroll
        for (int r = 0; r < kCols; ++r)
          if (r < nw) st_f32(a.h, row + r, UD, o[r]);
      }
    } else {
      // sum over the mode groups; the first two steps halve the columns a lane answers for
      const bool b0 = g & 1;
      float x0 = __shfl_xor_sync(0xffffffffu, b0 ? o[0] : o[2], 1);
      float x1 = __shfl_xor_sync(0xffffffffu, b0 ? o[1] : o[3], 1);
      x0 += b0 ? o[2] : o[0];
      x1 += b0 ? o[3] : o[1];
      const int r0 = b0 ? 2 : 0;
      if constexpr (G == 2) {
        if (a.h_vec && nw == kCols && UD != FRACSSM_F16) {
          if (UD == FRACSSM_F32)
            *reinterpret_cast<float2 *>(reinterpret_cast<float *>(a.h) + row + r0) = make_float2(x0, x1);
          else *reinterpret_cast<uint32_t *>(reinterpret_cast<__nv_bfloat16 *>(a.h) + row + r0) = tile::pack2(x0, x1);
        } else {
          if (r0 < nw) st_f32(a.h, row + r0, UD, x0);
          if (r0 + 1 < nw) st_f32(a.h, row + r0 + 1, UD, x1);
        }
      } else {
        const bool b1 = g & 2;
        float y = (b1 ? x1 : x0) + __shfl_xor_sync(0xffffffffu, b1 ? x0 : x1, 2);
#pragma unroll
        for (int o2 = 4; o2 < G; o2 *= 2) y += __shfl_xor_sync(0xffffffffu, y, o2);
        const int r1 = r0 + (b1 ? 1 : 0);
        if (g < 4 && r1 < nw) st_f32(a.h, row + r1, UD, y);
      }
    }
  };
  auto columns = [&](const float *tok, f2 (&uu)[kCols]) {
    const float4 u4 = *reinterpret_cast<const float4 *>(tok + kOffU + my);
    uu[0] = mk2(u4.x, u4.x); uu[1] = mk2(u4.y, u4.y); uu[2] = mk2(u4.z, u4.z); uu[3] = mk2(u4.w, u4.w);
  };
  // a group of n tokens in `tok`
  auto summarise = [&](const float *tok, int n) {   // state := group's decay (.) state + sum of u kappa^T decayed to its end
    f2 g8[4];
    ld_pairs(tok + kModes * g, g8);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      prod[p] = mul2(prod[p], g8[p]);
#pragma unroll
      for (int r = 0; r < kCols; ++r) st[r][p] = mul2(st[r][p], g8[p]);
    }
#pragma unroll 4
    for (int t = 0; t < n; ++t, tok += tok_floats) {
      f2 ka[4], uu[kCols];
      ld_pairs(tok + kOffK + kModes * g, ka);
      columns(tok, uu);
#pragma unroll
      for (int r = 0; r < kCols; ++r) {
#pragma unroll
        for (int p = 0; p < 4; ++p) st[r][p] = fma2(ka[p], uu[r], st[r][p]);
      }
    }
  };
  auto advance = [&](const float *tok) {
    f2 rr[4], ka[4], uu[kCols];
    ld_pairs(tok + kModes * g, rr);
    ld_pairs(tok + kOffK + kModes * g, ka);
    columns(tok, uu);
#pragma unroll
    for (int r = 0; r < kCols; ++r) {
#pragma unroll
      for (int p = 0; p < 4; ++p) st[r][p] = fma2(rr[p], st[r][p], mul2(ka[p], uu[r]));
    }
  };
  // the padding modes' state stays zero (an infinity of u times their zero coefficients would make NaN of it)
  auto clear_padding = [&]() {
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int m = kModes * g + 2 * p;
#pragma unroll
      for (int r = 0; r < kCols; ++r) {
        float lo, hi;
        un2(st[r][p], lo, hi);
        st[r][p] = mk2(m < a.M ? lo : 0.f, m + 1 < a.M ? hi : 0.f);
      }
    }
  };

  if (!PADDED && a.wide_loads) {
    // All columns are live, and where the readout exchanges between lanes a block has one segment (see few_wide_shape): no
    // thread idles along.
    for (int ib = 0; ib * kGroup < all_tok; ++ib) {
      if (kBuffers == 1 && ib > 0) __syncthreads();   // the previous group has been read
      float *const tok = wide + (kBuffers == 2 ? (ib & 1) * buf_floats : 0);
      store_group(ib, tok);
      request(ib + 1);
      __syncthreads();
      const int n = max(0, min(kGroup, ntok - ib * kGroup));
      if constexpr (!READOUT) {
        if (n > 0) summarise(tok, n);
      } else {
#pragma unroll 2
        for (int t = 0; t < n; ++t, row += a.R) {
          const float *const at = tok + t * tok_floats;
          advance(at);
          f2 cc[4];
          ld_pairs(at + kOffC + kModes * g, cc);
          read_state(cc, row, kCols);
        }
      }
    }
  } else {
    for (int ib = 0; ib * kGroup < all_tok; ++ib) {
      if (ib > 0) __syncthreads();   // the previous group has been read
      bool keep_zero = false;        // the padding modes' state
      const bool meets = copy_group(ib);
      if constexpr (PADDED) keep_zero = __syncthreads_or(meets);
      else __syncthreads();
      const int n = max(0, min(kGroup, ntok - ib * kGroup)), n_all = min(kGroup, all_tok - ib * kGroup);
      if constexpr (!READOUT) {
        suffix_kappa(n);
        __syncthreads();
        if (n > 0) summarise(wide, n);
        if (PADDED && keep_zero) clear_padding();
      } else {
        const float *tok = wide;
#pragma unroll 1
        for (int t = 0; t < n_all; ++t, row += a.R, tok += tok_floats) {
          f2 cc[4];
          ld_pairs(tok + kOffC + kModes * g, cc);
          if (t < n) {
            advance(tok);
            if (PADDED && keep_zero) clear_padding();
          }
          read_state(cc, row, t < n ? nr : 0);
        }
      }
    }
  }

  if (!READOUT) {
#pragma unroll
    for (int r = 0; r < kCols; ++r) {
      if (r < nr) {
        float *dst = a.states + (((int64_t)b * a.nseg + s) * a.R + col0 + my + r) * Mp + kModes * g;
        __stcg(reinterpret_cast<ulonglong2 *>(dst), make_ulonglong2(st[r][0], st[r][1]));
        __stcg(reinterpret_cast<ulonglong2 *>(dst + 4), make_ulonglong2(st[r][2], st[r][3]));
      }
    }
    if (owner && cl == 0 && blockIdx.y == 0) {
      f2 *dst = reinterpret_cast<f2 *>(a.decay + ((int64_t)b * a.nseg + s) * Mp + kModes * g);
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        float lo, hi;
        un2(prod[p], lo, hi);
        dst[p] = mk2(fmaxf(lo, kLeastDecay), fmaxf(hi, kLeastDecay));
      }
    }
  } else if (a.fin && s == a.nseg - 1) {
#pragma unroll
    for (int r = 0; r < kCols; ++r) {
      if (r < nr) {
        const int64_t dst = (int64_t)b * a.R * a.M + (int64_t)(col0 + my + r) * a.fin_sr;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const int m = kModes * g + 2 * p;
          float lo, hi;
          un2(st[r][p], lo, hi);
          if (m < a.M) st_f32(a.fin, dst + (int64_t)m * a.fin_sm, a.fin_dt, lo);
          if (m + 1 < a.M) st_f32(a.fin, dst + (int64_t)(m + 1) * a.fin_sm, a.fin_dt, hi);
        }
      }
    }
  }
}

// states[b][s] := the state entering segment s.  A thread composes the segments of its share, walks them again from
// the state that enters the share, and keeps up to BATCH of them in registers in between (read once, written once).
// A warp owns 32 / SUB neighbouring elements of a row's state, and its lanes SUB neighbouring shares of each.  Bound by the
// latency of the one read: with SUB = 1 throughout, 1185 segments (1 row x 32768 tokens, 64 columns x 8 modes) were read twice
// in four rounds, 24 us, 13 here.
constexpr int kCarryWarps = 32;
template <int BATCH, int SUB>
__global__ void __launch_bounds__(32 * kCarryWarps)
few_carry_kernel(float *__restrict__ states, const float *__restrict__ decay, const float *__restrict__ init,
                 int nseg, int R, int M, int Mp) {
  constexpr int kElems = 32 / SUB;
  __shared__ float ps[kCarryWarps][kElems], ss[kCarryWarps][kElems];
  const int lane = threadIdx.x % 32, w = threadIdx.x / 32, warps = blockDim.x / 32, el = lane % kElems, sub = lane / kElems;
  const int64_t b = blockIdx.y;
  const int RM = R * Mp, e = blockIdx.x * kElems + el;
  const bool live = e < RM;
  const int m = e % Mp, r = e / Mp;
  const int share = (nseg + warps * SUB - 1) / (warps * SUB);
  const int lo = min((w * SUB + sub) * share, nseg), hi = min(lo + share, nseg), last = nseg - 1;   // `last` has no summary
  float *sp = states + (b * nseg + lo) * RM + (live ? e : 0);
  const float *dp = decay + (b * nseg + lo) * Mp + m;
  grid_dep_launch();
  grid_dep_wait();
  float p = 1.f, v = 0.f;
  float x[BATCH], d[BATCH];
  auto load = [&](int s0) {
    const float *xs = sp + (int64_t)(s0 - lo) * RM, *ds = dp + (int64_t)(s0 - lo) * Mp;
    const int n = min(hi, last) - s0;
#pragma unroll
    for (int i = 0; i < BATCH; ++i, xs += RM, ds += Mp) {
      x[i] = i < n ? __ldcg(xs) : 0.f;
      d[i] = i < n ? __ldcg(ds) : 1.f;
    }
  };
  for (int s0 = lo; s0 < hi; s0 += BATCH) {
    load(s0);
#pragma unroll
    for (int i = 0; i < BATCH; ++i) {
      v = fmaf(d[i], v, x[i]);
      p *= d[i];
    }
  }
  p = fmaxf(p, kLeastDecay);
  // the warp's shares one after the other: (p, v) up to and with each, then without it
#pragma unroll
  for (int o = 1; o < SUB; o *= 2) {
    const float p0 = __shfl_up_sync(0xffffffffu, p, o * kElems), v0 = __shfl_up_sync(0xffffffffu, v, o * kElems);
    if (sub >= o) {
      v = fmaf(p, v0, v);
      p = fmaxf(p * p0, kLeastDecay);
    }
  }
  if (sub == SUB - 1) {
    ps[w][el] = p;
    ss[w][el] = v;
  }
  if constexpr (SUB > 1) {
    p = __shfl_up_sync(0xffffffffu, p, kElems);
    v = __shfl_up_sync(0xffffffffu, v, kElems);
  }
  __syncthreads();
  if (!live) return;
  float run = init && m < M ? init[(b * R + r) * M + m] : 0.f;
  for (int i = 0; i < w; ++i) run = fmaf(ps[i][el], run, ss[i][el]);
  if (SUB > 1 && sub > 0) run = fmaf(p, run, v);
  for (int s0 = lo; s0 < hi; s0 += BATCH) {
    if (share > BATCH) load(s0);
    float *xs = sp + (int64_t)(s0 - lo) * RM;
    const int n = hi - s0;
#pragma unroll
    for (int i = 0; i < BATCH; ++i, xs += RM) {
      if (i < n) __stcg(xs, run);
      run = fmaf(d[i], run, x[i]);
    }
  }
}

struct FewPlan {
  int G, Mp, block_cols, col_blocks, lanes, per_block, seg, nseg;
  size_t bytes;
};

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

FewPlan few_plan(int64_t B, int64_t L, int64_t R, int64_t M) {
  FewPlan p{};
  p.G = M <= 8 ? 1 : M <= 16 ? 2 : M <= 32 ? 4 : M <= 64 ? 8 : 16;
  p.Mp = kModes * p.G;
  p.col_blocks = (int)ceil_div(R, kMaxBlockCols);
  p.block_cols = (int)ceil_div(ceil_div(R, p.col_blocks), kCols) * kCols;
  p.lanes = p.block_cols / kCols * p.G;
  p.per_block = 1;
  while (p.lanes * p.per_block * 2 <= 32 && (p.lanes & (p.lanes - 1)) == 0) p.per_block *= 2;
  // Warps that a row keeps busy by itself.  From 8 warps per SM on the rows alone are enough (the cut costs a
  // second read of u, kappa and rho and two thirds more arithmetic); below, segments of at least kMinSeg
  // tokens such that about kWarpsPerSm warps per SM run.  (12 / 16 / 28 warps: 75 / 62 / 71 us at 2 rows x 32768
  // tokens x 16 modes; 16 / 32 / 64 tokens: 29.5 / 33.5 / 44 us at 8 rows x 1024 tokens x 64 modes.)
  constexpr int64_t kWarpsPerSm = 16, kMinSeg = 16;
  const double row_warps = (double)p.col_blocks * (p.per_block > 1 ? 1.0 / p.per_block : (double)ceil_div(p.lanes, 32));
  int64_t nseg = 1;
  if (B * row_warps < 148 * 8) nseg = (int64_t)(148 * kWarpsPerSm / (B * row_warps)) + 1;
  int64_t seg = ceil_div(ceil_div(L, nseg), kGroup) * kGroup;
  if (seg < kMinSeg) seg = kMinSeg;
  p.seg = (int)(seg < L ? seg : L);
  p.nseg = (int)ceil_div(L, p.seg);
  if (p.nseg > 1)
    p.bytes = align256((size_t)B * p.nseg * R * p.Mp * 4) + align256((size_t)B * p.nseg * p.Mp * 4);
  return p;
}

// 16-byte loads: every row starts on a 16-byte boundary and fills whole pieces, there is no padding among the modes or
// columns, and a segment has the threads for one piece of rho each (64 columns or more).
bool few_wide_shape(const FewPlan &p, int64_t R, int64_t M, int u_size) {
  const int pieces = p.block_cols * u_size / 16;
  return p.block_cols * u_size % 16 == 0 && M == p.Mp && R % p.block_cols == 0 && (pieces & (pieces - 1)) == 0 &&
         p.lanes >= 16 * p.G;
}
bool few_wide_rows(const Rows &u, const Rows &c, const Rows &kappa, const Rows &rho) {
  uint64_t bits = 0;
  for (const Rows *r : {&u, &c, &kappa, &rho}) bits |= (uint64_t)(uintptr_t)r->p | (uint64_t)r->sb | (uint64_t)r->sl;
  return (bits & 15) == 0;
}

// Work (B L R Mp) up to which these kernels are the faster ones for calls that are cut into segments and load element by
// element: such a load is waited for anew in every group of 8 tokens, and a cut row is loaded twice.  How long the chunked
// stages take depends on the chunk: at 32, 128 and 256 tokens 1.5, 1.1 and 1.4 times as long as at 64.  Stages / segments
// in us, bfloat16, chunk 64:
//      2 x 32768 tokens, 128 columns x 40 modes  422 / 310       2 x 32768, 256 x 72  1143 / 1877
//      8 x 8192,          64 x 60                236 / 172       8 x 8192,  128 x 60   412 / 428
//     16 x 16384,         64 x 24                668 / 491      16 x 16384, 64 x 40    855 / 1091
//     16 x 2048,         192 x 20                186 / 177       8 x 8192,  192 x 20   375 / 462
// (192 columns are three blocks' worth of 64 but lie in two of 96, whose loads also divide by a number that is no power
// of two.)  At 16 or fewer modes, at 32 or fewer columns and wherever rows are taken whole or loads are wide, the
// segments were the faster in every one of some 500 such pairs but for 4 % at 192 x 12.
double few_narrow_limit(const FewPlan &p, int64_t B, int64_t R, int64_t T) {
  if (R <= 32 || p.Mp <= 16) return 1e30;
  const bool odd = (p.block_cols & (p.block_cols - 1)) != 0;
  if (T < 48 || T >= 192) {
    if (p.Mp <= (odd ? 32 : 64)) return 1e30;
    return (odd ? 1.2e9 : 2e9) * (B > 32 ? 3 : 1);
  }
  double limit;
  if (odd) limit = p.Mp == 32 ? 256e6 : B <= 2 ? 100e6 : 64e6;
  else limit = B <= 2 ? 800e6 : p.Mp == 32 && B <= 32 ? 600e6 : 400e6;
  return T < 96 ? limit : 2 * limit;
}

template <typename... P, typename... Args>
cudaError_t few_launch_dep(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, bool dependent,
                           Args... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// The three launches follow one another by programmatic stream serialisation: the next one's blocks start and
// request their inputs while the last blocks of the previous one finish.
template <int G, int UD, int CK>
int few_launch(FewArgs &a, const FewPlan &p, cudaStream_t st) {
  constexpr int Mp = kModes * G, kUs = UD == FRACSSM_F32 ? 4 : 2;
  const int threads = (int)(ceil_div(p.lanes * p.per_block, 32) * 32);
  const int pieces = p.block_cols * kUs / 16;
  a.wide_loads = few_wide_shape(p, a.R, a.M, kUs) && few_wide_rows(a.u, a.c, a.kappa, a.rho);
  a.u_shift = 0;
  while ((1 << a.u_shift) < pieces) ++a.u_shift;
  const size_t tokens = (size_t)p.per_block * kGroup;
  const size_t sum_smem = tokens * (2 * Mp + p.block_cols + kTokPad) * 4 * (a.wide_loads ? few_buffers(G, false) : 1);
  const size_t out_smem = tokens * (3 * Mp + p.block_cols) * 4 * (a.wide_loads ? few_buffers(G, true) : 1);
  if (out_smem > 48 * 1024) return fail(FRACSSM_ERR_UNSUPPORTED, "frac_scan: shared memory of the segment kernel");
  cudaError_t e = cudaSuccess;
  auto blocks = [&](int64_t segs) { return dim3((unsigned)ceil_div((int64_t)a.B * segs, p.per_block), p.col_blocks); };
  if (p.nseg > 1) {
    auto summary = a.M < Mp ? few_scan_kernel<G, UD, CK, false, true> : few_scan_kernel<G, UD, CK, false, false>;
    e = few_launch_dep(summary, blocks(p.nseg - 1), threads, sum_smem, st, false, a);
    // (no more registers than a share needs: a place that stays empty costs its instructions all the same)
    auto carry = p.nseg <= 8 * kCarryWarps ? few_carry_kernel<8, 1>
                 : p.nseg <= 12 * kCarryWarps ? few_carry_kernel<12, 1>
                 : p.nseg <= 24 * kCarryWarps ? few_carry_kernel<12, 2>
                 : p.nseg <= 48 * kCarryWarps ? few_carry_kernel<12, 4>
                                              : few_carry_kernel<12, 8>;
    const int elems = p.nseg <= 12 * kCarryWarps ? 32 : p.nseg <= 24 * kCarryWarps ? 16 : p.nseg <= 48 * kCarryWarps ? 8 : 4;
    int warps = (int)ceil_div(p.nseg, 8);
    if (warps > kCarryWarps) warps = kCarryWarps;
    if (e == cudaSuccess)
      e = few_launch_dep(carry, dim3((unsigned)ceil_div((int64_t)a.R * Mp, elems), (unsigned)a.B), 32 * warps,
                         0, st, true, a.states, a.decay, a.init, p.nseg, a.R, a.M, Mp);
  }
  auto readout = a.M < Mp ? few_scan_kernel<G, UD, CK, true, true> : few_scan_kernel<G, UD, CK, true, false>;
  if (e == cudaSuccess)
    e = few_launch_dep(readout, blocks(p.nseg), threads, out_smem, st, p.nseg > 1, a);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(FRACSSM_ERR_CUDA, "frac_scan (segment kernels): %s", cudaGetErrorString(e));
  }
  return check_launch("frac_scan (segment kernels)");
}

template <int UD, int CK>
int few_launch_modes(FewArgs &a, const FewPlan &p, cudaStream_t st) {
  if (p.G == 1) return few_launch<1, UD, CK>(a, p, st);
  if (p.G == 2) return few_launch<2, UD, CK>(a, p, st);
  if (p.G == 4) return few_launch<4, UD, CK>(a, p, st);
  if (p.G == 8) return few_launch<8, UD, CK>(a, p, st);
  return few_launch<16, UD, CK>(a, p, st);
}

}  // namespace

// Up to 128 modes the state of 4 columns fits the registers of at most 16 threads (half a warp, which adds the
// readout by shuffles); beyond, the chunked stages stay.  The other limits are those of the chunked stages (a launch's
// grid).
bool scan_few_supported(int64_t B, int64_t L, int64_t R, int64_t M, int64_t T) {
  if (B < 1 || L < 1 || R < 1 || M < 1 || M > 128 || R > 65535 || B > 65535 || L >= (int64_t(1) << 30)) return false;
  if (ceil_div(L, T) > 65535) return false;
  const FewPlan p = few_plan(B, L, R, M);
  return B * p.nseg < (int64_t(1) << 31);
}

size_t scan_few_workspace_bytes(int64_t B, int64_t L, int64_t R, int64_t M) { return few_plan(B, L, R, M).bytes; }

// Whether the chunked stages are the faster kernels for a call that loads element by element; for one that takes its
// rows in 16-byte pieces they never are.
bool scan_few_narrow_slower(int64_t B, int64_t L, int64_t R, int64_t M, int64_t T) {
  const FewPlan p = few_plan(B, L, R, M);
  return p.nseg > 1 && (double)B * L * R * p.Mp > few_narrow_limit(p, B, R, T);
}
bool scan_few_shape_loads_wide(int64_t R, int64_t M) {
  const FewPlan p = few_plan(1, 1, R, M);
  return few_wide_shape(p, R, M, 2) && few_wide_shape(p, R, M, 4);
}
bool scan_few_loads_wide(const void *u, int u_dtype, int64_t u_sb, int64_t u_sl, const void *c, const void *kappa,
                         int ck_dtype, int64_t c_sb, int64_t c_sl, int64_t k_sb, int64_t k_sl, const float *rho,
                         int64_t r_sb, int64_t r_sl, int64_t R, int64_t M) {
  const int us = (int)dtype_size(u_dtype), ks = (int)dtype_size(ck_dtype);
  return few_wide_shape(few_plan(1, 1, R, M), R, M, us) &&
         few_wide_rows(few_rows(u, u_sb, u_sl, us), few_rows(c, c_sb, c_sl, ks), few_rows(kappa, k_sb, k_sl, ks),
                       few_rows(rho, r_sb, r_sl, 4));
}

int scan_few_launch(const void *u, int u_dtype, int64_t u_sb, int64_t u_sl, const void *c, const void *kappa,
                    int ck_dtype, int64_t c_sb, int64_t c_sl, int64_t k_sb, int64_t k_sl, const float *rho,
                    int64_t r_sb, int64_t r_sl, const float *initial_state, void *h, void *final_state,
                    int final_dtype, void *workspace, int64_t B, int64_t L, int64_t R, int64_t M, void *stream,
                    bool fin_modes_first) {
  const FewPlan p = few_plan(B, L, R, M);
  FewArgs a{};
  const int us = (int)dtype_size(u_dtype), ks = (int)dtype_size(ck_dtype);
  a.u = few_rows(u, u_sb, u_sl, us);
  a.c = few_rows(c, c_sb, c_sl, ks);
  a.kappa = few_rows(kappa, k_sb, k_sl, ks);
  a.rho = few_rows(rho, r_sb, r_sl, 4);
  a.init = initial_state;
  a.h = h;
  a.h_vec = R % 4 == 0 && (reinterpret_cast<uintptr_t>(h) & 15) == 0;
  a.fin = final_state;
  a.fin_dt = final_dtype;
  a.fin_sr = fin_modes_first ? 1 : (int)M;
  a.fin_sm = fin_modes_first ? (int)R : 1;
  a.states = reinterpret_cast<float *>(workspace);
  a.decay = reinterpret_cast<float *>(reinterpret_cast<char *>(workspace) + align256((size_t)B * p.nseg * R * p.Mp * 4));
  a.L = L;
  a.B = (int)B;
  a.R = (int)R;
  a.M = (int)M;
  a.nseg = p.nseg;
  a.seg = p.seg;
  a.block_cols = p.block_cols;
  a.lanes = p.lanes;
  a.per_block = p.per_block;
  const cudaStream_t st = (cudaStream_t)stream;
  if (u_dtype == FRACSSM_F32) return few_launch_modes<FRACSSM_F32, FRACSSM_F32>(a, p, st);
  if (u_dtype == FRACSSM_BF16)
    return ck_dtype == FRACSSM_F32 ? few_launch_modes<FRACSSM_BF16, FRACSSM_F32>(a, p, st)
                                   : few_launch_modes<FRACSSM_BF16, FRACSSM_BF16>(a, p, st);
  return ck_dtype == FRACSSM_F32 ? few_launch_modes<FRACSSM_F16, FRACSSM_F32>(a, p, st)
                                 : few_launch_modes<FRACSSM_F16, FRACSSM_F16>(a, p, st);
}

}  // namespace fracssm
