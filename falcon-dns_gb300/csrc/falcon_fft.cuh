// The azimuthal transforms and the nonlinear pass (Nr_maxLOOP,
// src/nonlin.F90:35-91) in 64-bit fixed point (falcon_fixed.h): the
// butterfly stages on integer instructions and, for radices 11 to 31 of
// prime-factor plans, on the fp16 tensor cores; the kernel and its launcher.
// Included by one translation unit per class of plans (falcon_fft8.cu,
// falcon_fft17.cu, falcon_fft31.cu), which compile in parallel; everything
// here has internal linkage.
#pragma once
#include <algorithm>
#include <mutex>

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>

#include "falcon_fixed.h"
#include "falcon_internal.h"
#include "falcon_slices.cuh"

namespace falcon {
namespace {

// ---------------------------------------------------------------------------
// Tensor-core butterflies.  The symmetric butterfly (fx_dft) of an odd prime
// p, h = (p - 1)/2:  A_j - v_0 = sum_q a_q cos(2 pi jq/p) and B_j = sum_q b_q
// sin(2 pi jq/p) as integer matrix products.  Coefficients (Q62) and values
// (|a|, |b| < 2^61) are cut into kFxS = 7 signed 9-bit digits, balanced in
// [-256, 255] (the top one by its sign), which fp16 holds exactly; the 28
// digit pairs s + t <= 6 are summed per diagonal d = s + t in FP32.  Every
// accumulator starts at 1.5 2^23: with balanced digits a diagonal's partial
// sums stay below 0.9 2^22 (p = 31: sum over pairs and products of |digit
// of c| 256), so the sums are exact and the accumulator's bits are
// 0x4b400000 + sum, an integer with no conversion instruction.  The dropped
// pairs weigh 3 units a product at most, 0.4 rms (tests/test_balanced_digits.py),
// of values whose largest is 2^54 (radix 23 to 31) or 2^55 units going in: grids
// of 345 and 1023 points 5e-16 of a result's norm, of 255 and 429 2e-16.
// ---------------------------------------------------------------------------
constexpr int kFxS = 7;
constexpr int kFxMagic = 0x4b400000;  // bits of 1.5 2^23
constexpr unsigned long long kFxBias = 256ull * ((1ull << 63) / 511ull);  // 256 (512^7 - 1)/511

constexpr int fx_digit(long long c, int s) {  // digit s (0 = leading) of a Q62 constant
  int d = 0;
  for (int i = kFxS - 1; i >= s; --i) {
    d = i ? (int)(((c + 256) % 512 + 512) % 512) - 256 : (int)c;
    c = (c - d) / 512;
  }
  return d;
}
constexpr uint32_t fx_half_bits(int q) {  // fp16 bits of an integer |q| <= 2048
  if (q == 0) return 0u;
  const uint32_t a = (uint32_t)(q < 0 ? -q : q);
  int e = 0;
  while ((2u << e) <= a) ++e;
  return (q < 0 ? 0x8000u : 0u) | (uint32_t)((15 + e) << 10) | ((a << (10 - e)) & 0x3ffu);
}
template <int p>
constexpr uint32_t fx_coef_pair(bool sine, int j, int q, int s) {  // digits of (j, q), (j, q + 1) as an fp16 pair
  constexpr int h = (p - 1) / 2;
  uint32_t r = 0;
  for (int i = 0; i < 2; ++i)
    if (j <= h && q + i <= h)
      r |= fx_half_bits(fx_digit(sine ? FxDft<p>::s[(j * (q + i)) % p] : FxDft<p>::c[(j * (q + i)) % p], s)) << (16 * i);
  return r;
}

// The A fragments of mma.m16n8k16, [digit][lane][words].  h <= 8: the
// block-diagonal [C 0; 0 S] (rows j; K = the h values a_q, then b_q), words
// (a0, a3).  h <= 15: C and S as two 16 x 16 tiles, words (a0, a1, a2, a3)
// of C, then of S.
template <int p>
struct FxFrag {
  static constexpr int kWords = p <= 17 ? 2 : 8;
  static constexpr int kInts = kFxS * 32 * kWords;
  uint32_t v[kInts];
};
template <int p>
constexpr FxFrag<p> fx_frag() {
  FxFrag<p> f{};
  constexpr int W = FxFrag<p>::kWords;
  for (int s = 0; s < kFxS; ++s)
    for (int lane = 0; lane < 32; ++lane) {
      const int j = (lane >> 2) + 1, q = 2 * (lane & 3) + 1;
      for (int w = 0; w < W; ++w) {
        uint32_t r = 0;
        if constexpr (W == 2) r = fx_coef_pair<p>(w == 1, j, q, s);
        else r = fx_coef_pair<p>(w >= 4, j + 8 * (w & 1), q + 8 * ((w >> 1) & 1), s);
        f.v[(s * 32 + lane) * W + w] = r;
      }
    }
  return f;
}
template <int p>
__device__ const FxFrag<p> kFxFrag = fx_frag<p>();

// 32-bit words of fragments a plan's block holds in shared memory.
__host__ __device__ constexpr int fx_frag_ints(int p) { return p <= 7 ? 0 : p <= 17 ? FxFrag<17>::kInts : FxFrag<31>::kInts; }

__device__ __forceinline__ void fx_mma(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                       unsigned b1, float c0, float c1, float c2, float c3) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%11,%12,%13};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
}

// Digit s of two biased values (u = v + kFxBias) as an fp16 pair: fp16(1536 +
// d) has the bits 0x6600 + d for 0 <= d < 512, so one packed subtraction of
// 1792 gives the balanced digits d - 256.
__device__ __forceinline__ uint32_t fx_digits(unsigned long long u0, unsigned long long u1, int s) {
  const int sh = 9 * (kFxS - 1 - s);
  const uint32_t both = __byte_perm((uint32_t)(u0 >> sh), (uint32_t)(u1 >> sh), 0x5410);
  const uint32_t biased = (both & 0x01ff01ffu) | 0x66006600u;
  const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&biased), __floats2half2_rn(1792.f, 1792.f));
  return *reinterpret_cast<const uint32_t*>(&v);
}

// The product sum_d q_d 512^(12 - d) 2^-62 from the accumulator bits of its
// diagonals (modulo 2^64 every term may wrap; the result is below 2^62):
// weights 2^(46 - 9 d), the last diagonal shifted down.
__device__ __forceinline__ long long fx_undigit(const float (&acc)[kFxS][4], int i) {
  constexpr unsigned long long B = (unsigned long long)kFxMagic;
  constexpr unsigned long long off = 0ull - ((B << 46) + (B << 37) + (B << 28) + (B << 19) + (B << 10) + (B << 1) + (B >> 8));
  const int b0 = __float_as_int(acc[0][i]), b1 = __float_as_int(acc[1][i]), b2 = __float_as_int(acc[2][i]),
            b3 = __float_as_int(acc[3][i]), b4 = __float_as_int(acc[4][i]), b5 = __float_as_int(acc[5][i]),
            b6 = __float_as_int(acc[6][i]);
  long long w = fx_madw(b2, 1 << 28, (long long)off);
  w = fx_madw(b3, 1 << 19, w);
  w = fx_madw(b4, 1 << 10, w);
  w = fx_madw(b5, 2, w);
  w = fx_madw(b6 >> 8, 1, w);
  const unsigned hi = (unsigned)b0 * (1u << 14) + (unsigned)b1 * (1u << 5);
  return (long long)((unsigned long long)w + ((unsigned long long)hi << 32));
}

// One stage (p = 11, 13, 17; no twiddles) of one buffer, inputs scaled by
// 2^-d: tiles of 4 butterflies x (re, im) = 8 columns to warps warp, warp +
// nw, ...  Lane (g, t) holds v_q, v_{p-q} for q = 2t + 1, 2t + 2 and v_0 of
// column g, and receives A_{g+1}, B_{g+1} of butterfly t, re and im, from
// which it stores y_j and y_{p-j}.  y_0 = v_0 + sum a_q by shuffles.  The
// caller synchronises before (inputs complete) and after (outputs stored).
// Results do not depend on the tiling.
template <int p>
__device__ void fx_mma_stage(longlong2* buf, int P, int m, int d, const uint32_t* frag, int lane, int warp, int nw,
                             FxMax& o) {
  constexpr int h = (p - 1) / 2;
  static_assert(h <= 8, "the block-diagonal form holds h <= 8");
  constexpr unsigned FULL = 0xffffffffu;
  const float magic = __int_as_float(kFxMagic);
  const int gid = lane >> 2, tig = lane & 3;
  const int nb = P / p, mp = m * p, ntile = (nb + 3) / 4;
  const float inv_m = 1.0f / (float)m;
  const int q1 = 2 * tig + 1, q2 = 2 * tig + 2;
  const bool has1 = q1 <= h, has2 = q2 <= h;
  const uint2* fr = reinterpret_cast<const uint2*>(frag) + lane;
  for (int tile = warp; tile < ntile; tile += nw) {
    const int bi = tile * 4 + (gid >> 1), comp = gid & 1;
    long long x1 = 0, y1 = 0, x2 = 0, y2 = 0, v0 = 0;
    long long* pi = nullptr;
    if (bi < nb) {
      const int g = (int)(((float)bi + 0.5f) * inv_m);
      pi = reinterpret_cast<long long*>(buf + g * mp + (bi - g * m)) + comp;
      if (has1) { x1 = pi[2 * q1 * m]; y1 = pi[2 * (p - q1) * m]; }
      if (has2) { x2 = pi[2 * q2 * m]; y2 = pi[2 * (p - q2) * m]; }
      v0 = pi[0];
    }
    if (d > 0) { x1 >>= d; y1 >>= d; x2 >>= d; y2 >>= d; v0 >>= d; }
    else if (d < 0) {
      x1 = fx_scale(x1, d); y1 = fx_scale(y1, d); x2 = fx_scale(x2, d); y2 = fx_scale(y2, d); v0 = fx_scale(v0, d);
    }
    const long long a1 = x1 + y1, a2 = x2 + y2;
    const unsigned long long ua1 = (unsigned long long)a1 + kFxBias, ua2 = (unsigned long long)a2 + kFxBias,
                             ub1 = (unsigned long long)(x1 - y1) + kFxBias,
                             ub2 = (unsigned long long)(x2 - y2) + kFxBias;
    long long ys = a1 + a2;
    ys += __shfl_xor_sync(FULL, ys, 1);
    ys += __shfl_xor_sync(FULL, ys, 2);
    __syncwarp();  // every load of the tile precedes its stores
    if (tig == 0 && pi) {
      pi[0] = v0 + ys;
      if (comp) fx_cover(o, fx_make(0, v0 + ys));
      else fx_cover(o, fx_make(v0 + ys, 0));
    }
    float acc[kFxS][4];
    uint32_t fa[kFxS], fb[kFxS];
#pragma unroll
    for (int t = 0; t < kFxS; ++t) {
      fa[t] = fx_digits(ua1, ua2, t);
      fb[t] = fx_digits(ub1, ub2, t);
    }
#pragma unroll
    for (int s = 0; s < kFxS; ++s) {
      const uint2 c = fr[s * 32];
#pragma unroll
      for (int t = 0; s + t < kFxS; ++t) {
        float(&ac)[4] = acc[s + t];
        if (s == 0) fx_mma(ac, c.x, 0u, 0u, c.y, fa[t], fb[t], magic, magic, magic, magic);
        else fx_mma(ac, c.x, 0u, 0u, c.y, fa[t], fb[t], ac[0], ac[1], ac[2], ac[3]);
      }
    }
    // this lane's butterfly bo; lanes 8t, 8t + 4 loaded its v_0
    const int bo = tile * 4 + tig;
    const long long w_re = __shfl_sync(FULL, v0, 8 * tig), w_im = __shfl_sync(FULL, v0, 8 * tig + 4);
    if (gid < h && bo < nb) {
      const int g = (int)(((float)bo + 0.5f) * inv_m);
      longlong2* po = buf + g * mp + (bo - g * m);
      const longlong2 A = fx_make(w_re + fx_undigit(acc, 0), w_im + fx_undigit(acc, 1));
      const longlong2 B = fx_make(fx_undigit(acc, 2), fx_undigit(acc, 3));
      longlong2 yj, yk;
      fx_pair(A, B, yj, yk);
      const int j = gid + 1;
      po[j * m] = yj;
      po[(p - j) * m] = yk;
      fx_cover(o, yj);
      fx_cover(o, yk);
    }
  }
}

// The same for p = 19, 23, 29, 31 (h = 9..15): C and S as two 16 x 16 tiles.
// Lane (g, t) holds v_q, v_{p-q} for q = 2t + 1, 2t + 2, 2t + 9, 2t + 10 of
// column g and receives A_j, B_j for j = g + 1 and g + 9 of butterfly t.
template <int p>
__device__ void fx_mma_stage_wide(longlong2* buf, int P, int m, int d, const uint32_t* frag, int lane, int warp,
                                  int nw, FxMax& o) {
  constexpr int h = (p - 1) / 2;
  static_assert(h > 8 && h <= 15, "two 16 x 16 tiles");
  constexpr unsigned FULL = 0xffffffffu;
  const float magic = __int_as_float(kFxMagic);
  const int gid = lane >> 2, tig = lane & 3;
  const int nb = P / p, mp = m * p, ntile = (nb + 3) / 4;
  const float inv_m = 1.0f / (float)m;
  const int qa = 2 * tig + 1;
  const uint4* fr = reinterpret_cast<const uint4*>(frag) + 2 * lane;
  for (int tile = warp; tile < ntile; tile += nw) {
    const int bi = tile * 4 + (gid >> 1), comp = gid & 1;
    long long av[4] = {0, 0, 0, 0}, bv[4] = {0, 0, 0, 0}, v0 = 0;
    long long* pi = nullptr;
    if (bi < nb) {
      const int g = (int)(((float)bi + 0.5f) * inv_m);
      pi = reinterpret_cast<long long*>(buf + g * mp + (bi - g * m)) + comp;
      v0 = fx_scale(pi[0], d);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int q = qa + (i & 1) + 8 * (i >> 1);
        if (q <= h) {
          const long long x = fx_scale(pi[2 * q * m], d), y = fx_scale(pi[2 * (p - q) * m], d);
          av[i] = x + y;
          bv[i] = x - y;
        }
      }
    }
    long long ys = (av[0] + av[1]) + (av[2] + av[3]);
    ys += __shfl_xor_sync(FULL, ys, 1);
    ys += __shfl_xor_sync(FULL, ys, 2);
    __syncwarp();  // every load of the tile precedes its stores
    if (tig == 0 && pi) {
      pi[0] = v0 + ys;
      if (comp) fx_cover(o, fx_make(0, v0 + ys));
      else fx_cover(o, fx_make(v0 + ys, 0));
    }
    long long r[2][4];  // [A - v_0 / B][(j0 re, j0 im, j1 re, j1 im)]
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      const long long* v = part ? bv : av;
      uint32_t fx[kFxS][2];
#pragma unroll
      for (int t = 0; t < kFxS; ++t) {
        fx[t][0] = fx_digits((unsigned long long)v[0] + kFxBias, (unsigned long long)v[1] + kFxBias, t);
        fx[t][1] = fx_digits((unsigned long long)v[2] + kFxBias, (unsigned long long)v[3] + kFxBias, t);
      }
      float acc[kFxS][4];
#pragma unroll
      for (int s = 0; s < kFxS; ++s) {
        const uint4 c = fr[s * 64 + part];
#pragma unroll
        for (int t = 0; s + t < kFxS; ++t) {
          float(&ac)[4] = acc[s + t];
          if (s == 0) fx_mma(ac, c.x, c.y, c.z, c.w, fx[t][0], fx[t][1], magic, magic, magic, magic);
          else fx_mma(ac, c.x, c.y, c.z, c.w, fx[t][0], fx[t][1], ac[0], ac[1], ac[2], ac[3]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) r[part][i] = fx_undigit(acc, i);
    }
    const int bo = tile * 4 + tig;
    const long long w_re = __shfl_sync(FULL, v0, 8 * tig), w_im = __shfl_sync(FULL, v0, 8 * tig + 4);
    if (bo < nb) {
      const int g = (int)(((float)bo + 0.5f) * inv_m);
      longlong2* po = buf + g * mp + (bo - g * m);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int j = gid + 1 + 8 * i;
        if (j <= h) {
          longlong2 yj, yk;
          fx_pair(fx_make(w_re + r[0][2 * i], w_im + r[0][2 * i + 1]), fx_make(r[1][2 * i], r[1][2 * i + 1]), yj, yk);
          po[j * m] = yj;
          po[(p - j) * m] = yk;
          fx_cover(o, yj);
          fx_cover(o, yk);
        }
      }
    }
  }
}

// Radices of one kernel instance: MAXP = 8 all register butterflies, 17 and
// 31 the tensor-core ones of prime-factor plans too (TWID = false), and
// TWID with MAXP = 31 every twiddled plan with a prime above 7.
template <int MAXP, bool TWID>
__device__ __forceinline__ void fx_run_stage(int p, longlong2* buf, const uint16_t* tab, int sp, int P, int m,
                                             const int4* tw, const int4* root, const uint32_t* frag, int lane, int nl, bool dif,
                                             int d, FxMax& o) {
  switch (p) {
    case 2: fx_stage<2, TWID>(buf, tab, sp, P, m, tw, lane, nl, dif, d, o); return;
    case 3: fx_stage<3, TWID>(buf, tab, sp, P, m, tw, lane, nl, dif, d, o); return;
    case 4: fx_stage<4, TWID>(buf, tab, sp, P, m, tw, lane, nl, dif, d, o); return;
    case 5: fx_stage<5, TWID>(buf, tab, sp, P, m, tw, lane, nl, dif, d, o); return;
    case 6: fx_stage<6, TWID>(buf, tab, sp, P, m, tw, lane, nl, dif, d, o); return;
    case 7: fx_stage<7, TWID>(buf, tab, sp, P, m, tw, lane, nl, dif, d, o); return;
    default: break;
  }
  if constexpr (TWID) {
    if (p == 8) { fx_stage<8, TWID>(buf, tab, sp, P, m, tw, lane, nl, dif, d, o); return; }
  }
  if constexpr (!TWID && MAXP >= 17) {
    const int ln = lane & 31, wp = lane >> 5, nw = nl >> 5;
    switch (p) {
      case 11: fx_mma_stage<11>(buf, P, m, d, frag, ln, wp, nw, o); return;
      case 13: fx_mma_stage<13>(buf, P, m, d, frag, ln, wp, nw, o); return;
      case 17: fx_mma_stage<17>(buf, P, m, d, frag, ln, wp, nw, o); return;
      default: break;
    }
    if constexpr (MAXP == 31) {
      switch (p) {
        case 19: fx_mma_stage_wide<19>(buf, P, m, d, frag, ln, wp, nw, o); return;
        case 23: fx_mma_stage_wide<23>(buf, P, m, d, frag, ln, wp, nw, o); return;
        case 29: fx_mma_stage_wide<29>(buf, P, m, d, frag, ln, wp, nw, o); return;
        case 31: fx_mma_stage_wide<31>(buf, P, m, d, frag, ln, wp, nw, o); return;
        default: break;
      }
    }
  }
  if constexpr (TWID && MAXP == 31) fx_stage_any(buf, P, p, m, tw, root, lane, nl, dif, d, o);
}

// The left shift that brings values covered by the high-word bits o (below
// 2^30) to just below 2^62.
__device__ __forceinline__ int fx_headroom(unsigned o) { return o ? __clz((int)o) - 2 : 30; }

// Barrier number first + i (i < COUNT <= 6) for N threads, with immediate
// ids: a block then holds only the hardware barriers it names.
template <int ID, int N>
__device__ __forceinline__ void fx_bar() {
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
template <int N, int COUNT, int FIRST>
__device__ __forceinline__ void fx_bar_of(int i) {
  static_assert(COUNT <= 6, "six barriers at most");
  if (COUNT > 5 && i == 5) fx_bar<FIRST + 5, N>();
  else if (COUNT > 4 && i == 4) fx_bar<FIRST + 4, N>();
  else if (COUNT > 3 && i == 3) fx_bar<FIRST + 3, N>();
  else if (COUNT > 2 && i == 2) fx_bar<FIRST + 2, N>();
  else if (COUNT > 1 && i == 1) fx_bar<FIRST + 1, N>();
  else fx_bar<FIRST, N>();
}

// Per-line scratch of the kernel: reduction slots of the two halves (the
// magnitudes' in two sets, used by turns), what the halves exchange, and the
// velocity maxima.
template <int S>
struct alignas(16) FxLine {
  unsigned eb[2][S][2];
  unsigned mx[2][2][S][2];
  unsigned prod[2 * S][2];
  int head[2][2], exp[2][2], bad[2];
  unsigned long long umax[2];
};

// ---------------------------------------------------------------------------
// Nonlinear pass (Nr_maxLOOP, src/nonlin.F90:55-86).  A radial line (r, b)
// takes 2 S warps: one half transforms T + i omega, the other u_phi + i u_r
// (two complex FFTs of length P, each carrying two real fields), the halves
// meet for the four grid products, and each half transforms two of them
// back: u_phi T + i u_r T, and u_phi omega + i u_r omega, truncated to modes
// 0..Nm and divided by P.
//
// Values are integers, |V| < 2^61, each of the two packed fields at its own
// power of two (59 bits from the largest exponent of its line, so neither
// loses digits to the other's magnitude) and both shifted together before a
// stage by what its growth can take, from the largest value of the stage
// before.  The grid values are shifted up to 62 bits (by the largest of each
// field) before they are multiplied.  Every sum is exact; errors are those
// of the truncation going in, the products with constants (half a unit rms each)
// and the grid products' low x low terms (a quarter unit).  All the maxima behind
// the scales are integers, so results do not depend on S.  A line with an
// Inf or NaN input gives NaN.
//
// Bound: issue of integer instructions (about half of the cycles) and their
// latency at the 16 warps an SM that registers and shared memory allow.
// Against FP64 butterflies on grids of 3 Nm points (radix 11 to 31 on the
// tensor cores), us of the kernel for Nr = 65, Nm = 170, 128 instances: 1085 -> 222;
// of a call for Nr = 129, Nm = 512, 8: 751 -> 153; one instance of Nr = 33, Nm = 341:
// 95 -> 23.
// The error against 64 bits fell from 7e-16 to 4e-16 (products with omega)
// and from 7e-14 to 4e-16 (with T, which FP64 packed with a larger omega).
// ---------------------------------------------------------------------------
template <int MAXP, bool TWID, int S, int LPB, int MINB>
__global__ void __launch_bounds__(64 * S * LPB, MINB) nonlin_kernel(NonlinArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int NH = 32 * S;  // threads of a half
  const int P = a.plan.P, M = a.M, B = a.B, Nm = a.Nm;
  const int PP = a.plan.rad[0] * a.plan.span[0], inner = a.plan.rad[a.plan.nrad - 1];
  int4* tw = reinterpret_cast<int4*>(smem_raw);
  longlong2* bufs = reinterpret_cast<longlong2*>(tw + (TWID ? P - inner : 0));
  FxLine<S>* lines = reinterpret_cast<FxLine<S>*>(bufs + (size_t)LPB * 2 * PP);
  uint32_t* frag = reinterpret_cast<uint32_t*>(lines + LPB);
  int nfrag = 0;
  if constexpr (!TWID && MAXP >= 17) {
    for (int i = 0; i < a.plan.nrad; ++i) {
      const uint32_t* src = nullptr;
      switch (a.plan.rad[i]) {
        case 11: src = kFxFrag<11>.v; break;
        case 13: src = kFxFrag<13>.v; break;
        case 17: src = kFxFrag<17>.v; break;
        default: break;
      }
      if constexpr (MAXP == 31) {
        switch (a.plan.rad[i]) {
          case 19: src = kFxFrag<19>.v; break;
          case 23: src = kFxFrag<23>.v; break;
          case 29: src = kFxFrag<29>.v; break;
          case 31: src = kFxFrag<31>.v; break;
          default: break;
        }
      }
      const int n = fx_frag_ints(a.plan.rad[i]);
      for (int k = threadIdx.x; k < n; k += blockDim.x) frag[nfrag + k] = src[k];
      nfrag += n;
    }
  }
  uint16_t* pos = reinterpret_cast<uint16_t*>(frag + nfrag);  // places of the spectrum and of the line's points
  uint16_t* tab = pos + P;
  for (int i = threadIdx.x; i < P; i += blockDim.x) {
    if (TWID && i < P - inner) tw[i] = a.tw[i];
    const unsigned both = a.pos[i];
    pos[i] = (uint16_t)both;
    tab[i] = (uint16_t)(both >> 16);
  }
  __syncthreads();
  const int lw = threadIdx.x / (2 * NH), lt = threadIdx.x - lw * 2 * NH;  // line of the block, thread of the line
  const int half = lt / NH, hl = lt - half * NH, lane = threadIdx.x & 31, hw = hl >> 5;
  const int line = blockIdx.x * LPB + lw;
  if (line >= a.R * B) return;
  // barriers of a half and of a line (immediate ids: a block then holds
  // only the hardware barriers it names)
  auto half_sync = [&]() {
    if constexpr (S == 1) {
      __syncwarp();
    } else {
      fx_bar_of<NH, (S > 1 ? 2 * LPB : 1), 1>(2 * lw + half);
    }
  };
  auto line_sync = [&]() { fx_bar_of<2 * NH, LPB, (S > 1 ? 2 * LPB : 0) + 1>(lw); };
  FxLine<S>& L = lines[lw];
  longlong2* bufA = bufs + (size_t)lw * 2 * PP;
  longlong2* bufB = bufA + PP;
  longlong2* buf = half ? bufB : bufA;
  const size_t row = (size_t)(line / B) * M * B + line % B;
  const double2* X = (half ? a.up : a.t) + row;
  const double2* Y = (half ? a.ur : a.w) + row;

  // The half's two fields: the first kHeld modes of a thread are read once
  // and held, longer spectra are read again for the conversion.
  constexpr int kHeld = 6;
  double2 xs[kHeld], ys[kHeld];
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    const int k = hl + i * NH;
    xs[i] = ys[i] = make_double2(0.0, 0.0);
    if (k <= Nm) {
      xs[i] = __ldg(X + (size_t)k * B);
      ys[i] = __ldg(Y + (size_t)k * B);
    }
  }
  if (hl == 0) xs[0].y = ys[0].y = 0.0;  // only Re of mode 0 counts, as in a c2r transform
  // The grid of 3 Nm points folds mode 2 Nm of a product, f_Nm g_Nm, onto
  // mode -Nm: its conjugate onto mode Nm.  Lane i < 4 of the half adds
  // component i of the two products' (re, im).
  const bool alias = P != 3 * Nm;
  double fold = 0.0;
  if (alias && hl < 4) {
    const size_t e = row + (size_t)Nm * B;
    const double2 F = __ldg((half ? a.w : a.t) + e), G = __ldg((hl < 2 ? a.up : a.ur) + e);
    fold = (hl & 1) ? -(F.x * G.y + F.y * G.x) : F.x * G.x - F.y * G.y;
  }
  // the largest high word of each field's magnitudes: its biased exponent, 0
  // for a field of zeros
  unsigned ex = 0, ey = 0;
  auto high = [](double2 v) {
    return max((unsigned)__double2hiint(v.x) & 0x7fffffffu, (unsigned)__double2hiint(v.y) & 0x7fffffffu);
  };
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    ex = max(ex, high(xs[i]));
    ey = max(ey, high(ys[i]));
  }
  for (int k = hl + kHeld * NH; k <= Nm; k += NH) {
    ex = max(ex, high(__ldg(X + (size_t)k * B)));
    ey = max(ey, high(__ldg(Y + (size_t)k * B)));
  }
  ex = __reduce_max_sync(FULL, ex);
  ey = __reduce_max_sync(FULL, ey);
  if constexpr (S > 1) {
    if (lane == 0) { L.eb[half][hw][0] = ex; L.eb[half][hw][1] = ey; }
    half_sync();
#pragma unroll
    for (int i = 0; i < S; ++i) { ex = max(ex, L.eb[half][i][0]); ey = max(ey, L.eb[half][i][1]); }
  }
  const bool bad = ex >= 0x7ff00000u || ey >= 0x7ff00000u;
  // products with a field of zeros are zeros: whatever the other field packed
  // with it leaves there, an exponent below all numbers
  const int zx = ex ? 0 : 1 << 20, zy = ey ? 0 : 1 << 20;
  ex = bad ? 4095u : max(ex >> 20, 1u);  // (4095: every value shifts to zero)
  ey = bad ? 4095u : max(ey >> 20, 1u);
  // Scatter conj(Z) at digit-reversed positions, Z_k = X_k + i Y_k for the
  // Hermitian spectra X, Y of two real lines.  IFFT(Z) = conj(FFT(conj(Z))).
  auto scatter = [&](int k, double2 x, double2 y) {
    auto fix = [&](double v, unsigned eb) -> long long {
      const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
      const unsigned long long t = fx_mag_of(bits, (int)eb);
      return (long long)bits < 0 ? -(long long)t : (long long)t;
    };
    const long long xr = fix(x.x, ex), yr = fix(y.x, ey), xi = fix(x.y, ex), yi = fix(y.y, ey);
    buf[pos[k]] = fx_make(xr - yi, -(xi + yr));
    if (k) buf[pos[P - k]] = fx_make(xr + yi, xi - yr);
  };
#pragma unroll
  for (int i = 0; i < kHeld; ++i)
    if (hl + i * NH <= Nm) scatter(hl + i * NH, xs[i], ys[i]);
  for (int k = hl + kHeld * NH; k <= Nm; k += NH) scatter(k, __ldg(X + (size_t)k * B), __ldg(Y + (size_t)k * B));
  for (int k = Nm + 1 + hl; k < P - Nm; k += NH) buf[pos[k]] = fx_make(0, 0);
  half_sync();
  // values are V 2^(E + e), e = ex - 1022 - 59 for the first field, ey - ...
  // for the second; every component is below 2^60
  int E = 0, bits = 60, turn = 0;
  FxMax o{0, 0};
  auto stage = [&](int s, int m, const uint32_t* fr, const int4* root, bool dif) {
    const int p = a.plan.rad[s];
    const int d = bits + fx_growth(p) - 61;
    E += d;
    o = FxMax{0, 0};
    fx_run_stage<MAXP, TWID>(p, buf, tab, a.plan.span[s], P, m, tw + (m - inner), root, fr, hl, NH, dif, d, o);
    o.x = __reduce_or_sync(FULL, o.x);
    o.y = __reduce_or_sync(FULL, o.y);
    if constexpr (S > 1) {
      if (lane == 0) { L.mx[turn][half][hw][0] = o.x; L.mx[turn][half][hw][1] = o.y; }
      half_sync();
#pragma unroll
      for (int i = 0; i < S; ++i) { o.x |= L.mx[turn][half][i][0]; o.y |= L.mx[turn][half][i][1]; }
      turn ^= 1;
    } else {
      __syncwarp();
    }
    bits = fx_bits(o.x | o.y);
  };
  {  // DIT: radices processed innermost first
    int m = 1, f = nfrag;
    const int4* root = a.tw + fx_table_size(a.plan);
    for (int s = a.plan.nrad - 1; s >= 0; --s) {
      const int p = a.plan.rad[s];
      f -= fx_frag_ints(p);
      root -= fx_root_size(a.plan, p);
      stage(s, m, frag + f, root, false);
      m *= p;
    }
  }
  if (hl == 0) {
    L.head[half][0] = fx_headroom(o.x);
    L.head[half][1] = fx_headroom(o.y);
    L.exp[half][0] = E + (int)ex - 1081 - zx;
    L.exp[half][1] = E + (int)ey - 1081 - zy;
    L.bad[half] = bad;
    L.umax[half] = 0;
  }
  line_sync();
  // Grid values: bufA = conj(t + i omg) -> t = A.x, omg = -A.y; likewise for
  // (u_phi, u_r) in bufB.  Products, in natural order for the DIF.
  const int ht = L.head[0][0], ho = L.head[0][1], hp = L.head[1][0], hr = L.head[1][1];
  const int e_half = L.exp[0][half] - (half ? ho : ht) + 64;  // of T, omega (in the products of this half)
  const int e1 = e_half + L.exp[1][0] - hp, e2 = e_half + L.exp[1][1] - hr;
  const bool any_bad = L.bad[0] || L.bad[1];
  unsigned long long urmax = 0, upmax = 0;
  FxMax oA{0, 0}, oB{0, 0};
  for (int j = lt; j < P; j += 2 * NH) {
    const int at = tab[j];
    const longlong2 za = bufA[at], zb = bufB[at];
    const long long tt = za.x << ht, om = -(za.y << ho), up = zb.x << hp, ur = -(zb.y << hr);
    const longlong2 pa = fx_make(fx_mulhi(up, tt), fx_mulhi(ur, tt)), pb = fx_make(fx_mulhi(up, om), fx_mulhi(ur, om));
    bufA[at] = pa;
    bufB[at] = pb;
    fx_cover(oA, pa);
    fx_cover(oB, pb);
    if (a.umax) {  // only when the CFL inputs are read
      urmax = max(urmax, (unsigned long long)(zb.y < 0 ? -zb.y : zb.y));
      upmax = max(upmax, (unsigned long long)(zb.x < 0 ? -zb.x : zb.x));
    }
  }
  const unsigned ma = __reduce_or_sync(FULL, oA.x | oA.y), mb = __reduce_or_sync(FULL, oB.x | oB.y);
  if (lane == 0) { L.prod[lt >> 5][0] = ma; L.prod[lt >> 5][1] = mb; }
  if (a.umax) {
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
      urmax = max(urmax, __shfl_xor_sync(FULL, urmax, w));
      upmax = max(upmax, __shfl_xor_sync(FULL, upmax, w));
    }
    if (lane == 0) {
      atomicMax(&L.umax[0], urmax);
      atomicMax(&L.umax[1], upmax);
    }
  }
  line_sync();
  if (a.umax && lt == 0) {
    a.umax[2 * (size_t)line] = L.bad[1] ? 0.0 : ldexp((double)L.umax[0], L.exp[1][1]);
    a.umax[2 * (size_t)line + 1] = L.bad[1] ? 0.0 : ldexp((double)L.umax[1], L.exp[1][0]);
  }
  {
    unsigned w = 0;
#pragma unroll
    for (int i = 0; i < 2 * S; ++i) w |= L.prod[i][half];
    bits = fx_bits(w);
  }
  E = 0;
  {  // DIF: outermost radix first
    int m = P, f = 0;
    const int4* root = a.tw + P;
    for (int s = 0; s < a.plan.nrad; ++s) {
      const int p = a.plan.rad[s];
      m /= p;
      stage(s, m, frag + f, root, true);
      f += fx_frag_ints(p);
      root += fx_root_size(a.plan, p);
    }
  }
  // Split the two-for-one spectra: X_k = (Z_k + conj Z_{P-k})/2,
  // Y_k = (Z_k - conj Z_{P-k})/(2i), then divide by P: an odd P's factor in
  // fixed point, the power of two in the exponent
  const int sh = 31 - __clz(P), odd = P & (P - 1);  // P = 2^sh (1 + ...)
  const FxC over = a.over_p;                          // 2^sh / P
  const int x1 = e1 + E - sh - 1, x2 = e2 + E - sh - 1;
  double* o1 = reinterpret_cast<double*>((half ? a.nwp : a.ntp) + row);
  double* o2 = reinterpret_cast<double*>((half ? a.nwr : a.ntr) + row);
  auto part = [&](int k, int i) {  // component i of mode k's (u, v) as an integer
    const longlong2 z = buf[pos[k]], c = buf[pos[k == 0 ? 0 : P - k]];
    const long long v = i == 0 ? z.x + c.x : i == 1 ? z.y - c.y : i == 2 ? z.y + c.y : c.x - z.x;
    return odd ? fx_mul(fx_prep(v >> 1), over) * 2 : v;
  };
  const int last = alias ? Nm - 1 : Nm;
  if (!any_bad && min(x1, x2) > -960 && max(x1, x2) < 960) {  // every result is a normal number or zero
    auto to_double = [&](long long v, int x) {
      const double r = (double)v;
      return v ? __hiloint2double(__double2hiint(r) + (x << 20), __double2loint(r)) : 0.0;
    };
    for (int k = hl; k <= last; k += NH) {
      const size_t e = (size_t)k * B;
      reinterpret_cast<double2*>(o1)[e] = make_double2(to_double(part(k, 0), x1), to_double(part(k, 1), x1));
      reinterpret_cast<double2*>(o2)[e] = make_double2(to_double(part(k, 2), x2), to_double(part(k, 3), x2));
    }
    if (alias && hl < 4)
      (hl < 2 ? o1 : o2)[2 * (size_t)Nm * B + (hl & 1)] = to_double(part(Nm, hl), hl < 2 ? x1 : x2) + fold;
  } else {
    for (int k = hl; k <= Nm; k += NH)
      for (int i = 0; i < 4; ++i)
        (i < 2 ? o1 : o2)[2 * (size_t)k * B + (i & 1)] =
            any_bad ? __longlong_as_double(0x7ff8000000000000LL) : ldexp((double)part(k, i), i < 2 ? x1 : x2);
    half_sync();
    if (alias && hl < 4) (hl < 2 ? o1 : o2)[2 * (size_t)Nm * B + (hl & 1)] += fold;
  }
}

template <int MAXP, bool TWID, int S, int LPB, int MINB>
static cudaError_t launch_nonlin_s(const NonlinArgs& a, cudaStream_t s) {
  const int P = a.plan.P;
  if (P > kMaxLine) return cudaErrorInvalidValue;
  int frag = 0;
  if (!TWID)
    for (int i = 0; i < a.plan.nrad; ++i) frag += fx_frag_ints(a.plan.rad[i]);
  const int PP = a.plan.rad[0] * a.plan.span[0];
  const int smem = (TWID ? P - a.plan.rad[a.plan.nrad - 1] : 0) * 16 + LPB * (2 * PP * 16 + (int)sizeof(FxLine<S>)) +
                   4 * (frag + (P + 3) / 4 * 4);
  // the limit only rises: a thread with a shorter line never takes it from one
  // that is about to launch a longer
  static std::mutex mu;
  static int limit[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  {
    std::lock_guard<std::mutex> lk(mu);
    int& most = limit[dev >= 0 && dev < 64 ? dev : 0];
    most = std::max(most, smem);
    const cudaError_t e = cudaFuncSetAttribute(nonlin_kernel<MAXP, TWID, S, LPB, MINB>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, most);
    if (e != cudaSuccess) return e;
  }
  nonlin_kernel<MAXP, TWID, S, LPB, MINB><<<(a.R * a.B + LPB - 1) / LPB, 64 * S * LPB, smem, s>>>(a);
  return cudaGetLastError();
}

}  // namespace
}  // namespace falcon
