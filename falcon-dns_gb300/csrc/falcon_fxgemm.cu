// Operator contractions Y = alpha A X in 60-bit fixed point on integer
// multiply-adds.
//
// GB300's FP64 pipe takes 64 cycles per warp instruction and sub-partition,
// its 32 x 32 + 64-bit multiply-add 5, so a product of two such numbers in
// three of those is 4 times cheaper than an FMA.  An operator row and an X
// column are taken as integers at the scale of their largest element (|a| <
// 2^e: a 2^(60 - e) rounded, exact for elements within 2^7 of it), split as h
// 2^30 + l with l signed.  Per product
//   ha hx 2^60 + (ha lx + la hx) 2^30
// is summed in two 64-bit integers and a word for the first one's carries
// (|h| <= 2^30 and |l| <= 2^29: exact for 7 products between carries).  la lx is
// left out: 2^-62 of the largest product at most, what the operands' rounding
// leaves out.  The sum is rounded once to FP64.  Sums of integers do not depend
// on their order, so results depend neither on the tile nor on the launch: the
// tile and the narrow kernel give the same bits.  A column (or row) with an Inf
// or NaN gives NaN.
//
// Operators weigh the rows of X very differently: the radial derivatives and
// their products with a field are largest at the walls (by n^2 for d/dr, n^4
// for the Laplacian), the solve operators smallest, where their right-hand sides
// are largest.  With one scale for a row the small elements, which meet the
// large values of fields that vanish at the walls, lose their digits; with
// columns divided by their largest element and X's rows multiplied, X's values
// away from the walls lose theirs.  So columns are divided by 2^w_k, w_k half the
// largest element's exponent, and the spread is shared.  A column of zeros
// weighs nothing, whatever X has there.
//
// Errors over the norm of a column's output against 64 bits (FP64 sums, this
// form; a form of 58 x 59 bits, truncated, with weights of 0 for the derivatives
// and 1 for the solves): d/dr of (1 - x^2)^2 f(x), 129 points, 1.2e-15, 1.4e-16
// (3e-14); the Laplacian of f(x) 2e-11, 1e-12 (3e-11), of (1 - x^2)^2 f(x) 8e-14,
// 6e-14 (3e-11); the vorticity solve of a run 5.7e-16, 1.3e-16 (2.7e-16).
//
// Bound: latency for the narrow forms (the radial and per-mode products of a
// few instances), the integer multiply-add pipe for the tiles.  FP64 FMA -> this, us
// with L2 cold: 97 x 97, 342 modes, 2 columns 22 -> 18, 1026 modes, 6 columns 180 ->
// 53; 33 x 33, 43 modes, 2 columns 12 -> 8; 65 x 65, 688 columns 15 -> 12, 43776
// columns 317 -> 123 (84 on tcgen05, which the autotuner takes there); 129 x 129,
// 11040 columns 324 -> 127.  (With 58 and 59 bits and carries every 16 k the large
// ones took 114 and 120; with carries every 4 k 126 and 129.)
//
// The operators' integers are made once per operator set
// (launch_fx_operator); X is converted by each block for its own columns.
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <unordered_map>

#include "falcon_fixed.h"
#include "falcon_internal.h"

namespace falcon {
namespace {

constexpr int kBits = 60, kLow = 30;      // of a row's and a column's integers, of their low halves
constexpr int kCarry = 7;                 // products between carries, at most
constexpr int kFollowRows = 6;           // deepest tiles that do what follows a product (deeper ones would spill)
constexpr int kFxKC = 2 * kCarry;         // k per staged operator chunk
constexpr int kBad = INT32_MIN;          // exponent of a row or column with an Inf or NaN
constexpr int kNone = -100000;           // exponent of a zero
constexpr int kNoWeight = -30000;        // of a column of zeros: below every other

// e with |a 2^w| < 2^e (kNone for a zero, INT32_MAX for Inf and NaN)
__device__ __forceinline__ int exponent_of(double a, int w) {
  const unsigned high = (unsigned)__double2hiint(a) & 0x7fffffffu;
  if (high >= 0x7ff00000u) return INT32_MAX;
  if (high == 0u && __double2loint(a) == 0) return kNone;
  return (int)max(high >> 20, 1u) - 1022 + w;
}
__device__ __forceinline__ int2 signed_split(unsigned long long t) {
  return make_int2((int)((long long)t >> kLow) + (int)((unsigned)t >> (kLow - 1) & 1),
                   (int)((unsigned)t << (32 - kLow)) >> (32 - kLow));
}
// a 2^w 2^(kBits - e) rounded, split into (h, l signed)
__device__ __forceinline__ int2 split_of(double a, int w, int e) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(a);
  const int eb = (int)(bits >> 52) & 0x7ff;
  const unsigned long long m = ((bits & 0xfffffffffffffULL) | (eb ? 1ULL << 52 : 0ULL)) << (kBits - 53);
  const unsigned sh = min((unsigned)(e - w + 1022 - max(eb, 1)), kBits + 1u);  // (negative only for a zero)
  unsigned long long t = (m + (1ULL << sh >> 1)) >> sh;
  if ((long long)bits < 0) t = 0ull - t;
  return signed_split(t);
}
// The scale of a row or column whose largest exponent is m, and its exponent.
__device__ __forceinline__ int scale_of(int m) { return m == INT32_MAX ? 100000 : m == kNone ? 0 : m; }
__device__ __forceinline__ int mark_of(int m) { return m == INT32_MAX ? kBad : scale_of(m); }

struct Sum {
  int top;  // top 2^40 + hh
  long long hh, mid;
};
// a b + c as one instruction (a product and a 64-bit add on two pipes, as the
// compiler makes of mad.wide, took 131 us for 65 x 65 x 43776 where this took
// 119, with a fourth multiply-add per product)
__device__ __forceinline__ long long madw1(int a, int b, long long c) {
  long long r;
  asm("{\n\t.reg .u32 lo, hi;\n\tmov.b64 {lo, hi}, %3;\n\tmad.lo.cc.s32 lo, %1, %2, lo;\n\t"
      "madc.hi.s32 hi, %1, %2, hi;\n\tmov.b64 %0, {lo, hi};\n\t}"
      : "=l"(r)
      : "r"(a), "r"(b), "l"(c));
  return r;
}
__device__ __forceinline__ void add_product(Sum& s, int2 a, int2 x) {
  s.hh = madw1(a.x, x.x, s.hh);
  s.mid = madw1(a.x, x.y, s.mid);
  s.mid = madw1(a.y, x.x, s.mid);
}
__device__ __forceinline__ void carry(Sum& s) {
  s.hh += s.mid >> kLow;
  s.mid &= (1 << kLow) - 1;
  s.top += (int)(s.hh >> 40);
  s.hh &= (1LL << 40) - 1;
}
// A sum as hi 2^64 + lo, in units of 2^(kLow - 2 kBits) of the scales.
struct alignas(16) Wide {
  long long hi;
  unsigned long long lo;
};
__device__ __forceinline__ Wide wide_of(Sum s) {
  carry(s);
  return {((long long)s.top << (40 + kLow - 64)) + (s.hh >> (64 - kLow)),
          ((unsigned long long)s.hh << kLow) | (unsigned long long)s.mid};
}
__device__ __forceinline__ Wide add(Wide a, Wide b) {
  const unsigned long long lo = a.lo + b.lo;
  return {a.hi + b.hi + (lo < b.lo), lo};
}
__device__ __forceinline__ Wide sub(Wide a, Wide b) {
  return {a.hi - b.hi - (a.lo < b.lo), a.lo - b.lo};
}
__device__ __forceinline__ Wide add(Wide a, long long b) { return add(a, Wide{b >> 63, (unsigned long long)b}); }
// RN of the sum times 2^(ea + ex)
__device__ __forceinline__ double value_of(Wide s, int ea, int ex, double alpha) {
  if (ea == kBad || ex == kBad) return __longlong_as_double(0x7ff8000000000000LL);
  long long v = (long long)s.lo;
  int e = ea + ex + kLow - 2 * kBits;
  if (s.hi != v >> 63) {  // the leading 64 bits, and whether others are set
    const int up = __clzll(s.hi ^ (s.hi >> 63)) - 1;
    v = (s.hi << up) | (long long)(s.lo >> (64 - up)) | (long long)((s.lo << up) != 0);
    e += 64 - up;
  }
  double y = (double)v;
  if (v) {
    const int top = ((__double2hiint(y) >> 20) & 0x7ff) + e;
    y = top > 0 && top < 2047 ? __hiloint2double(__double2hiint(y) + (e << 20), __double2loint(y)) : ldexp(y, e);
  }
  return alpha == 1.0 ? y : alpha * y;
}

__device__ __forceinline__ double* output_row(const GemmArgs& g, int z, int row) {
  if (g.nout == 0) return g.Y + (size_t)z * g.sY + (size_t)row * g.ldy;
  int o = 0;
  while (o + 1 < g.nout && row >= g.rend[o]) ++o;
  return g.Yo[o] + (size_t)z * g.sY + (size_t)(row - (o ? g.rend[o - 1] : 0)) * g.ldy;
}

// After output row `row` of entry z of a product, columns n (even), n + 1.
__device__ __forceinline__ void follow_row(const FxFollow& f, int b0, int z, int row, int n, double y0, double y1) {
  const int b = b0 + (n >> 1);
  if (f.kind == kBuoyancy) follow_buoyancy(f, f.m0 + z, row, b, y0, y1);
  if (f.kind == kVelocity && row >= f.R && row < 2 * f.R) follow_velocity(f, f.m0 + z, row - f.R, b, y0, y1);
}
// The grid's share of mode 0.
__device__ __forceinline__ void follow_modes(const FxFollow& f) {
  if (f.kind != kVelocity) return;
  const int nthr = blockDim.x, blk = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  const int step = gridDim.x * gridDim.y * gridDim.z * nthr;
  for (int i = blk * nthr + threadIdx.x; i < f.R * f.B; i += step) follow_mode0(f, i / f.B, i % f.B);
}

__device__ __forceinline__ void copy4(void* dst, const void* src) {
  const unsigned saddr = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(saddr), "l"(src) : "memory");
}
__device__ __forceinline__ void copy8(void* dst, const void* src, bool valid) {
  const unsigned saddr = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(saddr), "l"(src), "r"(valid ? 8 : 0) : "memory");
}

__device__ __forceinline__ void copy16(void* dst, const void* src, bool valid) {
  const unsigned saddr = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(saddr), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// One warp per (entry, column k): half the exponent of its largest element.
__global__ void fx_weight_kernel(const double* A, long lda, long sA, int rows, int K, int nb, int* wk) {
  const long t = (blockIdx.x * (long)blockDim.x + threadIdx.x) >> 5;
  if (t >= (long)nb * K) return;
  const int z = (int)(t / K), k = (int)(t - (long)z * K);
  const double* a = A + (size_t)z * sA + (size_t)k * lda;
  int m = kNone;
  for (int r = threadIdx.x & 31; r < rows; r += 32) {
    const int e = exponent_of(a[r], 0);
    if (e != INT32_MAX) m = max(m, e);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) wk[t] = m == kNone ? kNoWeight : m >> 1;
}

// Eight threads per (entry, row): the row's exponent, then its integers, in the
// operator's own layout.  (One thread a row waited for 2 K loads one after
// another: 40 us an operator of 65 points.)
__global__ void __launch_bounds__(256) fx_operator_kernel(const double* A, long lda, long sA, int rows, int K, int nb,
                                                          const int* wk, int2* out, int* ex) {
  __shared__ int part[8][32];
  const long t = blockIdx.x * 32L + threadIdx.x;
  const bool act = t < (long)nb * rows;
  const int z = act ? (int)(t / rows) : 0, r = act ? (int)(t - (long)z * rows) : 0;
  const double* a = A + (size_t)z * sA + r;
  const int* w = wk + (size_t)z * K;
  int m = kNone;
  if (act)
    for (int k = threadIdx.y; k < K; k += 8) m = max(m, exponent_of(a[(size_t)k * lda], -w[k]));
  part[threadIdx.y][threadIdx.x] = m;
  __syncthreads();
  if (!act) return;
  for (int i = 0; i < 8; ++i) m = max(m, part[i][threadIdx.x]);
  if (threadIdx.y == 0) ex[(size_t)z * lda + r] = mark_of(m);
  int2* o = out + (size_t)z * sA + r;
  for (int k = threadIdx.y; k < K; k += 8) o[(size_t)k * lda] = split_of(a[(size_t)k * lda], -w[k], scale_of(m));
}

// X panel of a block in shared memory, xs[k * (ncol + PAD) + c] (staged as
// doubles, complete when this is called): column exponents in cex, integers in
// place.  w: the operator's weights, staged with it (or null: fwd); part:
// blockDim.x words; spare: leading bits left free.
template <int PAD = 0>
__device__ __forceinline__ void convert_panel(double* xs, int K, int ncol, const int* w, int* cex, int* part,
                                              int spare = 0) {
  const int tid = threadIdx.x, J = blockDim.x / ncol, c = tid % ncol, j = tid / ncol, st = ncol + PAD;
  const bool act = j < J;
  int m = kNone;
  if (act) {
    for (int k = j; k < K; k += J) m = max(m, exponent_of(xs[k * st + c], w ? w[k] : 0));
    part[tid] = m;
  }
  __syncthreads();
  if (act) {
    for (int i = 0; i < J; ++i) m = max(m, part[i * ncol + c]);
    if (m != INT32_MAX && m != kNone) m += spare;
    if (j == 0) cex[c] = mark_of(m);
    for (int k = j; k < K; k += J) {
      const int2 v = split_of(xs[k * st + c], w ? w[k] : 0, scale_of(m));
      reinterpret_cast<int2*>(xs)[k * st + c] = v;
    }
  }
  __syncthreads();
}

// Tile: a block covers NCOL columns and nw * RG * RPT rows, RG = 64 / NCOL;
// lane = (row group rg, column pair cp).  The X panel (all of K) stays in
// shared memory, the operator is staged in double-buffered chunks of 14 k.
// With g.njobs, several products of one shape (rows, K) in one launch: the
// grid's column blocks run through the jobs.
template <int RPT, int NCOL>
__global__ void __launch_bounds__(512) fx_tile_kernel(const __grid_constant__ GemmArgs g) {
  constexpr int RG = 64 / NCOL, CP = NCOL / 2;
  extern __shared__ __align__(16) double fsm[];
  const int nthr = blockDim.x, nw = nthr >> 5;
  const int rows_blk = nw * RG * RPT;
  double* xs = fsm;                                                   // [K][NCOL]
  int2* as = reinterpret_cast<int2*>(fsm + (size_t)g.K * NCOL);       // [2][kFxKC][rows_blk]
  int* cex = reinterpret_cast<int*>(as + 2 * kFxKC * rows_blk);       // [NCOL]
  int* part = cex + NCOL;                                             // [nthr]
  int* ws = part + nthr;                                              // [K]
  const int z = blockIdx.z;
  int N = g.N, nblk = blockIdx.x, e = z, b0 = g.follow.b0;
  const int nz = g.nsub ? g.nsub * g.batch : g.batch;
  long lda = g.lda, ldx = g.ldx, ldy = g.ldy;
  const int2* A = g.fx + (size_t)z * g.sA;
  const int* aex = g.fx_ex + (size_t)z * g.lda;
  const int* w = g.fx_w + (size_t)z * g.K;
  const double* X = g.X + (size_t)z * g.sX;
  double* Y = nullptr;
  if (g.njobs || g.nsub || z >= nz) {
    int j = 0;
    e = 0;
    if (g.njobs) {
      for (int nb; nblk >= (nb = (g.job[j].N + NCOL - 1) / NCOL); ++j) nblk -= nb;
    } else if (z < nz) {
      j = z / g.batch;
      e = z - j * g.batch;
    } else {
      j = g.nsub + z - nz;
    }
    const FxJob& q = g.job[j];
    N = q.N;
    lda = q.lda;
    ldx = q.ldx;
    ldy = q.ldy;
    A = q.fx + (size_t)e * g.sA;
    aex = q.fx_ex + (size_t)e * lda;
    w = q.fx_w + (size_t)e * g.K;
    X = q.X + (size_t)e * g.sX;
    Y = q.Y + (size_t)e * g.sY;
    b0 = q.b0;
    if (nblk * NCOL >= N) return;  // a narrower product than the launch's
  }
  const int n0 = nblk * NCOL, row0 = blockIdx.y * rows_blk;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rg = lane / CP, cp = lane - rg * CP;
  const int rw = (warp * RG + rg) * RPT;
  for (int k = threadIdx.x; k < g.K; k += nthr) copy4(ws + k, w + k);
  {
    constexpr int KW = NCOL >= 32 ? 1 : 32 / NCOL, HW = NCOL >= 32 ? NCOL / 32 : 1;  // k, column halves per warp
    for (int i = warp; i < (g.K + KW - 1) / KW * HW; i += nw) {
      const int k = (i / HW) * KW + (NCOL >= 32 ? 0 : lane / NCOL), c = (i % HW) * 32 + (NCOL >= 32 ? lane : lane % NCOL);
      if (k < g.K) {
        const bool ok = n0 + c < N;
        copy8(xs + k * NCOL + c, ok ? X + (size_t)k * ldx + n0 + c : X, ok);
      }
    }
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  auto issue = [&](int k0, int2* buf) {
    const int kc = min(kFxKC, g.K - k0);
    for (int kk = warp; kk < kc; kk += nw)
      for (int rr = lane; rr < rows_blk; rr += 32) {
        const bool ok = row0 + rr < g.rows;
        copy8(buf + kk * rows_blk + rr, ok ? A + (size_t)(k0 + kk) * lda + row0 + rr : A, ok);
      }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  issue(0, as);
  asm volatile("cp.async.wait_group 1;\n" ::: "memory");
  __syncthreads();
  convert_panel(xs, g.K, NCOL, ws, cex, part);
  Sum acc[RPT][2];
#pragma unroll
  for (int i = 0; i < RPT; ++i) acc[i][0] = acc[i][1] = Sum{0, 0, 0};
  int cur = 0;
  for (int k0 = 0; k0 < g.K; k0 += kFxKC) {
    const int kc = min(kFxKC, g.K - k0);
    if (k0 + kFxKC < g.K) {
      issue(k0 + kFxKC, as + (cur ^ 1) * kFxKC * rows_blk);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const int2* Aw = as + cur * kFxKC * rows_blk + rw;
    const int4* Xw = reinterpret_cast<const int4*>(xs + (size_t)k0 * NCOL) + cp;
    auto one = [&](int kk) {
      const int4 xv = Xw[kk * (NCOL / 2)];
      const int2 x0 = make_int2(xv.x, xv.y), x1 = make_int2(xv.z, xv.w);
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int2 av = Aw[kk * rows_blk + i];
        add_product(acc[i][0], av, x0);
        add_product(acc[i][1], av, x1);
      }
    };
    for (int k4 = 0; k4 < kc; k4 += kCarry) {
      if (kc - k4 >= kCarry) {
#pragma unroll
        for (int kk = 0; kk < kCarry; ++kk) one(k4 + kk);
      } else {
        for (int kk = k4; kk < kc; ++kk) one(kk);
      }
#pragma unroll
      for (int i = 0; i < RPT; ++i) { carry(acc[i][0]); carry(acc[i][1]); }
    }
    __syncthreads();  // every thread is done with this buffer before it is refilled
    cur ^= 1;
  }
  const int n = n0 + 2 * cp, e0 = cex[2 * cp], e1 = cex[2 * cp + 1];
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int row = row0 + rw + i;
    if (row < g.rows && n < N) {
      const int ea = aex[row];
      double* yp = (Y ? Y + (size_t)row * ldy : output_row(g, z, row)) + n;
      const double y0 = value_of(wide_of(acc[i][0]), ea, e0, g.alpha);
      if (n + 1 < N) {
        const double y1 = value_of(wide_of(acc[i][1]), ea, e1, g.alpha);
        if ((reinterpret_cast<uintptr_t>(yp) & 15) == 0) {
          *reinterpret_cast<double2*>(yp) = make_double2(y0, y1);
        } else {  // odd leading dimension or offset
          yp[0] = y0;
          yp[1] = y1;
        }
        if constexpr (RPT <= kFollowRows)
          if (g.follow.kind && z < nz) follow_row(g.follow, b0, e, row, n, y0, y1);
      } else {
        yp[0] = y0;
      }
    }
  }
  if constexpr (RPT <= kFollowRows)
    if (g.follow.kind) follow_modes(g.follow);
}

// Narrow form (N <= 8 columns per batch entry): a block takes RB rows and all
// columns of an entry, thread (row, part) one of KS shares of k; the operator
// is read once, straight to registers, the next 7 k (and the first ones, before
// the X panel is converted) in flight while these are multiplied; the shares'
// sums meet in shared memory, where the threads of a row take its column pairs.
// Bound by latency for one small run, then by issue.  With 32 rows and eight
// shares in every block two thirds of the instructions were for converting X
// and adding shares: 97 x 97 x 6, 1026 entries 114 -> 53 us, 291 x 97 x 6 256 ->
// 117, 291 x 97 x 2, 341 entries 40 -> 30, 195 x 65 x 8, 170 entries 32 -> 28.  (With
// 8 k in flight, carried every 4: 57, 124, 31 and 30.)
template <int NC>
__global__ void __launch_bounds__(256) fx_narrow_kernel(const __grid_constant__ GemmArgs g, int RB, int KS) {
  extern __shared__ __align__(16) double fsm[];
  Wide* parts = reinterpret_cast<Wide*>(fsm);                       // [KS][NC][RB]
  double* xd = reinterpret_cast<double*>(parts + KS * NC * RB);     // [K][NC]
  __shared__ int cex[NC];
  __shared__ int part[256], ws[257];
  constexpr int U = kCarry;
  const int z = blockIdx.y, tid = threadIdx.x, nthr = blockDim.x;
  const int kp = tid / RB, rl = tid - kp * RB, row = blockIdx.x * RB + rl;
  const int kq = (g.K + KS - 1) / KS, kb = min(kp * kq, g.K), ke = min(kb + kq, g.K);
  int N = g.N, e = z, b0 = g.follow.b0;
  const int nz = g.nsub ? g.nsub * g.batch : g.batch;
  long lda = g.lda, ldx = g.ldx;
  const int2* A = g.fx + (size_t)z * g.sA;
  const int* aex = g.fx_ex + (size_t)z * g.lda;
  const int* w = g.fx_w + (size_t)z * g.K;
  const double* X = g.X + (size_t)z * g.sX;
  double* Y = nullptr;
  if (g.nsub || z >= nz) {
    const int j = z < nz ? z / g.batch : g.nsub + z - nz;
    e = z < nz ? z - j * g.batch : 0;
    const FxJob& q = g.job[j];
    N = q.N;
    lda = q.lda;
    ldx = q.ldx;
    A = q.fx + (size_t)e * g.sA;
    aex = q.fx_ex + (size_t)e * lda;
    w = q.fx_w + (size_t)e * g.K;
    X = q.X + (size_t)e * g.sX;
    Y = q.Y + (size_t)e * g.sY + (size_t)row * q.ldy;
    b0 = q.b0;
  }
  A += min(row, g.rows - 1);
  int2 av[U];
#pragma unroll
  for (int u = 0; u < U; ++u) av[u] = kb + u < ke ? __ldg(A + (size_t)(kb + u) * lda) : make_int2(0, 0);
  for (int i = tid; i < g.K * NC; i += nthr) {
    const int k = i / NC, c = i - k * NC;
    xd[i] = c < N ? X[(size_t)k * ldx + c] : 0.0;
  }
  for (int k = tid; k < g.K; k += nthr) ws[k] = __ldg(w + k);
  const int ea = row < g.rows ? __ldg(aex + row) : 0;
  __syncthreads();
  convert_panel(xd, g.K, NC, ws, cex, part);
  const int2* xs = reinterpret_cast<const int2*>(xd);
  Sum acc[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) acc[c] = Sum{0, 0, 0};
  for (int k0 = kb; k0 < ke; k0 += U) {
    int2 nv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) nv[u] = k0 + U + u < ke ? __ldg(A + (size_t)(k0 + U + u) * lda) : make_int2(0, 0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (k0 + u >= ke) break;
      const int4* xp = reinterpret_cast<const int4*>(xs + (k0 + u) * NC);
#pragma unroll
      for (int c = 0; c < NC; c += 2) {
        const int4 x = xp[c / 2];
        add_product(acc[c], av[u], make_int2(x.x, x.y));
        add_product(acc[c + 1], av[u], make_int2(x.z, x.w));
      }
    }
#pragma unroll
    for (int c = 0; c < NC; ++c) carry(acc[c]);
#pragma unroll
    for (int u = 0; u < U; ++u) av[u] = nv[u];
  }
#pragma unroll
  for (int c = 0; c < NC; ++c) parts[(kp * NC + c) * RB + rl] = wide_of(acc[c]);
  if (g.follow.kind) follow_modes(g.follow);
  __syncthreads();
  if (row >= g.rows) return;
  auto column = [&](int c) {
    Wide s{0, 0};
    for (int q = 0; q < KS; ++q) s = add(s, parts[(q * NC + c) * RB + rl]);
    return value_of(s, ea, cex[c], g.alpha);
  };
  double* y = Y ? Y : output_row(g, z, row);
  for (int c = 2 * kp; c < N; c += 2 * KS) {
    const double y0 = column(c);
    y[c] = y0;
    if (c + 1 >= N) break;
    const double y1 = column(c + 1);
    y[c + 1] = y1;
    if (g.follow.kind && z < nz) follow_row(g.follow, b0, e, row, c, y0, y1);
  }
}

// Complex columns x[c][0..n) through real n x n operators whose rows (or
// columns) i and n - 1 - i agree up to sign and a few bits (the Chebyshev
// transforms).  With h = ceil(n / 2) pairs p of X (points p, n - 1 - p summed and
// differenced, or coefficients 2 p, 2 p + 1) and h pairs of outputs j,
//   S0 = sum_p A0[p][j] X0[p], S1 = sum_p A1[p][j] X1[p]
// hold half the products of the dense operator.  What the mirrored half
// differs by (the rounding of its own cosines, 2^-40 of an element) is a
// third sum of one 32-bit product each, D = sum (24 bits of the difference)
// (30 bits of x), added at its scale: outputs are those of the dense operator.
//   FWD: X0, X1 = x_p +- x_{n-1-p};  out_{2j} = S0 + D0, out_{2j+1} = S1 + D1
//   else X0, X1 = x_{2p}, x_{2p+1};  out_j = S0 + S1, out_{n-1-j} = +-(S0 - S1) + D
// A block takes NCOL real columns (re and im side by side) of one operator, and
// all its output pairs or, with few columns, a share of them (grid z: not in
// place); loads, outputs (through shared memory) and the operator's chunks of 7 p are
// coalesced.  Bound: the integer multiply-adds (61 % of that pipe's cycles, 16
// to 20 warps an SM); 65 points, 10944 columns: fwd 56 us, d1 and d2 102 us
// (one FP64 dot product a thread: 684 us for the three; chunks of 8, carried every
// 4: 62 and 103).
constexpr int kFxPC = kCarry;  // p per staged operator chunk (g.pc: this, or all of them in one)
template <int RPT, int NCOL, bool FWD>
__global__ void __launch_bounds__(512) fx_columns_kernel(const __grid_constant__ FxColumns g) {
  constexpr int RG = 64 / NCOL, CP = NCOL / 2, ST = NCOL + 2;  // ST: columns' stores hit every bank
  extern __shared__ __align__(16) double fsm[];
  const int n = g.n, h = (n + 1) / 2, nthr = blockDim.x, nw = nthr >> 5, hb = nw * RG * RPT, PC = g.pc;
  double* xs = fsm;                                                  // [n + 1][ST]
  int4* as = reinterpret_cast<int4*>(fsm + (size_t)(n + 1) * ST);    // [1 or 2][PC][hb]
  const int nbuf = PC < h ? 2 : 1;
  int2* ds = reinterpret_cast<int2*>(as + nbuf * PC * hb);           // the same
  int* cex = reinterpret_cast<int*>(ds + nbuf * PC * hb);            // [NCOL]
  int* part = cex + NCOL;                                            // [nthr]
  int* ws = part + nthr;                                             // [n]
  const FxColumnsOp& op = g.op[blockIdx.y];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c0 = blockIdx.x * CP;
  const int rg = lane / CP, cp = lane - rg * CP, rw = (warp * RG + rg) * RPT;
  const int j0 = blockIdx.z * hb, hv = min(hb, h - j0);  // the block's output pairs
  if (!FWD)
    for (int k = threadIdx.x; k < n; k += nthr) copy4(ws + k, op.w + k);
  for (int c = warp; c < CP; c += nw) {
    const bool ok = c0 + c < g.ncol;
    const double2* x = g.in + (size_t)(ok ? c0 + c : 0) * n;
    for (int k = lane; k < n; k += 32) copy16(xs + k * ST + 2 * c, x + k, ok);
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  auto issue = [&](int p0, int buf) {
    const int pc = min(PC, h - p0);
    for (int i = threadIdx.x; i < pc * hv; i += nthr) {
      const int p = i / hv, j = i - p * hv, o = (buf * PC + p) * hb + j;
      const size_t at = (size_t)(p0 + p) * h + j0 + j;
      copy16(as + o, op.A + at, true);
      copy8(ds + o, op.D + at, true);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  issue(0, 0);
  // (few columns: ahead of the products; the wider shapes lack the registers)
  const int4 ex = NCOL == 8 ? __ldg(op.ex + min(j0 + rw, h - 1)) : make_int4(0, 0, 0, 0);
  asm volatile("cp.async.wait_group 1;\n" ::: "memory");
  __syncthreads();
  convert_panel<ST - NCOL>(xs, n, NCOL, FWD ? nullptr : ws, cex, part, FWD);
  if (FWD) {
    for (int i = threadIdx.x; i < n / 2 * NCOL; i += nthr) {
      const int p = i / NCOL, c = i - p * NCOL;
      int2* a = reinterpret_cast<int2*>(xs) + p * ST + c;
      int2* b = reinterpret_cast<int2*>(xs) + (n - 1 - p) * ST + c;
      const long long va = ((long long)a->x << kLow) + a->y, vb = ((long long)b->x << kLow) + b->y;
      *a = signed_split(va + vb);
      *b = signed_split(va - vb);
    }
    __syncthreads();
  }
  Sum s0[RPT][2], s1[RPT][2];
  long long d0[RPT][2], d1[RPT][2];
#pragma unroll
  for (int i = 0; i < RPT; ++i)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      s0[i][c] = s1[i][c] = Sum{0, 0, 0};
      d0[i][c] = d1[i][c] = 0;
    }
  int cur = 0;
  for (int p0 = 0; p0 < h; p0 += PC) {
    const int pc = min(PC, h - p0);
    if (p0 + PC < h) {
      issue(p0 + PC, cur ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const int4* Aw = as + cur * PC * hb + rw;
    const int2* Dw = ds + cur * PC * hb + rw;
    const int4* xp = reinterpret_cast<const int4*>(xs) + cp;
    auto one = [&](int pp) {
      const int p = p0 + pp;
      const int4 u = xp[(FWD ? p : 2 * p) * (ST / 2)], v = xp[(FWD ? n - 1 - p : 2 * p + 1) * (ST / 2)];
      const int2 u0 = make_int2(u.x, u.y), u1 = make_int2(u.z, u.w), v0 = make_int2(v.x, v.y), v1 = make_int2(v.z, v.w);
      const int m0 = FWD ? (u0.x - v0.x) >> 1 : 0, m1 = FWD ? (u1.x - v1.x) >> 1 : 0;  // x_{n-1-p}
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int4 a = Aw[pp * hb + i];
        const int2 d = Dw[pp * hb + i];
        const int2 a0 = make_int2(a.x, a.y), a1 = make_int2(a.z, a.w);
        add_product(s0[i][0], a0, u0);
        add_product(s0[i][1], a0, u1);
        add_product(s1[i][0], a1, v0);
        add_product(s1[i][1], a1, v1);
        if (FWD) {
          d0[i][0] = madw1(d.x, m0, d0[i][0]);
          d0[i][1] = madw1(d.x, m1, d0[i][1]);
          d1[i][0] = madw1(d.y, m0, d1[i][0]);
          d1[i][1] = madw1(d.y, m1, d1[i][1]);
        } else {
          d0[i][0] = madw1(d.y, v0.x, madw1(d.x, u0.x, d0[i][0]));
          d0[i][1] = madw1(d.y, v1.x, madw1(d.x, u1.x, d0[i][1]));
        }
      }
    };
    for (int p7 = 0; p7 < pc; p7 += kCarry) {
      const int pe = min(p7 + kCarry, pc);
#pragma unroll 2
      for (int pp = p7; pp < pe; ++pp) one(pp);
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        carry(s0[i][0]); carry(s0[i][1]);
        carry(s1[i][0]); carry(s1[i][1]);
      }
    }
    __syncthreads();  // the buffer is refilled, after the last chunk the panel
    cur ^= 1;
  }
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int j = j0 + rw + i;
    if (rw + i >= hv) break;
    const int4 e = NCOL == 8 && i == 0 ? ex : __ldg(op.ex + j);
    double y[2], z[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const Wide a = wide_of(s0[i][c]), b = wide_of(s1[i][c]);
      Wide f, m;
      if (FWD) {
        f = add(a, d0[i][c] >> e.z);
        m = add(b, d1[i][c] >> e.w);
      } else {
        f = add(a, b);
        m = add(op.sign > 0 ? sub(a, b) : sub(b, a), d0[i][c] >> e.z);
      }
      y[c] = value_of(f, e.x, cex[2 * cp + c], 1.0);
      z[c] = value_of(m, e.y, cex[2 * cp + c], 1.0);
    }
    const int r = FWD ? 2 * j : j, q = FWD ? 2 * j + 1 : n - 1 - j;
    if (q < n && q != r) *reinterpret_cast<double2*>(xs + q * ST + 2 * cp) = make_double2(z[0], z[1]);
    *reinterpret_cast<double2*>(xs + r * ST + 2 * cp) = make_double2(y[0], y[1]);
  }
  __syncthreads();
  for (int c = warp; c < CP && c0 + c < g.ncol; c += nw) {
    double2* y = op.out + (size_t)(c0 + c) * n;
    auto store = [&](int k) { y[k] = *reinterpret_cast<const double2*>(xs + k * ST + 2 * c); };
    if (gridDim.z == 1) {
      for (int k = lane; k < n; k += 32) store(k);
    } else if (FWD) {
      for (int k = 2 * j0 + lane; k < min(2 * (j0 + hv), n); k += 32) store(k);
    } else {
      for (int j = j0 + lane; j < j0 + hv; j += 32) {
        store(j);
        store(n - 1 - j);
      }
    }
  }
}

template <int RPT, int NCOL, bool FWD>
cudaError_t launch_fx_columns_shape(FxColumns g, int most, cudaStream_t s) {
  const int h = (g.n + 1) / 2, per = 64 / NCOL * RPT, nw = std::min(most, std::max(2, (h + per - 1) / per)), hb = nw * per;
  // the operator in one chunk where it is small: no barriers between chunks
  g.pc = (h <= 32 || NCOL == 8) && h * hb * 24 <= 64 * 1024 ? h : kFxPC;
  const size_t smem = (size_t)(g.n + 1) * (NCOL + 2) * 8 + (g.pc < h ? 2 : 1) * g.pc * hb * 24 + (NCOL + 32 * nw + g.n) * 4;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(fx_columns_kernel<RPT, NCOL, FWD>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
  }
  const dim3 grid((g.ncol + NCOL / 2 - 1) / (NCOL / 2), g.nop, (h + hb - 1) / hb);
  fx_columns_kernel<RPT, NCOL, FWD><<<grid, 32 * nw, smem, s>>>(g);
  return cudaGetLastError();
}
template <int RPT, int NCOL>
cudaError_t launch_fx_columns_dir(const FxColumns& g, cudaStream_t s, int most = 16) {
  return g.fwd ? launch_fx_columns_shape<RPT, NCOL, true>(g, most, s)
               : launch_fx_columns_shape<RPT, NCOL, false>(g, most, s);
}

// Batch entries of a launch: those of the product, or of each of its
// sub-products, and the extra ones.
int entries(const GemmArgs& g) { return g.batch * std::max(1, g.nsub) + g.nextra; }

long column_blocks(const GemmArgs& g, int ncol) {
  if (!g.njobs) return ((long)g.N + ncol - 1) / ncol;
  long n = 0;
  for (int j = 0; j < g.njobs; ++j) n += ((long)g.job[j].N + ncol - 1) / ncol;
  return n;
}

template <int RPT, int NCOL>
cudaError_t launch_fx_tile(const GemmArgs& g, int nw, int row_blocks, cudaStream_t s) {
  static std::atomic<unsigned long long> opted[64];
  const cudaError_t e = allow_shared((const void*)fx_tile_kernel<RPT, NCOL>, 227 * 1024, opted);
  if (e != cudaSuccess) return e;
  const int rows_blk = nw * (64 / NCOL) * RPT;
  const size_t smem = ((size_t)g.K * NCOL + 2 * kFxKC * rows_blk) * 8 + (size_t)(NCOL + 32 * nw + g.K) * 4;
  const dim3 grid((unsigned)column_blocks(g, NCOL), row_blocks, entries(g));
  fx_tile_kernel<RPT, NCOL><<<grid, 32 * nw, smem, s>>>(g);
  return cudaGetLastError();
}

// Launch shape from a cost model of the integer pipe: a block's work is
// rows_blk x NCOL per k and a share of 6 rows' worth for converting its X
// panel; blocks spread evenly over the SMs; an SM with fewer than 8 warps
// cannot fill the pipe.  The cheapest (columns, row blocks, warps, rows per
// thread) wins, ties going to deeper register tiles.
struct TileShape { int ncol, rb, nw, rpt; };
TileShape pick_shape(const GemmArgs& g, int nsm) {
  TileShape best{64, 1, 8, 1};
  double bcost = 1e300;
  for (int ncol = 16; ncol <= 64; ncol *= 2) {
    if (g.fma_ncol && ncol != g.fma_ncol) continue;
    const int rg = 64 / ncol;
    const long cb = column_blocks(g, ncol) * entries(g);
    for (int rb = 1; rb <= 16; ++rb)
      for (int nw = 4; nw <= 16; ++nw)
        for (int rpt = 1; rpt <= 7; ++rpt) {
          const int rows_blk = nw * rg * rpt;
          if ((long)rb * rows_blk < g.rows || (long)(rb - 1) * rows_blk >= g.rows || rows_blk > 256) continue;
          const long smem = ((long)g.K * ncol + 2 * kFxKC * rows_blk) * 8 + (ncol + 32 * nw + g.K) * 4;
          if (smem > 227 * 1024) continue;
          const long blocks = cb * rb;
          const long fit = std::max(1L, std::min({220L * 1024 / smem, 64L / nw, 65536L / (32L * nw * (40 + 12 * rpt))}));
          const long waves = (blocks + nsm - 1) / nsm;
          const double warps = (double)nw * (double)std::min(waves, fit);
          const double eff = std::min(1.0, warps / 8.0);
          const double cost = (double)waves * ncol * (rows_blk * (rpt == 1 ? 1.3 : rpt == 2 ? 1.1 : 1.0) + 6.0) / eff;
          if (cost < bcost * (1.0 - 1e-12) || (cost <= bcost * (1.0 + 1e-12) && rpt > best.rpt)) {
            bcost = cost;
            best = {ncol, rb, nw, rpt};
          }
        }
  }
  return best;
}

template <int NCOL>
cudaError_t launch_ncol(const GemmArgs& g, const TileShape& t, cudaStream_t s) {
  switch (t.rpt) {
    case 1: return launch_fx_tile<1, NCOL>(g, t.nw, t.rb, s);
    case 2: return launch_fx_tile<2, NCOL>(g, t.nw, t.rb, s);
    case 3: return launch_fx_tile<3, NCOL>(g, t.nw, t.rb, s);
    case 4: return launch_fx_tile<4, NCOL>(g, t.nw, t.rb, s);
    case 5: return launch_fx_tile<5, NCOL>(g, t.nw, t.rb, s);
    case 6: return launch_fx_tile<6, NCOL>(g, t.nw, t.rb, s);
    default: return launch_fx_tile<7, NCOL>(g, t.nw, t.rb, s);
  }
}

TileShape tile_shape(const GemmArgs& g) {
  const int nsm = sm_count();
  // shapes are memoised per problem size: the search runs on the host once
  struct Memo { int rows, K, N, total, batch, nsm, ncol; TileShape t; };
  thread_local std::unordered_map<unsigned long long, Memo> memo;
  unsigned long long key = 1469598103934665603ull;
  const int total = (int)column_blocks(g, 1);  // columns of all jobs
  const int batch = entries(g);
  for (int v : {g.rows, g.K, g.N, total, batch, nsm, g.fma_ncol}) key = (key ^ (unsigned)v) * 1099511628211ull;
  Memo& m = memo[key];
  if (m.rows != g.rows || m.K != g.K || m.N != g.N || m.total != total || m.batch != batch || m.nsm != nsm ||
      m.ncol != g.fma_ncol)
    m = Memo{g.rows, g.K, g.N, total, batch, nsm, g.fma_ncol, pick_shape(g, nsm)};
  return m.t;
}

}  // namespace

// Whether launch_fx_gemm can do what follows g: every narrow form, and tiles of
// up to kFollowRows rows a thread (a batch of 12 of 33 x 86: a step 63 -> 56 us,
// 59 with 3 rows at most; tiles of 7 would spill).
bool fx_follows(const GemmArgs& g) {
  return g.N <= 8 || tile_shape(g).rpt <= kFollowRows;
}

cudaError_t launch_fx_operator(const double* A, long lda, long sA, int rows, int K, int nb, int* wk, int2* out,
                               int* ex, cudaStream_t s) {
  const long n = (long)nb * rows, m = (long)nb * K;
  if (n <= 0) return cudaSuccess;
  fx_weight_kernel<<<(unsigned)((m + 3) / 4), 128, 0, s>>>(A, lda, sA, rows, K, nb, wk);
  fx_operator_kernel<<<(unsigned)((n + 31) / 32), dim3(32, 8), 0, s>>>(A, lda, sA, rows, K, nb, wk, out, ex);
  return cudaGetLastError();
}

cudaError_t launch_fx_gemm(const GemmArgs& g, cudaStream_t s) {
  if (g.rows <= 0 || g.N <= 0 || g.batch <= 0) return cudaSuccess;
  if (g.K > 257 || !g.fx) return cudaErrorInvalidValue;
  // mode 0 is shared out over the whole grid, of which blocks past a narrower
  // product's columns leave early
  if (g.follow.kind == kVelocity && (g.njobs || g.nsub || g.nextra)) return cudaErrorInvalidValue;
  if (g.N <= 8 && !g.njobs) {
    // k shares until there are 448 threads an SM (above that one, a warp at least), rows
    // in even blocks of at most 256 threads, of fewer while SMs are without two
    // (us at 1, 2, 4, 8 shares: 33 x 33 x 2, 43 entries 13.0, 11.9, 9.9, 8.5; 65 x 65 x 8,
    // 171 entries 26.3, 20.8, 16.0, 21.1; 291 x 97 x 2, 341 entries 30.4, 33.1, 38.5, 47.7)
    const int nz = entries(g), nsm = sm_count();
    const int KS = (int)std::min(8L, std::max((31L + g.rows) / g.rows, nsm * 448L / ((long)g.rows * nz)));
    int nb = (g.rows + 256 / KS - 1) / (256 / KS);
    while ((long)nb * nz < 2 * nsm && (g.rows + nb - 1) / nb > 16) ++nb;
    const int RB = (g.rows + nb - 1) / nb;
    const dim3 grid((g.rows + RB - 1) / RB, nz);
    auto run = [&](auto kernel, int nc) {
      const size_t smem = (size_t)nc * ((size_t)KS * RB * sizeof(Wide) + g.K * sizeof(double));
      if (smem > 45 * 1024) {  // (2.1 KB of static arrays beside it)
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
        if (e != cudaSuccess) return e;
      }
      kernel<<<grid, RB * KS, smem, s>>>(g, RB, KS);
      return cudaGetLastError();
    };
    if (g.N <= 2) return run(fx_narrow_kernel<2>, 2);
    if (g.N <= 4) return run(fx_narrow_kernel<4>, 4);
    return g.N <= 6 ? run(fx_narrow_kernel<6>, 6) : run(fx_narrow_kernel<8>, 8);
  }
  const TileShape t = tile_shape(g);
  if (g.follow.kind && t.rpt > kFollowRows) return cudaErrorInvalidValue;  // see fx_follows
  if (t.ncol == 16) return launch_ncol<16>(g, t, s);
  if (t.ncol == 32) return launch_ncol<32>(g, t, s);
  return launch_ncol<64>(g, t, s);
}

// Shape: NCOL real columns a block, RPT output pairs a thread (64 / NCOL x RPT
// pairs a warp).  Few columns: small blocks and one pair a thread, for more
// blocks and shorter chains (65 points, us of fwd / d1d2 at <1, 8>, <1, 16>, <3, 16>:
// 300 columns 10.4/10.4, 12.5/12.4, 16.5/16.5; 1000 columns 12.4/18.5, 12.5/18.5,
// 16.5/20.6; 10944 columns 64/111, 64/113, 57/102; 17 points, 700 columns, fwd 6.3,
// 6.3 and, at <1, 32>, 8.3), and while SMs are idle the pairs of a column on several
// of them (fwd of 257 points, 4 columns 53 -> 23, 129 points 20 -> 14.4).  Many: one
// pair a thread up to 32 pairs (17 points, 20000 columns <1, 16> 21/33, <1, 32>
// 19/31, <3, 16> 31/52), above that the shape that pads least (97 points, 10000
// columns <2, 16> 115/197, <3, 16> 133/236; 129 points, 2000 columns <3, 32> 41/78,
// <3, 16> 49/88; 193 points, 3000 columns <3, 32> 195/320, <3, 16> 161/258).
cudaError_t launch_fx_columns(const FxColumns& g, cudaStream_t s) {
  if (g.n < 3 || g.n > 257 || g.ncol < 1 || g.ncol > 65535) return cudaErrorInvalidValue;
  const int h = (g.n + 1) / 2;
  const long cols = (long)g.ncol * g.nop, nsm = sm_count();
  if (cols < 4 * nsm) {
    // pairs shared out over blocks of at least two warps while SMs are idle
    const long blocks = (g.ncol + 3) / 4 * (long)g.nop, share = std::max(1L, nsm / blocks), warps = (h + 7) / 8;
    if (g.apart && share > 1) return launch_fx_columns_dir<1, 8>(g, s, (int)std::min(16L, std::max(2L, (warps + share - 1) / share)));
    return h <= 128 ? launch_fx_columns_dir<1, 8>(g, s) : launch_fx_columns_dir<2, 8>(g, s);
  }
  if (h <= 64 && cols < 32 * nsm) return launch_fx_columns_dir<1, 16>(g, s);
  if (h <= 32) return launch_fx_columns_dir<1, 32>(g, s);
  if (h <= 64) {
    return (h + 11) / 12 * 120 <= 11 * h ? launch_fx_columns_dir<3, 16>(g, s) : launch_fx_columns_dir<2, 16>(g, s);
  }
  return h <= 96 ? launch_fx_columns_dir<3, 32>(g, s) : launch_fx_columns_dir<3, 16>(g, s);
}

}  // namespace falcon
