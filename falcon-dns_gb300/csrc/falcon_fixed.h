// Fixed-point arithmetic of the azimuthal transforms: complex values as two
// 64-bit integers at a power of two shared by a radial line's transform and
// renewed before every stage (block floating point), |V| < 2^61 in modulus,
// multiplied by Q62 constants (round(c 2^62)) with 32-bit multiply-adds.  GB300
// issues an FP64 instruction every 64 cycles per sub-partition and a 32-bit
// integer one every 2, so a 64-bit integer add (2 instructions) and a product
// with a constant (7) cost a fraction of their FP64 forms, and 61 bits against one scale leave the transform's rounding below that of
// FP64 butterflies.  Host and device: the CPU tests run these butterflies.
#pragma once
#include <stdint.h>

#include <vector_types.h>

#include "falcon_combine.h"

namespace falcon {

FALCON_HD longlong2 fx_make(long long x, long long y) {
  longlong2 r;
  r.x = x;
  r.y = y;
  return r;
}
FALCON_HD longlong2 fx_add(longlong2 a, longlong2 b) { return fx_make(a.x + b.x, a.y + b.y); }
FALCON_HD longlong2 fx_sub(longlong2 a, longlong2 b) { return fx_make(a.x - b.x, a.y - b.y); }

// a * b + c, 32 x 32 + 64 bits, signed.
FALCON_HD long long fx_madw(int a, int b, long long c) {
#ifdef __CUDA_ARCH__
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (long long)a * b + c;
#endif
}

// A value prepared as a multiplicand: a = h 2^32 + l with l signed, |a| <
// 2^61.
struct FxMul { int h2, h4, l; };
FALCON_HD FxMul fx_prep(long long a) {
  FxMul m;
  m.l = (int)a;
  const unsigned h = (unsigned)(a >> 32) + ((unsigned)a >> 31);
  m.h2 = (int)(h << 1);
  m.h4 = (int)(h << 2);
  return m;
}
// A Q62 constant, c = hi 2^32 + 2 lo1 with lo1 signed (c even: Q61).
struct FxC { int hi, lo1; };
FALCON_HD constexpr FxC fx_const(long long c) {
  const long long lo = (long long)(((unsigned long long)c + 0x80000000ull) & 0xffffffffull) - 0x80000000ll;
  return FxC{(int)((c - lo) >> 32), (int)(lo / 2)};
}
constexpr long long kFxHalf = 1LL << 29;  // half a unit of the products' middle sum

// c a for |c| <= 1: a c 2^-62 = 4 h c.hi + (h c.lo + l c.hi) 2^-30 + l c.lo
// 2^-62.  The last term (below 1 unit, of either sign) is left out and the
// middle sum rounded: exact for a = 0, unbiased, half a unit rms.
FALCON_HD long long fx_mul(FxMul a, FxC c) {
  const long long w = fx_madw(a.l, c.hi, fx_madw(a.h2, c.lo1, kFxHalf));
  return fx_madw(a.h4, c.hi, w >> 30);
}
// c a + d b, c a + d b + f e for |a| + |b| + |e| < 2^61 (one middle sum: each
// l term is below 2^61, the h terms sum below 2^61).
FALCON_HD long long fx_mul2(FxMul a, FxC c, FxMul b, FxC d) {
  long long w = fx_madw(a.l, c.hi, fx_madw(a.h2, c.lo1, kFxHalf));
  w = fx_madw(b.l, d.hi, fx_madw(b.h2, d.lo1, w));
  return fx_madw(b.h4, d.hi, fx_madw(a.h4, c.hi, w >> 30));
}
FALCON_HD long long fx_mul3(FxMul a, FxC c, FxMul b, FxC d, FxMul e, FxC f) {
  long long w = fx_madw(a.l, c.hi, fx_madw(a.h2, c.lo1, kFxHalf));
  w = fx_madw(b.l, d.hi, fx_madw(b.h2, d.lo1, w));
  w = fx_madw(e.l, f.hi, fx_madw(e.h2, f.lo1, w));
  return fx_madw(e.h4, f.hi, fx_madw(b.h4, d.hi, fx_madw(a.h4, c.hi, w >> 30)));
}
// A twiddle exp(-i t) = c + i s as multipliers: (c.hi, c.lo1, s.hi, s.lo1).
FALCON_HD int4 fx_twiddle(long long c, long long s) {
  const FxC p = fx_const(c), q = fx_const(s);
  int4 w;
  w.x = p.hi;
  w.y = p.lo1;
  w.z = q.hi;
  w.w = q.lo1;
  return w;
}
// v w = (x c - y s, x s + y c)
FALCON_HD longlong2 fx_cmul(longlong2 v, int4 w) {
  const FxC c{w.x, w.y}, s{w.z, w.w}, ns{-w.z, -w.w};
  const FxMul x = fx_prep(v.x), y = fx_prep(v.y);
  return fx_make(fx_mul2(x, c, y, ns), fx_mul2(x, s, y, c));
}

// 2^floor(log2 P) / P as a multiplier.
inline FxC fx_over(int P) {
  int n = 0;
  while ((2 << n) <= P) ++n;
  return fx_const((long long)((((__int128)1 << (62 + n)) / P) & ~(__int128)1));
}

// The product of two grid values below 2^62 in magnitude, times 2^-64
// (rounded to nearest but for the low x low term, below a quarter unit).
FALCON_HD long long fx_mulhi(long long a, long long b) {
  const int al = (int)a, bl = (int)b;
  const int ah = (int)((unsigned)(a >> 32) + ((unsigned)a >> 31)), bh = (int)((unsigned)(b >> 32) + ((unsigned)b >> 31));
  return fx_madw(ah, bh, fx_madw(al, bh, fx_madw(ah, bl, 1LL << 31)) >> 32);
}

// a 2^(59 - e) truncated toward zero as a magnitude, for |a| < 2^e with
// e = eb_max - 1022, eb_max >= 1 the largest biased exponent of the field on
// the line (subnormal numbers included): below 2^59.
FALCON_HD unsigned long long fx_mag_of(unsigned long long bits, int eb_max) {
  const int eb = (int)((bits >> 52) & 0x7ff);
  const unsigned long long m = ((bits & 0xfffffffffffffULL) | (eb ? 1ULL << 52 : 0ULL)) << 6;
  const int sh = eb_max - (eb ? eb : 1);
  return sh > 63 ? 0ULL : m >> sh;
}

// cos(2 pi i/p) and sin(2 pi i/p) rounded to Q61, as Q62.
template <int p> struct FxDft;

template <> struct FxDft<3> {
  static constexpr long long c[3] = {
      4611686018427387904LL, -2305843009213693952LL, -2305843009213693952LL};
  static constexpr long long s[3] = {
      0LL, 3993837246235628776LL, -3993837246235628774LL};
};
template <> struct FxDft<5> {
  static constexpr long long c[5] = {
      4611686018427387904LL, 1425089352415399812LL, -3730932361629093762LL, -3730932361629093762LL,
      1425089352415399812LL};
  static constexpr long long s[5] = {
      0LL, 4385974038932618942LL, 2710681029835013084LL, -2710681029835013082LL,
      -4385974038932618940LL};
};
template <> struct FxDft<7> {
  static constexpr long long c[7] = {
      4611686018427387904LL, 2875339201863983834LL, -1026196679933739316LL, -4154985531143938468LL,
      -4154985531143938468LL, -1026196679933739316LL, 2875339201863983834LL};
  static constexpr long long s[7] = {
      0LL, 3605561316464170520LL, 4496061421583520200LL, 2000935573311439104LL,
      -2000935573311439104LL, -4496061421583520198LL, -3605561316464170518LL};
};
template <> struct FxDft<11> {
  static constexpr long long c[11] = {
      4611686018427387904LL, 3879597155310203736LL, 1915763607305631188LL, -656311349879663986LL,
      -3020012090752568662LL, -4424880331197296226LL, -4424880331197296226LL, -3020012090752568662LL,
      -656311349879663986LL, 1915763607305631188LL, 3879597155310203736LL};
  static constexpr long long s[11] = {
      0LL, 2493265698851133052LL, 4194937154890639038LL, 4564745704261934814LL,
      3485279745481982534LL, 1299262093321420668LL, -1299262093321420666LL, -3485279745481982532LL,
      -4564745704261934814LL, -4194937154890639038LL, -2493265698851133050LL};
};
template <> struct FxDft<13> {
  static constexpr long long c[13] = {
      4611686018427387904LL, 4083445173437190590LL, 2619736250061566422LL, 555877323041125914LL,
      -1635326399640084756LL, -3451896551983290448LL, -4477678804130201670LL, -4477678804130201670LL,
      -3451896551983290448LL, -1635326399640084756LL, 555877323041125914LL, 2619736250061566422LL,
      4083445173437190590LL};
  static constexpr long long s[13] = {
      0LL, 2143157354953472948LL, 3795343187733095620LL, 4578061635046789726LL,
      4312001333394836946LL, 3058113491511478316LL, 1103648702985592706LL, -1103648702985592706LL,
      -3058113491511478314LL, -4312001333394836946LL, -4578061635046789724LL, -3795343187733095618LL,
      -2143157354953472948LL};
};
template <> struct FxDft<17> {
  static constexpr long long c[17] = {
      4611686018427387904LL, 4300269142915883484LL, 3408077091039676538LL, 2055605343211474242LL,
      425512703280142176LL, -1262047785076457606LL, -2779161726810289588LL, -3920934477471642334LL,
      -4533163300302480862LL, -4533163300302480862LL, -3920934477471642334LL, -2779161726810289588LL,
      -1262047785076457606LL, 425512703280142176LL, 2055605343211474242LL, 3408077091039676538LL,
      4300269142915883484LL};
  static constexpr long long s[17] = {
      0LL, 1665933141228706944LL, 3106872780480267796LL, 4128212034951583148LL,
      4592013378890122490LL, 4435637870785019510LL, 3680204889512471596LL, 2427739845191991132LL,
      847395082207451608LL, -847395082207451608LL, -2427739845191991130LL, -3680204889512471594LL,
      -4435637870785019510LL, -4592013378890122490LL, -4128212034951583146LL, -3106872780480267796LL,
      -1665933141228706944LL};
};
template <> struct FxDft<19> {
  static constexpr long long c[19] = {
      4611686018427387904LL, 4361812149538374340LL, 3639268253758015090LL, 2522353173617808178LL,
      1132101988774059760LL, -380830012925640000LL, -1852493173538351514LL, -3123409954404957594LL,
      -4055856802012852724LL, -4548788632020149484LL, -4548788632020149484LL, -4055856802012852724LL,
      -3123409954404957594LL, -1852493173538351514LL, -380830012925640000LL, 1132101988774059760LL,
      2522353173617808178LL, 3639268253758015090LL, 4361812149538374340LL};
  static constexpr long long s[19] = {
      0LL, 1497412002322033046LL, 2832556179451299332LL, 3860748942899398788LL,
      4470569652692201668LL, 4595934772580406286LL, 4223259046583865548LL, 3392927672274001582LL,
      2194919937976036780LL, 759058570706444932LL, -759058570706444930LL, -2194919937976036778LL,
      -3392927672274001582LL, -4223259046583865546LL, -4595934772580406284LL, -4470569652692201666LL,
      -3860748942899398788LL, -2832556179451299330LL, -1497412002322033044LL};
};
template <> struct FxDft<23> {
  static constexpr long long c[23] = {
      4611686018427387904LL, 4440672190963873514LL, 3940314021820095408LL, 3147720787415133508LL,
      2121675502072022936LL, 938275250759811386LL, -314712583577595456LL, -1544359625305322958LL,
      -2659468578599335178LL, -3577336913677835818LL, -4229890535096285048LL, -4568732525988256240LL,
      -4568732525988256240LL, -4229890535096285048LL, -3577336913677835818LL, -2659468578599335178LL,
      -1544359625305322958LL, -314712583577595456LL, 938275250759811386LL, 2121675502072022936LL,
      3147720787415133508LL, 3940314021820095408LL, 4440672190963873514LL};
  static constexpr long long s[23] = {
      0LL, 1244217997361702392LL, 2396158037777683532LL, 3370385998225322834LL,
      4094647847674581572LL, 4515228398029303128LL, 4600935113897670364LL, 4345411520245862336LL,
      3767608633072374428LL, 2910379449246539436LL, 1837300735770145308LL, 627957831813268718LL,
      -627957831813268718LL, -1837300735770145308LL, -2910379449246539436LL, -3767608633072374428LL,
      -4345411520245862334LL, -4600935113897670364LL, -4515228398029303126LL, -4094647847674581572LL,
      -3370385998225322834LL, -2396158037777683532LL, -1244217997361702390LL};
};
template <> struct FxDft<29> {
  static constexpr long long c[29] = {
      4611686018427387904LL, 4503867362076992632LL, 4185452873564921562LL, 3671331260481713114LL,
      2985542278050005772LL, 2160152656888596422LL, 1233756698328316722LL, 249671647776288480LL,
      -746087771535652956LL, -1706960955867587646LL, -2588018543053995438LL, -3348063259543216200LL,
      -3951556259121244536LL, -4370278879862106056LL, -4584652117396725814LL, -4584652117396725814LL,
      -4370278879862106056LL, -3951556259121244536LL, -3348063259543216200LL, -2588018543053995438LL,
      -1706960955867587646LL, -746087771535652956LL, 249671647776288480LL, 1233756698328316722LL,
      2160152656888596422LL, 2985542278050005772LL, 3671331260481713114LL, 4185452873564921562LL,
      4503867362076992632LL};
  static constexpr long long s[29] = {
      0LL, 991376173496360426LL, 1936396698955509658LL, 2790873466921854116LL,
      3514852093408005126LL, 4074480142483920830LL, 4443590028556714734LL, 4604922583589796564LL,
      4550934076618075698LL, 4284148950223634028LL, 3817041780406304214LL, 3171453979274412942LL,
      2377572514889581590LL, 1472518402190570094LL, 498610965591785386LL, -498610965591785386LL,
      -1472518402190570092LL, -2377572514889581590LL, -3171453979274412942LL, -3817041780406304214LL,
      -4284148950223634026LL, -4550934076618075698LL, -4604922583589796562LL, -4443590028556714732LL,
      -4074480142483920830LL, -3514852093408005126LL, -2790873466921854116LL, -1936396698955509656LL,
      -991376173496360426LL};
};
template <> struct FxDft<31> {
  static constexpr long long c[31] = {
      4611686018427387904LL, 4517284534705129514LL, 4237944891373646972LL, 3785103286251945642LL,
      3177299107860337356LL, 2439415930676133194LL, 1601662778670846500LL, 698337364319389532LL,
      -233578063778459554LL, -1155930778500961330LL, -2030959551335534200LL, -2822840601510815450LL,
      -3499154225790556354LL, -4032212064933267590LL, -4400190668372809880LL, -4588024948848718296LL,
      -4588024948848718296LL, -4400190668372809880LL, -4032212064933267590LL, -3499154225790556354LL,
      -2822840601510815450LL, -2030959551335534200LL, -1155930778500961330LL, -233578063778459554LL,
      698337364319389532LL, 1601662778670846500LL, 2439415930676133194LL, 3177299107860337356LL,
      3785103286251945642LL, 4237944891373646972LL, 4517284534705129514LL};
  static constexpr long long s[31] = {
      0LL, 928325570622998360LL, 1818645383311068024LL, 2634509640324623224LL,
      3342516763121549148LL, 3913680856907234958LL, 4324618396573163188LL, 4558505550962299990LL,
      4605766952493380320LL, 4464467713834742858LL, 4140392642419027822LL, 3646809409747198674LL,
      3003925371358407452LL, 2238060275319958444LL, 1380568728648993642LL, 466556536017201064LL,
      -466556536017201062LL, -1380568728648993640LL, -2238060275319958442LL, -3003925371358407452LL,
      -3646809409747198672LL, -4140392642419027822LL, -4464467713834742858LL, -4605766952493380320LL,
      -4558505550962299988LL, -4324618396573163188LL, -3913680856907234956LL, -3342516763121549146LL,
      -2634509640324623222LL, -1818645383311068024LL, -928325570622998360LL};
};
constexpr long long kFxSqrtHalf = 3260954456333195554LL;  // sqrt(1/2)
constexpr long long kFxSqrt5Q = 2578010857022246788LL;  // sqrt(5)/4

// Forward DFT of length p in registers, v_j <- sum_q v_q exp(-2 pi i j q/p),
// for sum_q |v_q| < 2^61.  Odd lengths in the symmetric form
//   y_0 = v_0 + sum a_q,  y_j = A_j - i B_j,  y_{p-j} = A_j + i B_j,
//   a_q = v_q + v_{p-q},  b_q = v_q - v_{p-q},
//   A_j = v_0 + sum_q a_q cos(2 pi jq/p),  B_j = sum_q b_q sin(2 pi jq/p):
// every add exact, each product within 2 units.
FALCON_HD void fx_pair(longlong2 A, longlong2 B, longlong2& yj, longlong2& yk) {
  yj = fx_make(A.x + B.y, A.y - B.x);
  yk = fx_make(A.x - B.y, A.y + B.x);
}
FALCON_HD void fx_dft3(longlong2& v0, longlong2& v1, longlong2& v2) {
  constexpr FxC s = fx_const(FxDft<3>::s[1]);
  const longlong2 a = fx_add(v1, v2), b = fx_sub(v1, v2);
  const longlong2 A = fx_make(v0.x - (a.x >> 1), v0.y - (a.y >> 1));  // cos(2 pi/3) = -1/2
  const longlong2 B = fx_make(fx_mul(fx_prep(b.x), s), fx_mul(fx_prep(b.y), s));
  v0 = fx_add(v0, a);
  fx_pair(A, B, v1, v2);
}
template <int p>
FALCON_HD void fx_dft(longlong2 (&v)[p]) {
  static_assert(p >= 2 && p <= 8, "register butterflies");
  if constexpr (p == 2) {
    const longlong2 a = v[0], b = v[1];
    v[0] = fx_add(a, b);
    v[1] = fx_sub(a, b);
  } else if constexpr (p == 3) {
    fx_dft3(v[0], v[1], v[2]);
  } else if constexpr (p == 4) {
    const longlong2 t0 = fx_add(v[0], v[2]), t1 = fx_sub(v[0], v[2]);
    const longlong2 t2 = fx_add(v[1], v[3]), t3 = fx_sub(v[1], v[3]);
    v[0] = fx_add(t0, t2);
    v[2] = fx_sub(t0, t2);
    fx_pair(t1, t3, v[1], v[3]);
  } else if constexpr (p == 5) {
    // cos(2 pi/5), cos(4 pi/5) = (-1 +- sqrt 5)/4
    constexpr FxC q = fx_const(kFxSqrt5Q), s1 = fx_const(FxDft<5>::s[1]), s2 = fx_const(FxDft<5>::s[2]),
                  n1 = fx_const(-FxDft<5>::s[1]);
    const longlong2 a1 = fx_add(v[1], v[4]), b1 = fx_sub(v[1], v[4]);
    const longlong2 a2 = fx_add(v[2], v[3]), b2 = fx_sub(v[2], v[3]);
    const longlong2 t = fx_add(a1, a2), u = fx_sub(a1, a2);
    const longlong2 w = fx_make(v[0].x - (t.x >> 2), v[0].y - (t.y >> 2));
    const longlong2 z = fx_make(fx_mul(fx_prep(u.x), q), fx_mul(fx_prep(u.y), q));
    const FxMul b1x = fx_prep(b1.x), b1y = fx_prep(b1.y), b2x = fx_prep(b2.x), b2y = fx_prep(b2.y);
    const longlong2 B1 = fx_make(fx_mul2(b1x, s1, b2x, s2), fx_mul2(b1y, s1, b2y, s2));
    const longlong2 B2 = fx_make(fx_mul2(b1x, s2, b2x, n1), fx_mul2(b1y, s2, b2y, n1));
    v[0] = fx_add(v[0], t);
    fx_pair(fx_add(w, z), B1, v[1], v[4]);
    fx_pair(fx_sub(w, z), B2, v[2], v[3]);
  } else if constexpr (p == 6) {
    // Good-Thomas 2 x 3: inputs n = (3 n1 + 2 n2) mod 6, two 3-point DFTs
    // over n2, then y_k = W_0[k mod 3] +- W_1[k mod 3], sign (-1)^k
    longlong2 w0 = v[0], w1 = v[2], w2 = v[4], z0 = v[3], z1 = v[5], z2 = v[1];
    fx_dft3(w0, w1, w2);
    fx_dft3(z0, z1, z2);
    v[0] = fx_add(w0, z0);
    v[3] = fx_sub(w0, z0);
    v[4] = fx_add(w1, z1);
    v[1] = fx_sub(w1, z1);
    v[2] = fx_add(w2, z2);
    v[5] = fx_sub(w2, z2);
  } else if constexpr (p == 8) {
    // one decimation-in-frequency split: even outputs from the sums, odd
    // ones from the differences turned by exp(-2 pi i j/8)
    constexpr int h = p / 2;
    constexpr FxC r = fx_const(kFxSqrtHalf);
    longlong2 t[h], u[h];
#pragma unroll
    for (int j = 0; j < h; ++j) {
      t[j] = fx_add(v[j], v[j + h]);
      u[j] = fx_sub(v[j], v[j + h]);
    }
    auto turn1 = [&](longlong2 z) {  // exp(-i pi/4)
      return fx_make(fx_mul(fx_prep(z.x + z.y), r), fx_mul(fx_prep(z.y - z.x), r));
    };
    auto turn2 = [&](longlong2 z) { return fx_make(z.y, -z.x); };  // -i
    u[1] = turn1(u[1]);
    u[2] = turn2(u[2]);
    u[3] = turn2(turn1(u[3]));
    fx_dft<h>(t);
    fx_dft<h>(u);
#pragma unroll
    for (int j = 0; j < h; ++j) {
      v[2 * j] = t[j];
      v[2 * j + 1] = u[j];
    }
  } else {
    constexpr int h = 3;
    longlong2 a[h], b[h];
#pragma unroll
    for (int q = 0; q < h; ++q) {
      a[q] = fx_add(v[q + 1], v[p - 1 - q]);
      b[q] = fx_sub(v[q + 1], v[p - 1 - q]);
    }
    const longlong2 v0 = v[0];
    FxMul ax[h], ay[h], bx[h], by[h];
#pragma unroll
    for (int q = 0; q < h; ++q) {
      ax[q] = fx_prep(a[q].x);
      ay[q] = fx_prep(a[q].y);
      bx[q] = fx_prep(b[q].x);
      by[q] = fx_prep(b[q].y);
    }
    v[0] = fx_add(v0, fx_add(a[0], fx_add(a[1], a[2])));
    constexpr FxC c1 = fx_const(FxDft<7>::c[1]), c2 = fx_const(FxDft<7>::c[2]), c3 = fx_const(FxDft<7>::c[3]);
    constexpr FxC s1 = fx_const(FxDft<7>::s[1]), s2 = fx_const(FxDft<7>::s[2]), s3 = fx_const(FxDft<7>::s[3]),
                  n1 = fx_const(-FxDft<7>::s[1]), n3 = fx_const(-FxDft<7>::s[3]);
    auto out = [&](int j, FxC p0, FxC p1, FxC p2, FxC q0, FxC q1, FxC q2) {
      const longlong2 A = fx_make(v0.x + fx_mul3(ax[0], p0, ax[1], p1, ax[2], p2),
                                  v0.y + fx_mul3(ay[0], p0, ay[1], p1, ay[2], p2));
      const longlong2 B = fx_make(fx_mul3(bx[0], q0, bx[1], q1, bx[2], q2), fx_mul3(by[0], q0, by[1], q1, by[2], q2));
      fx_pair(A, B, v[j], v[p - j]);
    };
    out(1, c1, c2, c3, s1, s2, s3);
    out(2, c2, c3, c1, s2, n3, n1);  // cos 8 pi/7 = cos 6 pi/7, sin 8 pi/7 = -sin 6 pi/7, ...
    out(3, c3, c1, c2, s3, n1, s2);
  }
}

// The magnitudes of a set of values: the bits of every high word's
// magnitude (one's complement), by component; |V| <= 2^fx_bits.
struct FxMax { unsigned x, y; };
FALCON_HD void fx_cover(FxMax& o, longlong2 v) {
  const int x = (int)(v.x >> 32), y = (int)(v.y >> 32);
  o.x |= (unsigned)(x ^ (x >> 31));
  o.y |= (unsigned)(y ^ (y >> 31));
}
FALCON_HD int fx_bits(unsigned o) { return 64 - (o ? clz64(o) - 32 : 32); }

// ceil(log2(p sqrt 2)): how far the moduli of p summed values can exceed
// their largest component.
FALCON_HD constexpr int fx_growth(int p) {
  return p <= 2 ? 2 : p <= 5 ? 3 : p <= 11 ? 4 : p <= 22 ? 5 : p <= 45 ? 6 : 7;
}

// Stage inputs scaled by 2^-d (d < 0: up).
FALCON_HD long long fx_scale(long long v, int d) { return d >= 0 ? v >> d : (long long)((unsigned long long)v << -d); }

// One in-place stage of radix p and span m of a line whose element i lies at
// buf[tab[i]] (tab null: at buf[i]): butterfly t -> g = t / m, k = t - g m,
// elements g m p + k + q m, sp apart; the stage's inputs scaled by 2^-d.  DIT
// twiddles exp(-2 pi i q k / (m p)) on the inputs, DIF on the outputs, from
// tw[(q - 1) m + k]; none for the prime-factor plans and m = 1.  The
// outputs' magnitudes are added to o.
template <int p, bool TWID>
FALCON_HD void fx_stage(longlong2* buf, const uint16_t* tab, int sp, int P, int m, const int4* tw, int lane, int nl,
                        bool dif, int d, FxMax& o) {
  const int nb = P / p, mp = m * p;
  const float inv_m = 1.0f / (float)m;
  for (int t = lane; t < nb; t += nl) {
    const int g = (int)(((float)t + 0.5f) * inv_m);
    const int k = t - g * m, base = g * mp + k;
    const bool tk = TWID && m > 1;
    longlong2* at = buf + (tab ? tab[base] : base);
    longlong2 v[p];
#pragma unroll
    for (int q = 0; q < p; ++q) v[q] = at[q * sp];
    if (d > 0) {
#pragma unroll
      for (int q = 0; q < p; ++q) v[q] = fx_make(v[q].x >> d, v[q].y >> d);
    } else if (d < 0) {
#pragma unroll
      for (int q = 0; q < p; ++q) v[q] = fx_make(fx_scale(v[q].x, d), fx_scale(v[q].y, d));
    }
    if (tk && !dif) {
#pragma unroll
      for (int q = 1; q < p; ++q) v[q] = fx_cmul(v[q], tw[(q - 1) * m + k]);
    }
    fx_dft<p>(v);
    if (tk && dif) {
#pragma unroll
      for (int q = 1; q < p; ++q) v[q] = fx_cmul(v[q], tw[(q - 1) * m + k]);
    }
#pragma unroll
    for (int q = 0; q < p; ++q) {
      at[q * sp] = v[q];
      fx_cover(o, v[q]);
    }
  }
}

// The same for any odd prime p <= 61 of an unpadded twiddled plan, with the
// p-th roots of unity root[i] = exp(-2 pi i j/p).
FALCON_HD void fx_stage_any(longlong2* buf, int P, int p, int m, const int4* tw, const int4* root, int lane,
                            int nl, bool dif, int d, FxMax& o) {
  const int nb = P / p, mp = m * p, h = (p - 1) / 2;
  for (int t = lane; t < nb; t += nl) {
    const int g = t / m, k = t - g * m;
    longlong2* at = buf + g * mp + k;
    const bool tk = m > 1;
    longlong2 a[30], b[30];
    const longlong2 v0 = fx_make(fx_scale(at[0].x, d), fx_scale(at[0].y, d));
    longlong2 y0 = v0;
    for (int q = 1; q <= h; ++q) {
      longlong2 x = at[q * m], y = at[(p - q) * m];
      x = fx_make(fx_scale(x.x, d), fx_scale(x.y, d));
      y = fx_make(fx_scale(y.x, d), fx_scale(y.y, d));
      if (tk && !dif) {
        x = fx_cmul(x, tw[(q - 1) * m + k]);
        y = fx_cmul(y, tw[(p - q - 1) * m + k]);
      }
      a[q - 1] = fx_add(x, y);
      b[q - 1] = fx_sub(x, y);
      y0 = fx_add(y0, a[q - 1]);
    }
    at[0] = y0;
    fx_cover(o, y0);
    for (int j = 1; j <= h; ++j) {
      __int128 ax = 0, ay = 0, bx = 0, by = 0;  // exact sums, in 2^-62
      int i = 0;
      for (int q = 0; q < h; ++q) {
        i += j;
        if (i >= p) i -= p;
        const int4 w = root[i];
        const long long c = (long long)w.x * (1LL << 32) + 2LL * w.y, s = (long long)w.z * (1LL << 32) + 2LL * w.w;
        ax += (__int128)a[q].x * c;
        ay += (__int128)a[q].y * c;
        bx -= (__int128)b[q].x * s;
        by -= (__int128)b[q].y * s;
      }
      const longlong2 A = fx_make(v0.x + (long long)(ax >> 62), v0.y + (long long)(ay >> 62));
      const longlong2 B = fx_make((long long)(bx >> 62), (long long)(by >> 62));
      longlong2 yj, yk;
      fx_pair(A, B, yj, yk);
      if (tk && dif) {
        yj = fx_cmul(yj, tw[(j - 1) * m + k]);
        yk = fx_cmul(yk, tw[(p - j - 1) * m + k]);
      }
      at[j * m] = yj;
      at[(p - j) * m] = yk;
      fx_cover(o, yj);
      fx_cover(o, yk);
    }
  }
}

}  // namespace falcon
