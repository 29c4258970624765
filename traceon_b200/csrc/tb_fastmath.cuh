// tb_fastmath.cuh -- branch-free FP64 reciprocal, reciprocal square root and
// logarithm for the ring-pair loops.
//
// The library functions behind 1.0/x, sqrt(x) and log(x) carry special-case
// branches (zero, infinity, NaN, subnormals) that split the hot loops into
// divergence regions and keep the compiler from interleaving consecutive
// pairs.  The ring-pair arguments are always positive normal numbers, so
// these versions drop the special cases:
//
//  * rcp_nr / rsqrt_nr: the PTX hardware approximations rcp.approx.ftz.f64 /
//    rsqrt.approx.ftz.f64 (about 2^-22 relative) refined by Newton-Raphson
//    iterations written out below (for 1/x: y <- y + y e, e = 1 - x y; for
//    1/sqrt(x): y <- y + y e (1/2 + 3/8 e), e = 1 - x y^2), which square
//    (resp. cube) the relative error per step.
//  * log_bf: Cody & Waite argument reduction t = 2^k m, m in [sqrt(1/2),
//    sqrt(2)), then log m = 2 atanh(s), s = (m - 1)/(m + 1), summed as the
//    odd series 2 (s + s^3/3 + s^5/5 + ...) through s^21 (|s| <= 0.1716, so
//    the next term is below 2^-55 of the sum), and k log 2 added in two parts
//    (log 2 split into a 32-bit head and its remainder).
// All three are accurate to about 1 ulp (checked against the library
// functions by tests/test_gpu_kernels.py through tb_probe_math).
//
// The ring-pair field sums use two shorter forms:
//
//  * rsqrt_h3: one third-order step from the hardware approximation.  The
//    step cubes the relative error (2^-22 -> about 2^-67), so its result is
//    already rounding-limited and a second step adds nothing.
//  * neglog_tab: table-driven logarithm (the method of P. T. P. Tang, ACM
//    TOMS 16, 1990): t = 2^k m with m in [0.707, 1.414), 1/c of the m's
//    interval from a 128-entry table, r = m (1/c) - 1 with |r| <= 2^-8, and
//    log(1 + r) by its Taylor sum through r^6 (the next term is below
//    2^-58).  The entries are the exact reciprocals' roundings and their
//    logarithms; the interval around 1 takes c = 1, so log 1 is exactly 0.
//    Absolute error below 2e-16 (1 + |log t| 1e-16): what the sums need,
//    since L = -log t always enters as L B(t) + A(t) with A of order 1.
#pragma once

#include <cstdint>

namespace tb {

__device__ __forceinline__ double rcp_approx(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

__device__ __forceinline__ double rsqrt_approx(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}

// 1/x for positive normal x.
__device__ __forceinline__ double rcp_nr(double x) {
  double y = rcp_approx(x);
  double e = fma(-x, y, 1.0);
  y = fma(y, e, y);
  e = fma(-x, y, 1.0);
  return fma(y, e, y);
}

// 1/sqrt(x) for positive normal x.
__device__ __forceinline__ double rsqrt_nr(double x) {
  double y = rsqrt_approx(x);
  double e = fma(-x * y, y, 1.0);
  y = fma(y * e, fma(0.375, e, 0.5), y);
  e = fma(-x * y, y, 1.0);
  return fma(y * e, 0.5, y);
}

// 1/sqrt(x) for positive normal x, one third-order step.
__device__ __forceinline__ double rsqrt_h3(double x) {
  const double y = rsqrt_approx(x);
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// a / b from y = 1 / b rounded to nearest: the product, its exact remainder by
// a fused multiply-add, and one correction (P. Markstein, IBM J. Res. Dev. 34,
// 1990: the rounded quotient).  For divisors that stay the same over a launch:
// three dependent operations instead of a division.
__device__ __forceinline__ double div_by(double a, double b, double y) {
  const double q = a * y;
  return fma(fma(-b, q, a), y, q);
}

// Coefficients 1/(2j+1), j = 1..10, of the atanh series.
__constant__ double C_ATANH[10] = {1.0 / 3,  1.0 / 5,  1.0 / 7,  1.0 / 9,  1.0 / 11,
                                   1.0 / 13, 1.0 / 15, 1.0 / 17, 1.0 / 19, 1.0 / 21};

// log(t) for positive normal t.
__device__ __forceinline__ double log_bf(double t) {
  const long long bits = __double_as_longlong(t);
  int k = int((bits >> 52) & 0x7ff) - 1023;
  double m = __longlong_as_double((bits & 0x000fffffffffffffLL) | 0x3ff0000000000000LL);  // [1, 2)
  const bool big = m > 1.4142135623730951;
  m = big ? 0.5 * m : m;
  k += big ? 1 : 0;
  const double f = m - 1.0;            // exact (Sterbenz)
  const double s = f * rcp_nr(2.0 + f);
  const double s2 = s * s;
  double p = C_ATANH[9];
#pragma unroll
  for (int j = 8; j >= 0; j--) p = fma(p, s2, C_ATANH[j]);
  // log m = 2 s + 2 s^3 P(s^2)
  const double logm = fma(2.0 * s * s2, p, 2.0 * s);
  const double kd = double(k);
  const double LN2_HI = 0.6931471803691238;     // log 2 with its significand cut to 32 bits
  const double LN2_LO = 1.9082149292705877e-10;  // log 2 - LN2_HI, rounded
  return fma(kd, LN2_HI, fma(kd, LN2_LO, logm));
}

// {1/c, log(1/c)} of the 128 intervals of the significand's high word
// [0x3fe6a09e + 2^13 i, 0x3fe6a09e + 2^13 (i + 1)).
__device__ const double2 LOG_TAB[128] = {
    {1.4103184519766565, 0.3438155313549622}, {1.4025914962433068, 0.33832159424995306},
    {1.3949487491602313, 0.33285767564519786}, {1.3873888416242057, 0.3274234492844264},
    {1.3799104340513786, 0.32201859420151163}, {1.3725122155859488, 0.3166427946067132},
    {1.3651929033341623, 0.31129573977596214}, {1.357951241622689, 0.30597712394309085},
    {1.3507860012804807, 0.3006866461949136}, {1.3436959789432408, 0.2954240103690672},
    {1.336679996379689, 0.29018892495452653}, {1.32973689983882, 0.28498110299471047},
    {1.322865559417401, 0.279800261993097}, {1.3160648684469802, 0.2746461238212719},
    {1.309333742899705, 0.26951841462933446}, {1.3026711208122812, 0.26441686475858805},
    {1.2960759617274322, 0.2593412086564471}, {1.289547246152238, 0.2542911847934929},
    {1.2830839750327632, 0.24926653558261266}, {1.2766851692444057, 0.24426700730015966},
    {1.2703498690974204, 0.23929235000907614}, {1.2640771338570906, 0.23434231748391626},
    {1.257866041278048, 0.2294166671377185}, {1.251715687152252, 0.22451515995066773},
    {1.2456251848701663, 0.21963756040049867}, {1.2395936649946862, 0.21478363639458817},
    {1.2336202748473821, 0.20995315920368723}, {1.227704178106651, 0.20514590339724612},
    {1.2218445544173733, 0.20036164678028645}, {1.216040599011698, 0.19560017033177668},
    {1.2102915223405815, 0.1908612581444669}, {1.2045965497157312, 0.1861446973661437},
    {1.19895492096161, 0.18145027814226292}, {1.1933658900771733, 0.17677779355992254},
    {1.1878287249070254, 0.17212703959313994}, {1.182342706821685, 0.1674978150493933},
    {1.176907130406674, 0.1628899215173975}, {1.171521303160141, 0.1583031633160757},
    {1.1661845451987487, 0.15373734744469594}, {1.1608961889715659, 0.14919228353414213},
    {1.1556555789817082, 0.1446677837992871}, {1.1504620715154827, 0.1401636629924366},
    {1.1453150343788059, 0.13567973835781957}, {1.1402138466406635, 0.13121582958709244},
    {1.1351578983833968, 0.12677175877583266}, {1.1301465904596026, 0.12234735038099498},
    {1.125179334255445, 0.11794243117930435}, {1.1202555514601795, 0.1135568302265606},
    {1.1153746738417059, 0.10919037881783387}, {1.110536143027959, 0.10484291044852244},
    {1.1057394102939673, 0.10051426077625472}, {1.100983936354406, 0.09620426758361304},
    {1.0962691911614801, 0.091912770741656}, {1.0915946537079777, 0.08763961217422067},
    {1.0869598118353414, 0.08338463582298414}, {1.082364162046609, 0.07914768761326572},
    {1.0778072093240783, 0.07492861542055027}, {1.0732884669515597, 0.0707272690377143},
    {1.0688074563410803, 0.06654350014293824}, {1.0643637068639125, 0.06237716226828727},
    {1.0599567556857985, 0.0582281107689434}, {1.0555861476062531, 0.054096202793073506},
    {1.0512514349018252, 0.04998129725231766}, {1.0469521771732044, 0.04588325479288138},
    {1.042687941196066, 0.04180193776721824}, {1.038458300775544, 0.037737210206288306},
    {1.034262836604234, 0.03368893779237754}, {1.0301011361236228, 0.029656987832465734},
    {1.0259727933888503, 0.025641229232128283}, {1.0218774089367106, 0.02164153246996069},
    {1.0178145896568025, 0.01765776957251247}, {1.0137839486657405, 0.013689814089718222},
    {1.0097851051843434, 0.00973754107081363}, {1.0058176844177185, 0.005800827040727015},
    {1.0, 0.0}, {0.9959594616414805, -0.004048723389025799},
    {0.9882698002491938, -0.011799541337757248}, {0.9806979706588204, -0.01949074586425325},
    {0.9732412850865876, -0.02712324697647434}, {0.9658971368775551, -0.03469793400300379},
    {0.9586629974675211, -0.04221567621490813}, {0.9515364134804379, -0.049677323424396465},
    {0.9445150039543351, -0.057083706561310885}, {0.9375964576891643, -0.0644356382284239},
    {0.9307785307103584, -0.07173391323647184}, {0.924059043842256, -0.07897930911980584},
    {0.9174358803858813, -0.08617258663349578}, {0.9109069838958801, -0.09331449023268218},
    {0.9044703560517059, -0.10040574853493305}, {0.8981240546184298, -0.10744707476632047},
    {0.8918661914928001, -0.11443916719190325}, {0.8856949308304235, -0.12138270953126369},
    {0.8796084872501665, -0.1282783713597164}, {0.8736051241120866, -0.1351268084957789},
    {0.8676831518654042, -0.14192866337546475}, {0.8618409264632152, -0.14868456541393268},
    {0.856076847840818, -0.1553951313550011}, {0.8503893584546987, -0.16206096560901295},
    {0.8447769418793696, -0.16868266057951545}, {0.8392381214594081, -0.17526079697919342},
    {0.8337714590141775, -0.18179594413547992}, {0.8283755535928432, -0.1882886602862456},
    {0.8230490402774224, -0.19473949286594974}, {0.8177905890317156, -0.20114897878262217},
    {0.8125989035940849, -0.20751764468602327}, {0.8074727204121394, -0.21384600722732058},
    {0.802410807617491, -0.22013457331059885}, {0.7974119640388327, -0.22638384033651202},
    {0.7924750182516782, -0.2325942964383686}, {0.787598827663183, -0.23876642071093182},
    {0.7827822776305475, -0.24490068343220134}, {0.778024280611571, -0.25099754627843446},
    {0.7733237753459977, -0.2570574625326522}, {0.7686797260663605, -0.2630808772868657},
    {0.76409112173709, -0.2690682276382479}, {0.7595569753207148, -0.2750199428794679},
    {0.7550763230700323, -0.280936444683395}, {0.7506482238451879, -0.28681814728237026},
    {0.7462717584546427, -0.29266545764223634}, {0.7419460290190607, -0.29847877563131014},
    {0.7376701583571936, -0.3042584941844707}, {0.7334432893928775, -0.31000499946253335},
    {0.7292645845823011, -0.3157186710070708}, {0.7251332253607423, -0.32139988189083574},
    {0.7210484116080036, -0.32704899886393485}, {0.7170093611318149, -0.3326663824958973},
    {0.7130153091685015, -0.33825238731377577}, {0.7090655079002498, -0.3438073619364099}};

// -log(t) for positive normal t.
__device__ __forceinline__ double neglog_tab(double t) {
  const int hi = __double2hiint(t);
  const int d = hi - 0x3fe6a09e;
  const int k = d >> 20;
  const double2 e = __ldg(&LOG_TAB[(d >> 13) & 127]);
  const double m = __hiloint2double(hi - (k << 20), __double2loint(t));
  const double r = fma(m, e.x, -1.0);
  double p = fma(r, -1.0 / 6.0, 0.2);
  p = fma(p, r, -0.25);
  p = fma(p, r, 1.0 / 3.0);
  p = fma(p, r, -0.5);
  const double l1 = fma(p, r * r, r);  // log(1 + r)
  // k as a double: 2^52 + 2^31 + k built from its bits, less 2^52 + 2^31
  const double kd = __hiloint2double(0x43300000, k ^ 0x80000000) - 4503601774854144.0;
  return fma(kd, -0.6931471805599453, e.y) - l1;
}

}  // namespace tb
