// Shared helpers of the FFNO3D kernels: activations, the level-fraction head, the deterministic depth-weighted GroupNorm
// statistics, launches.
//
// Activation layout: channels last, one row of C floats per voxel, voxel v = (d * H + h) * W + w of one cube.
// A "tile" is BM = 64 consecutive voxels processed by one CTA of NT = 256 threads (the FP32 chains' tile GEMM and its
// thread mapping: gemm_f32.cuh).
#pragma once
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include <cmath>

#include "../../include/ffnoml_gb300.h"

namespace ffno {

constexpr int BM = 64;
constexpr int NT = 256;
constexpr int GMAX = 8;  // DepthWeightedGroupNorm uses at most 8 groups (models/ffno_model.py:21-25)

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752440f)); }

// d gelu / dx = Phi(x) + x phi(x)
__device__ __forceinline__ float gelu_grad(float x) {
  const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752440f));
  const float pdf = 0.39894228040143267794f * expf(-0.5f * x * x);
  return cdf + x * pdf;
}

__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + expf(-x)); }

// Activations of the tensor-core (split-BF16) kernels: the normal CDF from the rational approximation of erfc in
// Abramowitz & Stegun, Handbook of Mathematical Functions, eq. 7.1.26 (|error of erf| <= 1.5e-7), whose exp(-x^2/2)
// factor is also the normal density in the GELU derivative: one exponential and one reciprocal (hardware
// approximations) per element instead of erff and expf. The absolute error of gelu and gelu' stays near 1e-6, well
// below the 2^-16 relative rounding of a split-BF16 operand; the FP32 kernels keep erff / expf.
struct Cdf {
  float cdf, pdf;   // Phi(x), phi(x)
};
__device__ __forceinline__ Cdf cdf_tc(float x) {
  const float u = fabsf(x) * 0.70710678118654752440f;
  const float t = __fdividef(1.f, fmaf(0.3275911f, u, 1.f));
  const float e = __expf(-0.5f * x * x);
  float p = fmaf(t, 1.061405429f, -1.453152027f);
  p = fmaf(t, p, 1.421413741f);
  p = fmaf(t, p, -0.284496736f);
  p = fmaf(t, p, 0.254829592f);
  const float h = 0.5f * (p * t) * e;   // (1 - erf(u)) / 2
  return Cdf{x < 0.f ? h : 1.f - h, 0.39894228040143267794f * e};
}
__device__ __forceinline__ float gelu_grad_tc(float x) {
  const Cdf c = cdf_tc(x);
  return fmaf(x, c.pdf, c.cdf);
}
// Two FP32 lanes in one 64-bit register (fma.rn.f32x2 and its relatives: two IEEE operations per issued instruction).
__device__ __forceinline__ uint64_t pk2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void upk2(uint64_t v, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// cdf_tc of two values at once, the same operations: the epilogues and conversions of the
// tensor-core kernels are bound by issue slots, and the packed polynomial takes half of them.
struct Cdf2 {
  uint64_t cdf, e;   // Phi(x) and exp(-x^2 / 2), two lanes each
};
__device__ __forceinline__ Cdf2 cdf_tc2(float x0, float x1) {
  const uint64_t x = pk2(x0, x1);
  const uint64_t u = mul2(pk2(fabsf(x0), fabsf(x1)), pk2(0.70710678118654752440f, 0.70710678118654752440f));
  float d0, d1, q0, q1;
  upk2(fma2(pk2(0.3275911f, 0.3275911f), u, pk2(1.f, 1.f)), d0, d1);
  upk2(mul2(mul2(pk2(-0.5f, -0.5f), x), x), q0, q1);
  const uint64_t t = pk2(__fdividef(1.f, d0), __fdividef(1.f, d1));
  const uint64_t e = pk2(__expf(q0), __expf(q1));
  uint64_t p = fma2(t, pk2(1.061405429f, 1.061405429f), pk2(-1.453152027f, -1.453152027f));
  p = fma2(t, p, pk2(1.421413741f, 1.421413741f));
  p = fma2(t, p, pk2(-0.284496736f, -0.284496736f));
  p = fma2(t, p, pk2(0.254829592f, 0.254829592f));
  const uint64_t h = mul2(mul2(pk2(0.5f, 0.5f), mul2(p, t)), e);   // (1 - erf(u)) / 2
  float h0, h1, g0, g1;
  upk2(h, h0, h1);
  upk2(fma2(h, pk2(-1.f, -1.f), pk2(1.f, 1.f)), g0, g1);
  return Cdf2{pk2(x0 < 0.f ? h0 : g0, x1 < 0.f ? h1 : g1), e};
}
__device__ __forceinline__ void gelu_tc2(float& x0, float& x1) {
  upk2(mul2(pk2(x0, x1), cdf_tc2(x0, x1).cdf), x0, x1);
}
// y *= gelu'(x)
__device__ __forceinline__ void mul_gelu_grad_tc2(float x0, float x1, float& y0, float& y1) {
  const Cdf2 c = cdf_tc2(x0, x1);
  const uint64_t pdf = mul2(pk2(0.39894228040143267794f, 0.39894228040143267794f), c.e);
  upk2(mul2(pk2(y0, y1), fma2(pk2(x0, x1), pdf, c.cdf)), y0, y1);
}
__device__ __forceinline__ float sigmoid_tc(float x) { return __fdividef(1.f, 1.f + __expf(-x)); }

// Math of the level-fraction head in the scalar type of the caller: FP64 (the reference's arithmetic) or FP32.
__device__ __forceinline__ double mexp10(double x) { return exp10(x); }
__device__ __forceinline__ float mexp10(float x) { return exp10f(x); }
__device__ __forceinline__ double msqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float msqrt(float x) { return sqrtf(x); }

// MULTI3D constants, cgs (models/ffno_model.py:111-112)
constexpr double kEE = 1.602189e-12, kBK = 1.380662e-16;
constexpr double kLN10 = 2.302585092994045684;
constexpr double kINV_LN10 = 0.434294481903251827651;

// log(0.5 * (HH / sqrt(2 pi EM) / sqrt(BK))^3) with HH = 6.626176e-27, EM = 9.109534e-28, BK = 1.380662e-16 and
// pi = 3.14159265359: MULTI3D's Saha constant (models/ffno_model.py:112), evaluated once in 40-digit arithmetic (a
// CPU test recomputes it from the formula); as a literal it costs no FP64 log and square roots per voxel
constexpr double kLN_CCON = -36.113482555935598575;

// ------------------------------------------------------------------------------------------ level-fraction head
// One voxel of FFNO3D.head_output after proj2 (models/ffno_model.py:729-748): per species, logits = head channels + the
// LTE Boltzmann/Saha log-weights of (T, ne), log-softmax over the levels, plus the bounded total b tanh(u / b),
// log10 rho and the particle mass; normalised with mean_Y / std_Y. o: the voxel's head channels (species s: its L
// level logits, then its total channel). The LTE math and the log-softmax run in T: double is the reference's FP64
// (torch.log_softmax on float64 logits, :741); float is the split-BF16 path's FP32, where the sum of the max-shifted
// exponentials (each in (0, 1]) is compensated (below), so that the level shares of a voxel add up to 1 within a few
// FP32 roundings. The total term is FP64 in both; the final sum of log10 n is FP64 or two floats (HeadBase32).

// What the head's kernels take: the caller's parameters and whether every constant among them is an ordinary number:
// finite, the divisors (the bound of the totals, the scales std_Y) not zero either. Otherwise every voxel takes CUDA's
// functions and divisions, whose infinities and NaN the table functions below do not reproduce. So it does for a bound
// above 1e6 (a model whose totals are not to be bounded): b tanh(u / b) multiplies tanh_tab's absolute error by b, and
// up to 1e6 that stays four digits below a float32 rounding of the output. The host looks, at the launch (a warp of
// every CTA doing it took 3-9 us a launch).
struct HeadParams : ffno_head_params {
  int ordinary;
  explicit HeadParams(const ffno_head_params& p) : ffno_head_params(p) {
    auto divisor = [](float x, float most) { return fabsf(x) >= FLT_MIN && fabsf(x) <= most; };
    int levels = 0;
    for (int s = 0; s < nspecies && s < FFNO_MAX_SPECIES; ++s) levels += p.levels[s];
    bool ok = divisor(total_bound, 1e6f);
    for (int g = 0; g < levels && g < FFNO_MAX_LEVELS; ++g)
      ok = ok && divisor(std_y[g], FLT_MAX) && std::isfinite(log_g[g]) && std::isfinite(ev[g]) &&
           std::isfinite(ndxi[g]) && std::isfinite(dion[g]);
    ordinary = ok;
  }
};

struct HeadInputs {
  float lt, lne, lrho;   // log10 T, log10 ne (SI), log10 rho of the voxel (denormalised)
};

__device__ __forceinline__ HeadInputs head_inputs(const ffno_head_params& hp, const float* __restrict__ xin, long V,
                                                  long v) {
  const int tc = hp.temperature_channel, ec = hp.ne_channel, rc = hp.rho_channel;
  return HeadInputs{__ldg(xin + (long)tc * V + v), __ldg(xin + (long)ec * V + v), __ldg(xin + (long)rc * V + v)};
}

// FP64 elementary functions of the head. The FP64 pipe of this chip takes about two lanes a cycle and SM, so the head is
// bound by the number of its FP64 operations: about 1100 a voxel of two six-level species with CUDA's exp, log, exp10,
// tanh, division and square root, about 370 with these. Each is the textbook method, to a few 2^-53 of the result (tanh:
// of 1) on the range that the caller checks; outside it the head takes CUDA's functions.
//   exp(x) = 2^(n / 128) e^r, n = round(128 x / ln 2), |r| <= ln 2 / 256: a table of 2^(i / 128) (filled once per CTA
//     with exp2) and the Taylor polynomial of e^r - 1 to r^5 (remainder 5e-19);
//   10^x the same with n = round(128 x log2 10);
//   log(s), s near 1 .. 32: one Newton step y + e - e^2 / 2, e = s exp(-y) - 1, from FP32's y (e < 1e-6);
//   tanh(x) = sign(x) (1 - q) / (1 + q), q = exp(-2 |x|), to a few 2^-53 absolutely (1 - q cancels for small x);
//   1 / x: two Newton-Raphson steps from the hardware's 20-bit reciprocal.
constexpr int EXP_TAB = 128;
// ln 2 / 128 and log10(2) / 128 in two parts, the first with 32 trailing zero bits (its products with n are exact)
constexpr double LN2HI = 0.005415208637714386, LN2LO = 3.710410186743494e-09;
constexpr double LG2HI = 0.002351796254515648, LG2LO = 5.866092051994237e-10;

__device__ __forceinline__ void fill_exp_table(double* tab) {
  for (int i = threadIdx.x; i < EXP_TAB; i += blockDim.x) tab[i] = exp2((double)i / EXP_TAB);
}

__device__ __forceinline__ double rcp64(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// 2^(n / 128) e^r for |r| <= 0.003, n in a double's exponent range; t = n + 1.5 2^52 carries n in its low word
__device__ __forceinline__ double exp_parts(const double* tab, double t, double r) {
  const int n = __double2loint(t);
  double c = fma(r, 1.0 / 120, 1.0 / 24);
  c = fma(r, c, 1.0 / 6);
  c = fma(r, c, 0.5);
  const double p = fma(r * r, c, r);
  const double b = tab[n & (EXP_TAB - 1)];
  const double v = fma(b, p, b);
  return __hiloint2double(__double2hiint(v) + ((n >> 7) << 20), __double2loint(v));
}
constexpr double kRoundMagic = 6755399441055744.0;   // 1.5 2^52

// exp(x), x finite and below 700; 0 below -700 (a level's share there is under 1e-304)
__device__ __forceinline__ double exp_tab(const double* tab, double x) {
  const double t = fma(x, 184.6649652337873, kRoundMagic);
  const double n = t - kRoundMagic;
  const double r = fma(n, -LN2LO, fma(n, -LN2HI, x));
  const double v = exp_parts(tab, t, r);
  return (unsigned)__double2hiint(x) > 0xc085e000u ? 0.0 : v;
}
// 10^x, |x| < 300
__device__ __forceinline__ double exp10_tab(const double* tab, double x) {
  const double t = fma(x, 425.20679614558236, kRoundMagic);
  const double n = t - kRoundMagic;
  return exp_parts(tab, t, fma(n, -LG2LO, fma(n, -LG2HI, x)) * kLN10);
}
__device__ __forceinline__ double log_tab(const double* tab, double s) {
  const double y = (double)logf((float)s);
  const double e = fma(s, exp_tab(tab, -y), -1.0);
  return y + fma(-0.5 * e, e, e);
}
__device__ __forceinline__ double tanh_tab(const double* tab, double x) {
  const double q = exp_tab(tab, -2.0 * fabs(x));
  return copysign((1.0 - q) * rcp64(1.0 + q), x);
}

// The head's functions in T: FP64 by table where `fast`, else CUDA's.
template <typename T>
struct HeadMath;
template <>
struct HeadMath<double> {
  const double* tab;
  bool fast;   // ordinary constants, every head channel below 1e6 in size, 0.5 < log10 T < 15, |log10 ne| < 40
  __device__ __forceinline__ double exp_(double x) const { return fast ? exp_tab(tab, x) : exp(x); }
  __device__ __forceinline__ double log_(double x) const { return fast ? log_tab(tab, x) : log(x); }
  __device__ __forceinline__ double tanh_(double x) const { return fast ? tanh_tab(tab, x) : tanh(x); }
  __device__ __forceinline__ double inv_(double x) const { return fast ? rcp64(x) : 1.0 / x; }
};
template <>
struct HeadMath<float> {
  const double* tab;
  bool fast;
  __device__ __forceinline__ float exp_(float x) const { return expf(x); }
  __device__ __forceinline__ float log_(float x) const { return logf(x); }
  __device__ __forceinline__ float tanh_(float x) const { return tanhf(x); }
  __device__ __forceinline__ float inv_(float x) const { return 1.f / x; }
};

__device__ __forceinline__ bool head_fast(const HeadParams& hp, const float* o, int nh, const HeadInputs& in) {
  const float lt = fmaf(in.lt, hp.std_x[hp.temperature_channel], hp.mean_x[hp.temperature_channel]);
  const float ln = fmaf(in.lne, hp.std_x[hp.ne_channel], hp.mean_x[hp.ne_channel]);
  bool ok = hp.ordinary && lt > 0.5f && lt < 15.f && fabsf(ln) < 40.f;
  for (int c = 0; c < nh; ++c) ok = ok && fabsf(o[c]) < 1e6f;
  return ok;
}
__device__ __forceinline__ int head_channels(const ffno_head_params& hp) {
  int n = 0;
  for (int s = 0; s < hp.nspecies; ++s) n += hp.levels[s] + 1;
  return n;
}

template <typename T>
struct Lte {
  T lt, lne, conl, dxi, ek_t;
  __device__ __forceinline__ Lte(const ffno_head_params& hp, const HeadInputs& in, const HeadMath<T>& hm) {
    const int tc = hp.temperature_channel, ec = hp.ne_channel;
    const T LN10 = (T)kLN10;
    lt = (T)in.lt * (T)hp.std_x[tc] + (T)hp.mean_x[tc];
    lne = (T)in.lne * (T)hp.std_x[ec] + (T)hp.mean_x[ec];
    conl = (T)kLN_CCON + (lne - (T)6) * LN10 - (T)1.5 * lt * LN10;
    if constexpr (sizeof(T) == 8) {
      if (hm.fast) {   // 4.98e-4 5040 sqrt(BK) sqrt(ne / T), ne in cm^-3; E / (k T)
        dxi = 2.9491955176246003e-08 * exp10_tab(hm.tab, 0.5 * (lne - 6.0 - lt));
        ek_t = (kEE / kBK) * exp10_tab(hm.tab, -lt);
        return;
      }
    }
    const T tk = mexp10(lt);
    const T ne = mexp10(lne - (T)6);  // cm^-3
    dxi = (T)(4.98e-4 * 5040.0) / tk * msqrt(ne * (T)kBK * tk);
    ek_t = (T)(kEE / kBK) / tk;
  }
  // the LTE log-weight of level g
  __device__ __forceinline__ T weight(const ffno_head_params& hp, int g) const {
    return (T)hp.log_g[g] - ek_t * ((T)hp.ev[g] - dxi * (T)hp.ndxi[g]) - (T)hp.dion[g] * conl;
  }
};

// sum_i exp(logit[i] - mx), i < L. FP64: a plain sum (the reference's float64 logsumexp). FP32: Neumaier's
// improved Kahan-Babuska summation (A. Neumaier, "Rundungsfehleranalyse einiger Verfahren zur Summation endlicher
// Summen", ZAMM 54 (1974) 39-51): the rounding error of every addition is carried in c and added once at the end,
// so the result is the exactly rounded sum of the rounded terms up to O(L u^2).
__device__ __forceinline__ double shifted_exp_sum(const HeadMath<double>& hm, const double* logit, int L, double mx) {
  double s = 0;
  for (int i = 0; i < L; ++i) s += hm.exp_(logit[i] - mx);
  return s;
}
__device__ __forceinline__ float shifted_exp_sum(const HeadMath<float>&, const float* logit, int L, float mx) {
  float s = 0.f, c = 0.f;
  for (int i = 0; i < L; ++i) {
    const float t = expf(logit[i] - mx);
    const float u = s + t;
    c += fabsf(s) >= fabsf(t) ? (s - u) + t : (t - u) + s;
    s = u;
  }
  return s + c;
}

// log10 n - mean_y of one level from base (log10 n of the whole species), the level's shifted logit d and the log-sum lse:
// base + (d - lse) / ln 10 - mean, the large terms cancelling. FP64: in FP64.
struct HeadBase64 {
  double base;
  __device__ __forceinline__ explicit HeadBase64(double b) : base(b) {}
  __device__ __forceinline__ float level(double d, double lse, float mean) const {
    return (float)(base + (d - lse) * kINV_LN10 - (double)mean);
  }
};
// FP32 (the split-BF16 path): in pairs of floats (value and rounding error, 48 bits), by the error-free sum of Knuth and
// the error-free product by fused multiply-add: 20 FP32 operations where the FP64 form has 6 at 1 / 64 of the rate. The
// result, rounded to float, is the FP64 form's in all but 2 of 4 million random assemblies (log10 n of 5 to 40).
__device__ __forceinline__ float two_sum(float a, float b, float& err) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  err = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
  return s;
}
struct HeadBase32 {
  float hi, lo;
  __device__ __forceinline__ explicit HeadBase32(double b) : hi((float)b) { lo = (float)(b - (double)hi); }
  __device__ __forceinline__ float level(float d, float lse, float mean) const {
    constexpr float IH = 0.4342944920063019f, IL = -1.0103050052231683e-08f;   // 1 / ln 10 in two floats
    float de, me, se;
    const float dd = two_sum(d, -lse, de);
    const float p = __fmul_rn(dd, IH);
    const float pe = fmaf(dd, IL, fmaf(de, IH, fmaf(dd, IH, -p)));
    const float m = two_sum(hi, -mean, me);
    const float r = two_sum(m, p, se);
    // an infinite base or level: the plain sum is the answer (-inf for a density of zero or an empty level), and the
    // error terms are inf - inf
    return fabsf(r) <= 3.402823466e38f ? __fadd_rn(r, __fadd_rn(se, __fadd_rn(__fadd_rn(me, lo), pe))) : r;
  }
};
__device__ __forceinline__ HeadBase64 head_base(double b, double) { return HeadBase64(b); }
__device__ __forceinline__ HeadBase32 head_base(double b, float) { return HeadBase32(b); }

// Forward: out[g * V + v] = the normalised log10 population of level g. tab: fill_exp_table's.
template <typename T>
__device__ __forceinline__ void head_voxel_fwd(const HeadParams& hp, const float* o, const HeadInputs& in,
                                               float* __restrict__ out, long V, long v, const double* tab) {
  HeadMath<T> hm{tab, false};
  if constexpr (sizeof(T) == 8) hm.fast = head_fast(hp, o, head_channels(hp), in);
  const Lte<T> e(hp, in, hm);
  // the total term and the assembly of log10 n (log10 rho - log10 m + s ~ 20, minus mean_Y) stay beyond FP32 for both
  // T: in FP32 their rounding (~1e-6 dex at that magnitude, and a few ulp of b for tanh) would move every level of
  // the voxel against its total, past the 1e-6 bar on the level shares' sum
  const double lrho = (double)in.lrho * (double)hp.std_x[hp.rho_channel] + (double)hp.mean_x[hp.rho_channel];
  int hc = 0, lvl = 0;
  for (int s = 0; s < hp.nspecies; ++s) {
    const int L = hp.levels[s];
    T logit[FFNO_MAX_LEVELS];
    T mx = (T)-1e30;
    for (int i = 0; i < L; ++i) {
      logit[i] = (T)o[hc + i] + e.weight(hp, lvl + i);
      mx = fmax(mx, logit[i]);
    }
    const T lse = hm.log_(shifted_exp_sum(hm, logit, L, mx));
    const double tb = (double)hp.total_bound;
    const float u = o[hc + L];
    const double th =
        hp.ordinary && fabsf(u) < 1e6f ? tanh_tab(tab, (double)u * rcp64(tb)) : tanh((double)u / tb);
    const auto base = head_base(lrho - (double)hp.log10_particle_mass[s] + tb * th, T(0));
    for (int i = 0; i < L; ++i) {
      const int g = lvl + i;
      // the large terms cancel before the difference (a few units) is normalised in FP32
      out[(long)g * V + v] = base.level(logit[i] - mx, lse, hp.mean_y[g]) / hp.std_y[g];
    }
    hc += L + 1;
    lvl += L;
  }
}

// Backward: with ybar[g * V + v] the cotangent of the normalised output, overwrites o[0..nhp) with the gradient of the
// head channels (zero past the last species) and writes x_in_bar[k * V + v] for every input channel k.
template <typename T>
__device__ __forceinline__ void head_voxel_bwd(const HeadParams& hp, float* o, int nhp, const HeadInputs& in,
                                               const float* __restrict__ ybar, long V, long v,
                                               float* __restrict__ xinbar, const double* tab) {
  HeadMath<T> hm{tab, false};
  if constexpr (sizeof(T) == 8) hm.fast = head_fast(hp, o, head_channels(hp), in);
  const Lte<T> e(hp, in, hm);
  T gsum = 0, ltb = 0, lneb = 0;
  int hc = 0, lvl = 0;
  for (int s = 0; s < hp.nspecies; ++s) {
    const int L = hp.levels[s];
    T logit[FFNO_MAX_LEVELS], gl[FFNO_MAX_LEVELS];
    T mx = (T)-1e30;
    for (int i = 0; i < L; ++i) {
      logit[i] = (T)o[hc + i] + e.weight(hp, lvl + i);
      mx = fmax(mx, logit[i]);
    }
    const T se = shifted_exp_sum(hm, logit, L, mx), ise = hm.inv_(se);
    T G = 0;
    for (int i = 0; i < L; ++i) {
      gl[i] = (T)__ldg(ybar + (long)(lvl + i) * V + v);
      gl[i] = sizeof(T) == 8 ? gl[i] * hm.inv_((T)hp.std_y[lvl + i]) : gl[i] / (T)hp.std_y[lvl + i];
      G += gl[i];
    }
    gsum += G;
    const T tb = (T)hp.total_bound;
    const T th = hm.tanh_(sizeof(T) == 8 ? (T)o[hc + L] * hm.inv_(tb) : (T)o[hc + L] / tb);
    const float ubar = (float)(G * ((T)1 - th * th));
    for (int i = 0; i < L; ++i) {
      const int g = lvl + i;
      const T ex = hm.exp_(logit[i] - mx), p = sizeof(T) == 8 ? ex * ise : ex / se;
      const T d = gl[i] - p * G;                    // the logit's gradient times ln 10
      const T lb = d * (T)kINV_LN10;
      o[hc + i] = (float)lb;
      ltb += d * (e.ek_t * ((T)hp.ev[g] - (T)1.5 * e.dxi * (T)hp.ndxi[g]) + (T)1.5 * (T)hp.dion[g]);
      lneb += d * ((T)0.5 * e.ek_t * e.dxi * (T)hp.ndxi[g] - (T)hp.dion[g]);
    }
    o[hc + L] = ubar;
    hc += L + 1;
    lvl += L;
  }
  for (int c = hc; c < nhp; ++c) o[c] = 0.f;
  const int tc = hp.temperature_channel, ec = hp.ne_channel, rc = hp.rho_channel;
  for (int k = 0; k < hp.in_channels; ++k) {
    T val = 0;
    if (k == tc) val += ltb * (T)hp.std_x[tc];
    if (k == ec) val += lneb * (T)hp.std_x[ec];
    if (k == rc) val += gsum * (T)hp.std_x[rc];
    xinbar[(long)k * V + v] = (float)val;
  }
}

// Copy rows v0 .. v0 + rows - 1 (C floats each, row-major, contiguous) into shared memory with row stride lds; rows at
// or beyond V are zero.
template <int C>
__device__ __forceinline__ void load_rows(float* __restrict__ s, int lds, const float* __restrict__ g, long v0, long V,
                                          int rows = BM) {
  constexpr int Q = C / 4;  // float4 per row
  for (int e = threadIdx.x; e < rows * Q; e += NT) {
    const int r = e / Q, q = e % Q;
    float4 val = make_float4(0.f, 0.f, 0.f, 0.f);
    if (v0 + r < V) val = __ldg(reinterpret_cast<const float4*>(g + (v0 + r) * C) + q);
    float* d = s + r * lds + 4 * q;
    d[0] = val.x; d[1] = val.y; d[2] = val.z; d[3] = val.w;
  }
}

// Running weighted group statistics (total weight, mean, M2) of one CTA, merged tile by tile with Chan's parallel
// update so that no long single-precision sum and no E[x^2] - E[x]^2 cancellation occurs.
struct GroupAcc {
  double w, mean, m2;
};

__device__ __forceinline__ void chan_merge(GroupAcc& a, double wt, double mt, double m2t) {
  if (wt <= 0.0) return;
  const double wn = a.w + wt;
  const double delta = mt - a.mean;
  a.mean += delta * (wt / wn);
  a.m2 += m2t + delta * delta * (a.w * wt / wn);
  a.w = wn;
}

// The same running statistics without a division per merge: sums of w, w (mean - ref) and m2 + w (mean - ref)^2 about
// the first merged mean, in FP64. A Chan merge has two dependent FP64 divisions, microseconds of a serial chain on this
// chip's FP64 pipe, where a tile's whole budget is three; this is five FP64 multiply-adds whose results nothing waits
// for. get(): the (w, mean, m2) that the Chan merges would have given, to FP64 rounding about ref.
struct ShiftAcc {
  double w = 0.0, s1 = 0.0, s2 = 0.0, ref = 0.0;
  __device__ __forceinline__ void add(float wt, float mean, float m2) {
    if (wt <= 0.f) return;   // a NaN weight counts
    if (w == 0.0) ref = (double)mean;
    const double d = (double)mean - ref, wd = (double)wt * d;
    w += (double)wt;
    s1 += wd;
    s2 += (double)m2 + wd * d;
  }
  __device__ __forceinline__ GroupAcc get() const {
    if (w == 0.0) return GroupAcc{0.0, 0.0, 0.0};
    const double m = s1 / w;
    const double m2 = s2 - s1 * m;
    return GroupAcc{w, ref + m, m2 < 0.0 ? 0.0 : m2};
  }
};

// Sum of s[g] over the warp's lanes, for the group g = lane / 4: a butterfly that halves the groups a lane carries at
// each step (9 shuffles for the eight sums; 40 when every lane reduces all of them).
__device__ __forceinline__ float warp_group_sum(const float (&s)[GMAX]) {
  static_assert(GMAX == 8, "three halving steps");
  const int lane = threadIdx.x & 31;
  float a[4], b[2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float keep = (lane & 16) ? s[4 + i] : s[i], send = (lane & 16) ? s[i] : s[4 + i];
    a[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const float keep = (lane & 8) ? a[2 + i] : a[i], send = (lane & 8) ? a[i] : a[2 + i];
    b[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  float r = ((lane & 4) ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, (lane & 4) ? b[0] : b[1], 4);
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  r += __shfl_xor_sync(0xffffffffu, r, 1);
  return r;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The partials row of a CTA from NW warps' statistics acc[warp][group] (shared memory, written before a barrier), merged
// in warp order by thread g.
template <int NW>
__device__ __forceinline__ void write_warp_partials(double* partials, const double (&acc)[NW][GMAX][3]) {
  if (threadIdx.x < GMAX) {
    const int g = threadIdx.x;
    GroupAcc a{0.0, 0.0, 0.0};
#pragma unroll 1
    for (int w = 0; w < NW; ++w) chan_merge(a, acc[w][g][0], acc[w][g][1], acc[w][g][2]);
    double* o = partials + ((long)blockIdx.x * GMAX + g) * 3;
    o[0] = a.w;
    o[1] = a.mean;
    o[2] = a.m2;
  }
}

// Lane 4 g's running statistics of group g into the warp's row of acc.
__device__ __forceinline__ void put_warp_stats(double (*acc)[3], const ShiftAcc& st) {
  const int lane = threadIdx.x & 31;
  if ((lane & 3) == 0) {
    const GroupAcc a = st.get();
    acc[lane >> 2][0] = a.w;
    acc[lane >> 2][1] = a.mean;
    acc[lane >> 2][2] = a.m2;
  }
}

// Partials row [groups][2] of this CTA (8 warps) from every lane's VW channel sums (channels VW q ..): over the lanes that
// hold the same channels by shuffles, over the warps per channel, then over each group's channels, in a fixed order. The
// FP64 pipe is narrow (about two lanes a cycle and SM), so each value is added a few times only: eight groups by a
// full-warp double reduction each were 80 double additions a lane, 25 us a launch. Rows past the grid hold zeros.
template <int C, int VW>
__device__ __forceinline__ void stats_partial_rows(double (&d1)[VW], double (&d2)[VW], bool active, int q, int cpg,
                                                   int groups, int nparts, double* __restrict__ partials) {
  constexpr int LPV = C / VW;
  constexpr bool POW2 = LPV <= 32 && (LPV & (LPV - 1)) == 0;
  __shared__ double ch[2][8][C];
  __shared__ double sum[2][C];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < VW; ++j) {
    if constexpr (POW2) {
#pragma unroll
      for (int o = 16; o >= LPV; o >>= 1) {
        d1[j] += __shfl_xor_sync(0xffffffffu, d1[j], o);
        d2[j] += __shfl_xor_sync(0xffffffffu, d2[j], o);
      }
    }
    if (active && lane < LPV) {
      ch[0][warp][VW * q + j] = d1[j];
      ch[1][warp][VW * q + j] = d2[j];
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 2 * C; e += blockDim.x) {
    const int i = e / C, c = e % C;
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += ch[i][w][c];
    sum[i][c] = s;
  }
  __syncthreads();
  if (threadIdx.x < 2 * groups) {
    const int g = threadIdx.x >> 1, i = threadIdx.x & 1;
    double s = 0.0;
    for (int c = g * cpg; c < (g + 1) * cpg; ++c) s += sum[i][c];
    partials[((long)blockIdx.x * groups + g) * 2 + i] = s;
    for (long p = blockIdx.x + gridDim.x; p < nparts; p += gridDim.x) partials[(p * groups + g) * 2 + i] = 0.0;
  }
}

// The dynamic shared memory a kernel may take is a process-wide attribute of that kernel. The service launches the
// same kernels from several host threads with different sizes (one request per thread), and a thread that lowered the
// attribute to its own size between another thread's setting and that thread's launch made the launch fail. So the
// attribute is set once per kernel and device, under a lock, to the most the kernel can have there (the opt-in maximum
// per block less the kernel's static shared memory), and each launch only checks its own size against that cap.
bool smem_cap_lookup(const void* kernel, size_t* cap);

template <typename K>
inline bool smem_cap_ok(K kernel, size_t bytes) {
  if (bytes <= 40 * 1024) return true;   // 48 KB without the attribute, the kernel's static shared memory included
  size_t cap = 0;
  if (!smem_cap_lookup(reinterpret_cast<const void*>(kernel), &cap)) return false;
  return bytes <= cap;
}

// Programmatic dependent launch. The model kernels are launched with it allowed (launch below): the next kernel
// of the stream is set up and its CTAs placed while this one drains, which takes the 2-3 us between two dependent
// kernels (half of a small cube's kernels last 5-25 us) down to about 1. A kernel touches global memory only after
// griddep_wait, which returns once the kernel before it in the stream has completed with its writes visible; it lets
// its own successor be placed only after that (and, where it owns tensor memory, after it has allocated it: a placed
// successor never holds what its predecessor still needs). With every kernel waiting for its predecessor, completion
// stays in stream order. Kernels of other libraries before or after see ordinary stream order.
__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void griddep_sync() {
  griddep_wait();
  griddep_launch();
}

// launch_if(early, ...) allows it only if early. Kernels placed while their predecessor drains go to the SMs that free up
// first: some then run longer (their L1 / shared-memory split is the predecessor's, and grids below the resident limit
// pile up on few SMs). Measured against an ordinary launch: width-96 gate backward 1.07 -> 1.32 ms and fusion output
// 1.39 -> 1.61 ms (1.0 M voxels), gate forward 310 -> 328 us, gate backward 728 -> 759, MLP forward 379 -> 396, GroupNorm
// backward 320 -> 348 (2.4 M voxels, C = 64). These kernels pass early_launch(V, C): at 61 k voxels, C = 64, their
// 15-25 us gain 2 us from it; at 250-340 k (about 100 us) gain and loss are equal.
inline bool early_launch(long V, int C) { return V * C <= (1L << 24); }

template <typename... P, typename... A>
inline void launch_if(bool early, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream,
                      A&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = early ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);   // its error is read by FFNO_CHECK_LAUNCH
}

template <typename... P, typename... A>
inline void launch(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t stream, A&&... args) {
  launch_if(true, kernel, grid, block, smem, stream, static_cast<A&&>(args)...);
}

}  // namespace ffno

#define FFNO_CHECK_LAUNCH()                                   \
  do {                                                        \
    cudaError_t e_ = cudaGetLastError();                      \
    if (e_ != cudaSuccess) return FFNO_ELAUNCH;               \
  } while (0)
