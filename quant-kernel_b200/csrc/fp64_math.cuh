// fp64_math.cuh -- FP64 elementary functions on bounded arguments.
//
// The terminal Monte Carlo and Fourier kernels are bound by the FP64 pipe
// (64 lanes per SM and clock) and by the instructions around it.  CUDA's
// exp, log, sincos, atan2, sqrt and division serve every argument; here the
// callers know theirs to be finite and in range, so special cases, scaling and
// slow-path branches go, and small tables in shared memory shorten the
// polynomials (the load/store pipe is idle in these kernels):
//   exp     16-entry table of 2^(j/16), degree-6 remainder     11 FP64 ops
//   log     32-entry reciprocal table, degree-8 log1p          14
//   sincos  32-entry table at multiples of pi/16, degree 9/8   18
//   atan2   17-entry table at multiples of 1/16, degree 9      22
//   1/x, sqrt  hardware seed and one third-order step          3 + seed, 5 + seed
// Table sizes keep a warp's random 8-byte lookups within two shared-memory
// wavefronts per half-warp.  The remainder polynomials are interpolants at
// Chebyshev nodes (near-minimax) of exp, log1p, sin, cos and atan; their
// errors, and the tables', are given beside each.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace qkb {

struct Fp64Tables {
    double exp_hi[16], exp_lo[16];  // 2^(j/16) as hi + lo
    double cs_cos[32], cs_sin[32];  // cos, sin of j pi/16
    double log_v[32];               // -log(c_j)
    double atan_v[18];              // atan(j/16), one word of padding
    uint32_t log_c[32];             // high word of c_j ~ 1 / (centre of interval j), low word 0
};
constexpr int kFp64TableWords = (int)(sizeof(Fp64Tables) / sizeof(double));
static_assert(sizeof(Fp64Tables) % sizeof(double) == 0, "copied in 8-byte words");

static __device__ const Fp64Tables g_fp64_tables = {
    {0x1.0000000000000p+0, 0x1.0b5586cf9890fp+0, 0x1.172b83c7d517bp+0, 0x1.2387a6e756238p+0,
     0x1.306fe0a31b715p+0, 0x1.3dea64c123422p+0, 0x1.4bfdad5362a27p+0, 0x1.5ab07dd485429p+0,
     0x1.6a09e667f3bcdp+0, 0x1.7a11473eb0187p+0, 0x1.8ace5422aa0dbp+0, 0x1.9c49182a3f090p+0,
     0x1.ae89f995ad3adp+0, 0x1.c199bdd85529cp+0, 0x1.d5818dcfba487p+0, 0x1.ea4afa2a490dap+0},
    {0x0.0p+0, 0x1.8a62e4adc610bp-54, -0x1.19041b9d78a76p-55, 0x1.9b07eb6c70573p-54,
     0x1.6f46ad23182e4p-55, 0x1.ada0911f09ebcp-55, 0x1.d4397afec42e2p-56, 0x1.6324c054647adp-54,
     -0x1.bdd3413b26456p-54, -0x1.41577ee04992fp-55, 0x1.6e9f156864b27p-54,
     0x1.c7c46b071f2bep-56, 0x1.7a1cd345dcc81p-54, 0x1.11065895048ddp-55, 0x1.2ed02d75b3707p-55,
     -0x1.e9c23179c2893p-54},
    {0x1.0000000000000p+0, 0x1.f6297cff75cb0p-1, 0x1.d906bcf328d46p-1, 0x1.a9b66290ea1a3p-1,
     0x1.6a09e667f3bcdp-1, 0x1.1c73b39ae68c8p-1, 0x1.87de2a6aea963p-2, 0x1.8f8b83c69a60bp-3,
     0x0.0p+0, -0x1.8f8b83c69a60bp-3, -0x1.87de2a6aea963p-2, -0x1.1c73b39ae68c8p-1,
     -0x1.6a09e667f3bcdp-1, -0x1.a9b66290ea1a3p-1, -0x1.d906bcf328d46p-1, -0x1.f6297cff75cb0p-1,
     -0x1.0000000000000p+0, -0x1.f6297cff75cb0p-1, -0x1.d906bcf328d46p-1, -0x1.a9b66290ea1a3p-1,
     -0x1.6a09e667f3bcdp-1, -0x1.1c73b39ae68c8p-1, -0x1.87de2a6aea963p-2, -0x1.8f8b83c69a60bp-3,
     0x0.0p+0, 0x1.8f8b83c69a60bp-3, 0x1.87de2a6aea963p-2, 0x1.1c73b39ae68c8p-1,
     0x1.6a09e667f3bcdp-1, 0x1.a9b66290ea1a3p-1, 0x1.d906bcf328d46p-1, 0x1.f6297cff75cb0p-1},
    {0x0.0p+0, 0x1.8f8b83c69a60bp-3, 0x1.87de2a6aea963p-2, 0x1.1c73b39ae68c8p-1,
     0x1.6a09e667f3bcdp-1, 0x1.a9b66290ea1a3p-1, 0x1.d906bcf328d46p-1, 0x1.f6297cff75cb0p-1,
     0x1.0000000000000p+0, 0x1.f6297cff75cb0p-1, 0x1.d906bcf328d46p-1, 0x1.a9b66290ea1a3p-1,
     0x1.6a09e667f3bcdp-1, 0x1.1c73b39ae68c8p-1, 0x1.87de2a6aea963p-2, 0x1.8f8b83c69a60bp-3,
     0x0.0p+0, -0x1.8f8b83c69a60bp-3, -0x1.87de2a6aea963p-2, -0x1.1c73b39ae68c8p-1,
     -0x1.6a09e667f3bcdp-1, -0x1.a9b66290ea1a3p-1, -0x1.d906bcf328d46p-1, -0x1.f6297cff75cb0p-1,
     -0x1.0000000000000p+0, -0x1.f6297cff75cb0p-1, -0x1.d906bcf328d46p-1, -0x1.a9b66290ea1a3p-1,
     -0x1.6a09e667f3bcdp-1, -0x1.1c73b39ae68c8p-1, -0x1.87de2a6aea963p-2, -0x1.8f8b83c69a60bp-3},
    {-0x1.68ac7fe9c69f4p-2, -0x1.522ad0738a1d8p-2, -0x1.3c251f7333104p-2, -0x1.269611134d992p-2,
     -0x1.1178f9227e23ap-2, -0x1.f991aacb3b069p-3, -0x1.d103772655e3bp-3, -0x1.a93ecbc8ad9a3p-3,
     -0x1.823c18551a3bep-3, -0x1.5bf422b543aa2p-3, -0x1.365fb90158ed2p-3, -0x1.117918227db7cp-3,
     -0x1.da72063842e22p-4, -0x1.93358dd593a69p-4, -0x1.4d30bdd206f8cp-4, -0x1.08597b59e3987p-4,
     -0x1.894a0949f9cb3p-5, -0x1.0415c89e74404p-5, -0x1.0205258935647p-6, 0x0.0p+0,
     0x1.f82990e783380p-6, 0x1.f0a32c01163a6p-5, 0x1.6f0d38ae56bccp-4, 0x1.e27086e2af366p-4,
     0x1.29553581ff547p-3, 0x1.5ff2f30a79564p-3, 0x1.9525b1cf456f4p-3, 0x1.c8ff5c79a9e22p-3,
     0x1.fb9162d5e433bp-3, 0x1.1675cebaba62ep-2, 0x1.2e8e36ae11e23p-2, 0x1.4618d021c61e2p-2},
    {0x0.0p+0, 0x1.ff55bb72cfdeap-5, 0x1.fd5ba9aac2f6ep-4, 0x1.7b97b4bce5b02p-3,
     0x1.f5b75f92c80ddp-3, 0x1.362773707ebccp-2, 0x1.6f61941e4def1p-2, 0x1.a64eec3cc23fdp-2,
     0x1.dac670561bb4fp-2, 0x1.0657e94db30d0p-1, 0x1.1e00babdefeb4p-1, 0x1.345f01cce37bbp-1,
     0x1.4978fa3269ee1p-1, 0x1.5d58987169b18p-1, 0x1.700a7c5784634p-1, 0x1.819d0b7158a4dp-1,
     0x1.921fb54442d18p-1, 0.0},
    {0x3FF6C16Cu, 0x3FF642C8u, 0x3FF5C988u, 0x3FF55555u, 0x3FF4E5E1u, 0x3FF47AE1u, 0x3FF41414u,
     0x3FF3B13Bu, 0x3FF3521Du, 0x3FF2F685u, 0x3FF29E41u, 0x3FF24925u, 0x3FF1F704u, 0x3FF1A7B9u,
     0x3FF15B1Eu, 0x3FF11111u, 0x3FF0C971u, 0x3FF08421u, 0x3FF04104u, 0x3FF00000u, 0x3FEF07C2u,
     0x3FEE1E1Eu, 0x3FED41D4u, 0x3FEC71C7u, 0x3FEBACF9u, 0x3FEAF287u, 0x3FEA41A4u, 0x3FE9999Au,
     0x3FE8F9C2u, 0x3FE86186u, 0x3FE7D05Fu, 0x3FE745D1u}};

// Coefficients with a nonzero low word, read by the FMAs straight from the
// constant bank: as immediates each took two moves, a third of the
// instructions of a Sobol point (152 -> 125 a point, 402 -> 380 us for 64
// options of 2^20 points).
struct Fp64Consts {
    double exp_scale, exp_hi, exp_lo, exp_p[4];
    double log_p[6], ln2_hi, ln2_lo;
    double sin_p[4], cos_p[3];
    double pi16_scale, pi16_hi, pi16_lo;
    double atan_p[4], pi_2, pi;
};
static __constant__ Fp64Consts c_fp64 = {
    // 16/ln2, ln2/16 in two parts; (e^r - 1 - r)/r^2 on |r| <= ln2/32, highest first (then 1/2)
    0x1.71547652b82fep+4, 0x1.62e42fefa39efp-5, 0x1.abc9e3b39803fp-60,
    {0x1.6c17bb5ebddb4p-10, 0x1.11120b03cd855p-7, 0x1.555555551946fp-5, 0x1.55555554dd388p-3},
    // (log(1 + r) - r)/r^2 on |r| <= 1/64 (then -1/2); ln2, the first part in 40 bits
    {-0x1.00174fa61038ep-3, 0x1.24ac2fd4eb4f0p-3, -0x1.555554934b74fp-3, 0x1.999998c200bfcp-3,
     -0x1.0000000000c9ep-2, 0x1.555555555635ap-2},
    0x1.62e42fefa2000p-1, 0x1.9ef35793c7673p-41,
    // (sin r - r)/r^3 and (cos r - 1)/r^2 (then -1/2) in r^2 on |r| <= pi/32
    {0x1.71cda20bfd969p-19, -0x1.a01a0139b7e26p-13, 0x1.111111111046fp-7, -0x1.5555555555555p-3},
    {0x1.a00330523baa9p-16, -0x1.6c16c0df50911p-10, 0x1.5555555553298p-5},
    // 16/pi, pi/16 in two parts
    0x1.45f306dc9c883p+2, 0x1.921fb54442d18p-3, 0x1.1a62633145c07p-57,
    // (atan r - r)/r^3 in r^2 on |r| <= 1/31
    {0x1.c65ebd82ab3b3p-4, -0x1.24923a079cf0bp-3, 0x1.99999998d44abp-3, -0x1.5555555555549p-2},
    0x1.921fb54442d18p+0, 0x1.921fb54442d18p+1};

// The CTA's copy of the tables; the caller synchronises before using it.
__device__ __forceinline__ void fp64_load_tables(Fp64Tables& t) {
    const double* src = reinterpret_cast<const double*>(&g_fp64_tables);
    double* dst = reinterpret_cast<double*>(&t);
    for (int i = threadIdx.x; i < kFp64TableWords; i += blockDim.x) dst[i] = src[i];
}

// Seeds from the special-function unit: the operand's and the result's upper
// 32 bits, relative error below 2^-19.
__device__ __forceinline__ double fp64_rcp_seed(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
__device__ __forceinline__ double fp64_rsqrt_seed(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}

// 1/x for normal x with a normal reciprocal: from 1/x = y (1 - e)^-1, e = 1 - x y,
// the geometric series to its square (Householder's method of the third order
// for 1/y - x), which leaves e^3 < 2^-57.
__device__ __forceinline__ double fp64_rcp(double x) {
    const double y = fp64_rcp_seed(x);
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// 1/sqrt(x), sqrt(x) for normal x > 0: from x^(-1/2) = y (1 - e)^(-1/2), e = 1 -
// x y^2, the binomial series 1 + e/2 + 3 e^2/8 (the same method for y^-2 - x),
// which leaves (5/16) e^3 < 2^-55 (e < 2^-18).
__device__ __forceinline__ double fp64_rsqrt(double x) {
    const double y = fp64_rsqrt_seed(x);
    const double e = fma(-(x * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ double fp64_sqrt(double x) {
    const double y = fp64_rsqrt_seed(x);
    const double t = x * y;
    const double e = fma(-t, y, 1.0);
    return fma(t * e, fma(0.375, e, 0.5), t);
}

// exp(x), |x| <= 700: x = k ln2/16 + r, |r| <= ln2/32; e^r to 2.8e-17.  LO
// adds the table's low part: below 0.8 ulp (CUDA's exp: 1 ulp); without it
// below 1.3 ulp.
template <bool LO>
__device__ __forceinline__ double fp64_exp(double x, const Fp64Tables& t) {
    constexpr double kMagic = 0x1.8p+52;
    const double kf = fma(x, c_fp64.exp_scale, kMagic);
    const int32_t k = __double2loint(kf);
    const double kd = kf - kMagic;
    const double r = fma(-kd, c_fp64.exp_lo, fma(-kd, c_fp64.exp_hi, x));
    double p = fma(c_fp64.exp_p[0], r, c_fp64.exp_p[1]);
    p = fma(p, r, c_fp64.exp_p[2]);
    p = fma(p, r, c_fp64.exp_p[3]);
    p = fma(p, r, 0.5);
    const double q = fma(p, r * r, r);
    const double T = t.exp_hi[k & 15];
    const double y = LO ? T + fma(T, q, t.exp_lo[k & 15]) : fma(T, q, T);
    return __hiloint2double(__double2hiint(y) + (k & ~15) * 65536, __double2loint(y));
}

// log(x) for normal x > 0: x = 2^e m with m in [0.695, 1.39), interval j of 32
// (an interval around 1 has c = 1, so results near 0 keep their relative
// accuracy), r = m c - 1, |r| <= 1/64; log1p(r) to 8e-18 relative.
__device__ __forceinline__ double fp64_log(double x, const Fp64Tables& t) {
    const int32_t hi = __double2hiint(x);
    const int32_t d = hi - 0x3FE64000;
    const int32_t e = d >> 20;
    const double m = __hiloint2double(hi - (e << 20), __double2loint(x));
    const int32_t j = (d >> 15) & 31;
    // e as a double, exactly: e + 2^31 into the mantissa of 2^52
    const double ed = __hiloint2double(0x43300000, (int32_t)((uint32_t)e ^ 0x80000000u)) -
                      (0x1p+52 + 0x1p+31);
    const double r = fma(m, __hiloint2double((int32_t)t.log_c[j], 0), -1.0);
    double p = fma(c_fp64.log_p[0], r, c_fp64.log_p[1]);
#pragma unroll
    for (int i = 2; i < 6; ++i) p = fma(p, r, c_fp64.log_p[i]);
    p = fma(p, r, -0.5);
    // e ln2 in two parts, the first exact; the low part joins the small terms
    const double base = fma(ed, c_fp64.ln2_hi, t.log_v[j]);
    return base + (r + fma(p, r * r, ed * c_fp64.ln2_lo));
}

// sin and cos of the angle (j pi/16 + r) given |r| <= pi/32 (table index j).
__device__ __forceinline__ void fp64_sincos_at(int32_t j, double r, const Fp64Tables& t, double& s,
                                               double& c) {
    const double S = t.cs_sin[j & 31], C = t.cs_cos[j & 31];
    const double y = r * r;
    double a = fma(c_fp64.sin_p[0], y, c_fp64.sin_p[1]);
    a = fma(a, y, c_fp64.sin_p[2]);
    a = fma(a, y, c_fp64.sin_p[3]);
    const double sn = fma(a, r * y, r);
    double b = fma(c_fp64.cos_p[0], y, c_fp64.cos_p[1]);
    b = fma(b, y, c_fp64.cos_p[2]);
    b = fma(b, y, -0.5);
    const double cm = b * y;  // cos r - 1
    s = fma(C, sn, fma(S, cm, S));
    c = fma(-S, sn, fma(C, cm, C));
}

// x = k pi/16 + r for |x| < 2^48 (two-part pi/16; r to 2^-56 while |k| < 2^51).
__device__ __forceinline__ double fp64_reduce_pi16(double x, int32_t& k) {
    constexpr double kMagic = 0x1.8p+52;
    const double kf = fma(x, c_fp64.pi16_scale, kMagic);
    k = __double2loint(kf);
    const double kd = kf - kMagic;
    return fma(-kd, c_fp64.pi16_lo, fma(-kd, c_fp64.pi16_hi, x));
}
__device__ __forceinline__ void fp64_sincos(double x, const Fp64Tables& t, double& s, double& c) {
    int32_t k;
    const double r = fp64_reduce_pi16(x, k);
    fp64_sincos_at(k, r, t, s, c);
}

// atan2(y, x) for finite x, y with x^2 + y^2 normal: q = min/max = tan(atan(j/16) + a),
// a = atan((lo - c hi) / (hi + c lo)), |a| <= 1/31; the octant from the signs.
__device__ __forceinline__ double fp64_atan2(double y, double x, const Fp64Tables& t) {
    const double ax = fabs(x), ay = fabs(y);
    const bool swap = ay > ax;
    const double hi = swap ? ay : ax, lo = swap ? ax : ay;
    constexpr double kMagic = 0x1.8p+52;
    const double kf = fma(lo * 16.0, fp64_rcp_seed(hi), kMagic);
    const int32_t j = __double2loint(kf);
    const double c = (kf - kMagic) * 0.0625;
    const double num = fma(-c, hi, lo), den = fma(c, lo, hi);
    const double r = num * fp64_rcp(den);
    const double z = r * r;
    double p = fma(c_fp64.atan_p[0], z, c_fp64.atan_p[1]);
    p = fma(p, z, c_fp64.atan_p[2]);
    p = fma(p, z, c_fp64.atan_p[3]);
    double a = t.atan_v[j] + fma(p, r * z, r);
    if (swap) a = c_fp64.pi_2 - a;
    if (x < 0.0) a = c_fp64.pi - a;
    return copysign(a, y);
}

}  // namespace qkb
