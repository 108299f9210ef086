// cf_kernels.cu -- batch Heston Fourier pricers on the GPU.
//
// 1. Characteristic-function price (heston_cf_kernel):
// Restates yluoc/Quant-Kernel closed_form_semi_analytical/heston/heston.cpp:7-53
// (little-trap characteristic function) and the P1/P2 integration of
// closed_form_semi_analytical/common/internal_util.h:80-142:
// ceil(steps/64) panels of the 64-point Gauss-Legendre rule on [1e-8, limit],
// two characteristic-function values per node.  The rule's nodes and weights
// are computed on the host (Newton on the Legendre recurrence) and held in
// constant memory.
//
// 2. COS expansion (heston_cos_kernel): yluoc/Quant-Kernel
// fourier_transform_methods/cos_method/cos_method.cpp:30-58 with the
// log-price characteristic function of common/charfn_concepts.h:54-78 and
// the cosine sum of cos_method.h:13-57: n_terms terms on [a, b].
//
// Both read the caller's columns (uploaded in chunks that overlap the pricing
// of earlier chunks), apply the reference's entry checks on the device and sum
// in FP64 over 128 virtual threads, node k on k mod 128, merged in a fixed
// tree: one warp carries all 128 in a large batch, four warps share them in a
// small one, and the sums are the same bits.  Well-conditioned options take
// the bounded functions of fp64_math.cuh and a characteristic function with
// one complex division (HestonFast); the others the general form.
#include "cf_kernels.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>

#include "fp64_math.cuh"
#include "mc_plan.h"
#include "qk_fault.h"

namespace qkb {

namespace {

__constant__ double c_gl_x[32];
__constant__ double c_gl_w[32];

struct Cx {
    double re, im;
};
__device__ __forceinline__ Cx cx(double r, double i) { return Cx{r, i}; }
__device__ __forceinline__ Cx operator+(Cx a, Cx b) { return cx(a.re + b.re, a.im + b.im); }
__device__ __forceinline__ Cx operator-(Cx a, Cx b) { return cx(a.re - b.re, a.im - b.im); }
__device__ __forceinline__ Cx operator*(double s, Cx a) { return cx(s * a.re, s * a.im); }
__device__ __forceinline__ Cx operator/(Cx a, Cx b) {
    // Smith's algorithm (scaled division)
    if (fabs(b.re) >= fabs(b.im)) {
        const double r = b.im / b.re, d = b.re + b.im * r;
        return cx((a.re + a.im * r) / d, (a.im - a.re * r) / d);
    }
    const double r = b.re / b.im, d = b.re * r + b.im;
    return cx((a.re * r + a.im) / d, (a.im * r - a.re) / d);
}
__device__ __forceinline__ Cx cexp_(Cx a) {
    double s, c;
    sincos(a.im, &s, &c);
    const double e = exp(a.re);
    return cx(e * c, e * s);
}
// Principal logarithm.  Near |a| = 1 the real part is 0.5 log1p(x^2 + y^2 - 1)
// with x^2 and y^2 split into exact FMA products: log(hypot(x, y)) would carry
// an absolute error of one ulp of 1 there, which the 1/u factor of the P1/P2
// integrands magnifies at small u.
__device__ __forceinline__ Cx clog_(Cx a) {
    const double ax = fabs(a.re), ay = fabs(a.im);
    const double big = fmax(ax, ay), small = fmin(ax, ay);
    const double hb = big * big;
    double lr;
    if (hb >= 0.5 && hb <= 2.0) {
        const double lb = fma(big, big, -hb);
        const double hs = small * small;
        const double ls = fma(small, small, -hs);
        const double s = hb - 1.0;  // exact for hb in [0.5, 2]
        const double t = s + hs;    // two-sum of s and hs
        const double bp = t - s;
        const double err = (s - (t - bp)) + (hs - bp);
        lr = 0.5 * log1p(t + (err + lb + ls));
    } else {
        lr = log(hypot(a.re, a.im));
    }
    return cx(lr, atan2(a.im, a.re));
}
// Principal square root (branch cut on the negative real axis).  The smaller
// component comes from a division, not from sqrt(|a| - |re|), which cancels
// when |im| << |re|.
__device__ __forceinline__ Cx csqrt_(Cx a) {
    const double m = hypot(a.re, a.im);
    if (m == 0.0) return cx(0.0, a.im);
    if (a.re >= 0.0) {
        const double t = sqrt(0.5 * (m + a.re));
        return cx(t, a.im / (2.0 * t));
    }
    const double t = sqrt(0.5 * (m - a.re));
    return cx(fabs(a.im) / (2.0 * t), copysign(t, a.im));
}

// Complex product and quotient for the characteristic function, with the
// multiply-adds fused explicitly (one rounding per component) and Smith's
// scaled division taking one reciprocal instead of two quotients.
__device__ __forceinline__ Cx fmul(Cx a, Cx b) {
    return cx(fma(a.re, b.re, -(a.im * b.im)), fma(a.re, b.im, a.im * b.re));
}
__device__ __forceinline__ Cx fdiv(Cx a, Cx b) {
    if (fabs(b.re) >= fabs(b.im)) {
        const double r = b.im / b.re, inv = 1.0 / fma(b.im, r, b.re);
        return cx(fma(a.im, r, a.re) * inv, fma(-a.re, r, a.im) * inv);
    }
    const double r = b.re / b.im, inv = 1.0 / fma(b.re, r, b.im);
    return cx(fma(a.re, r, a.im) * inv, fma(a.im, r, -a.re) * inv);
}

struct HestonCf {
    double kappa, theta_k_s2, rho_sigma, sigma2, inv_sigma2, v0, t, drift;
    // heston.cpp:33-44.  Not inlined: the body is large and is called at three
    // places; one copy keeps the kernel inside the instruction cache.
    __device__ __noinline__ Cx operator()(Cx u) const {
        const Cx iu = cx(-u.im, u.re);
        const Cx beta = cx(kappa, 0.0) - rho_sigma * iu;
        const Cx d = csqrt_(fmul(beta, beta) + sigma2 * (iu + fmul(u, u)));
        const Cx bmd = beta - d;
        const Cx g = fdiv(bmd, beta + d);
        const Cx e = cexp_(cx(-d.re * t, -d.im * t));
        const Cx one = cx(1.0, 0.0);
        const Cx one_ge = one - fmul(g, e);
        const Cx C = drift * iu + theta_k_s2 * (t * bmd - 2.0 * clog_(fdiv(one_ge, one - g)));
        const Cx D = fmul(inv_sigma2 * bmd, fdiv(one - e, one_ge));
        return cexp_(C + v0 * D);
    }
};

// The caller's columns of one chunk on the device: kFourierF64 double columns
// (spot, strike, t, r, q, v0, kappa, theta, sigma, rho, limit or width), then
// option_type and steps or terms, each m long.
struct FourierIn {
    double spot, strike, t, r, q, v0, kappa, theta, sigma, rho, limit;
    int32_t option_type, count;
};
__device__ __forceinline__ FourierIn load_columns(const double* __restrict__ in, int32_t m,
                                                  int32_t i) {
    FourierIn o;
    const double* p = in + i;
    const size_t c = (size_t)m;
    o.spot = __ldg(p);
    o.strike = __ldg(p + c);
    o.t = __ldg(p + 2 * c);
    o.r = __ldg(p + 3 * c);
    o.q = __ldg(p + 4 * c);
    o.v0 = __ldg(p + 5 * c);
    o.kappa = __ldg(p + 6 * c);
    o.theta = __ldg(p + 7 * c);
    o.sigma = __ldg(p + 8 * c);
    o.rho = __ldg(p + 9 * c);
    o.limit = __ldg(p + 10 * c);
    const int32_t* q = reinterpret_cast<const int32_t*>(in + kFourierF64 * c) + i;
    o.option_type = __ldg(q);
    o.count = __ldg(q + c);
    return o;
}

__device__ __forceinline__ double nan_() { return __longlong_as_double(0x7FF8000000000000ll); }

__device__ __forceinline__ double intrinsic_(double s, double k, int32_t ot) {
    const double d = ot == 0 ? s - k : k - s;
    return (0.0 < d) ? d : 0.0;
}

// The entry checks both methods share (heston.cpp:10-20, cos_method.cpp:38-46):
// false when they decide the result, which is then in `price`.
__device__ __forceinline__ bool shared_checks(const FourierIn& o, double& price) {
    price = nan_();
    if (!(o.option_type == 0 || o.option_type == 1)) return false;
    if (!isfinite(o.spot) || !isfinite(o.strike) || !isfinite(o.t) || !isfinite(o.r) ||
        !isfinite(o.q) || !isfinite(o.v0) || !isfinite(o.kappa) || !isfinite(o.theta) ||
        !isfinite(o.sigma) || !isfinite(o.rho))
        return false;
    return o.spot > 0.0 && o.strike > 0.0 && o.t >= 0.0 && o.v0 >= 0.0;
}

// ---------------------------------------------------------------------------
// The characteristic function on well-conditioned options.
//
// With iu' = i(u - i) for the share measure (P1), both of a node's values have
// beta = kp - i rho sigma u and d^2 = beta^2 + sigma^2 (u^2 + s i u), with
// (kp, s) = (kappa, 1) for phi(u) and (kappa - rho sigma, -1) for
// phi(u - i) / phi(-i): phi(-i) is exp(log S + (r - q) t) exactly, since d =
// beta there, so the quotient drops the real drift.  Writing P = beta + d, M =
// beta - d, e = exp(-d t), Q = P - M e:
//   (1 - g e)/(1 - g) = Q / (2 d),   M P = -sigma^2 (u^2 + s i u),
//   C = k2 (t M - 2 log(Q / 2d)),    D = -(u^2 + s i u)(1 - e) / Q,
// with k2 = kappa theta / sigma^2: one complex division instead of three.
// Re d^2 = kp^2 + (1 - rho^2) sigma^2 u^2 > 0, so the square root needs one
// half-plane; |d|^2 is the modulus taken for it.  The caller's phase joins the
// exponent, so only exp(Re) and the sine or cosine of Im are taken.
// About 160 FP64 operations a value; the general form with CUDA's functions
// took 400 and as many integer ones.
// ---------------------------------------------------------------------------
struct HestonFast {
    double kp, kp2, c_re, c_im, b_im, sgn, s_sigma2, t, k2, v0, phase;
    __device__ __forceinline__ void operator()(double u, double u2, const Fp64Tables& tab,
                                               double& er, double& ei) const {
        const double re = fma(c_re, u2, kp2), im = c_im * u;
        const double m2 = fma(re, re, im * im);
        const double inv_m = fp64_rsqrt(m2);
        const double h = fma(0.5 * m2, inv_m, 0.5 * re);
        const double yh = fp64_rsqrt(h);
        const double dr = h * yh, di = 0.5 * im * yh;
        const double bi = b_im * u;
        const double pr = kp + dr, pi = bi + di;
        // M = beta - d without the cancellation that k2 t would magnify:
        // kp - dr = (kp^2 - dr^2) / (kp + dr) with dr^2 = Re d^2 + di^2, and
        // bi - di = u (2 rho sigma (kp - dr) - s sigma^2) / (2 dr)
        const double mr = -fma(c_re, u2, di * di) * fp64_rcp(pr);
        const double mi = fma(-2.0 * b_im, mr, -s_sigma2) * (0.5 * yh * u);
        double sn, cs;
        fp64_sincos(di * t, tab, sn, cs);
        const double ex = fp64_exp<false>(-(dr * t), tab);
        const double e_r = ex * cs, e_i = -(ex * sn);
        const double qr = fma(-mr, e_r, fma(mi, e_i, pr));
        const double qi = fma(-mr, e_i, fma(-mi, e_r, pi));
        const double q2 = fma(qr, qr, qi * qi);
        const double log2a = fp64_log(q2 * (0.25 * inv_m), tab);  // 2 log|Q / 2d|
        const double arg = fp64_atan2(fma(qi, dr, -(qr * di)), fma(qr, dr, qi * di), tab);
        const double n1 = 1.0 - e_r, su = sgn * u;
        const double nr = fma(u2, n1, su * e_i), ni = fma(su, n1, -(u2 * e_i));
        const double vi = v0 * fp64_rcp(q2);
        er = fma(k2, fma(t, mr, -log2a), -(fma(nr, qr, ni * qi) * vi));
        ei = fma(k2, fma(t, mi, -2.0 * arg), fma(-vi, fma(ni, qr, -(nr * qi)), phase * u));
        // exp(er) below 1e-304 is as good as zero, and stays in exp's range
        er = __hiloint2double((int32_t)min((uint32_t)__double2hiint(er), 0xC085E000u),
                              __double2loint(er));
    }
};

// Constants of HestonFast, and whether they keep every argument in range over
// (0, u_max]: log-moneyness, rates and times of any market; sigma away from
// the Black-Scholes limit, where 1/sigma^2 magnifies the rounding of M (k2 t
// kappa <= 1e5 leaves 1e-11); kappa > rho sigma, where phi(-i) is as above;
// |d| t inside exp's range.
__device__ __forceinline__ bool fast_constants(const FourierIn& o, double u_max, HestonFast& f2,
                                               HestonFast& f1) {
    const double s2 = o.sigma * o.sigma, rs = o.rho * o.sigma;
    const double kp1 = o.kappa - rs;
    const double k2 = o.kappa * o.theta / s2;
    f2.kp = o.kappa;
    f1.kp = kp1;
    f2.kp2 = o.kappa * o.kappa;
    f1.kp2 = kp1 * kp1;
    f2.c_re = f1.c_re = s2 - rs * rs;
    f2.c_im = s2 - 2.0 * o.kappa * rs;
    f1.c_im = -s2 - 2.0 * kp1 * rs;
    f2.b_im = f1.b_im = -rs;
    f2.sgn = 1.0;
    f1.sgn = -1.0;
    f2.s_sigma2 = s2;
    f1.s_sigma2 = -s2;
    f2.t = f1.t = o.t;
    f2.k2 = f1.k2 = k2;
    f2.v0 = f1.v0 = o.v0;
    const bool ok = o.spot >= 1e-6 && o.spot <= 1e9 && o.strike >= 1e-6 && o.strike <= 1e9 &&
                    o.t >= 1e-6 && o.t <= 100.0 && fabs(o.r) <= 10.0 && fabs(o.q) <= 10.0 &&
                    o.v0 <= 10.0 && o.theta >= 0.0 && o.theta <= 10.0 && o.kappa >= 0.01 &&
                    o.kappa <= 100.0 && o.sigma >= 0.02 && o.sigma <= 10.0 && o.rho >= -0.9999 &&
                    o.rho <= 0.9999 && kp1 >= 0.01 && u_max <= 1e5;
    if (!(ok && k2 * (1.0 + o.t * (o.kappa + 1.0)) <= 1e5)) return false;
    const double uu = u_max * u_max;
    const double d2 = fmax(f2.kp2, f1.kp2) + f2.c_re * uu + fmax(fabs(f2.c_im), fabs(f1.c_im)) * u_max;
    return sqrt(d2) * o.t <= 690.0;
}

// Sums of the virtual threads v = lane (+ 32 j) over WARPS warps: `one(v)` is
// virtual thread v's sums, merged as the 128-leaf tree t += t + 64, t + 32, ...
struct Sums {
    double a, b;
};
__device__ __forceinline__ Sums operator+(Sums x, Sums y) { return Sums{x.a + y.a, x.b + y.b}; }

template <int WARPS, class One>
__device__ __forceinline__ Sums tree_sum(const One& one, Sums* smem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Sums s;
    if constexpr (WARPS == 1) {
        s = one(lane);
        s = s + one(lane + 64);
        Sums r = one(lane + 32);
        r = r + one(lane + 96);
        s = s + r;
    } else {
        s = one(lane + 32 * warp);
        smem[threadIdx.x] = s;
        __syncthreads();
        if (warp == 0)
            s = (smem[lane] + smem[lane + 64]) + (smem[lane + 32] + smem[lane + 96]);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        s = s + Sums{__shfl_down_sync(0xffffffffu, s.a, off), __shfl_down_sync(0xffffffffu, s.b, off)};
    return s;
}

// Virtual thread v's nodes with the general characteristic function.
struct CfGeneral {
    HestonCf cf;
    Cx phi_mi;
    double phi_abs, inv_phi_abs2, lk, width;
    int64_t nodes;
};
__device__ __noinline__ void cf_general_setup(const FourierIn& o, CfGeneral& g) {
    g.cf.kappa = o.kappa;
    g.cf.sigma2 = o.sigma * o.sigma;
    g.cf.inv_sigma2 = 1.0 / g.cf.sigma2;
    g.cf.theta_k_s2 = o.kappa * o.theta * g.cf.inv_sigma2;
    g.cf.rho_sigma = o.rho * o.sigma;
    g.cf.v0 = o.v0;
    g.cf.t = o.t;
    g.cf.drift = log(o.spot) + (o.r - o.q) * o.t;
    g.lk = log(o.strike);
    g.phi_mi = g.cf(cx(0.0, -1.0));
    g.phi_abs = hypot(g.phi_mi.re, g.phi_mi.im);
    g.inv_phi_abs2 = 1.0 / (g.phi_mi.re * g.phi_mi.re + g.phi_mi.im * g.phi_mi.im);
}
__device__ __noinline__ Sums cf_general_nodes(const CfGeneral& g, int v) {
    double s1 = 0.0, s2 = 0.0;
    // 64-bit node counter: panels * 64 and the strided index can pass INT32_MAX
    for (int64_t k = v; k < g.nodes; k += 128) {
        const int64_t p = k >> 6;
        const int32_t j = static_cast<int32_t>((k >> 1) & 31), side = static_cast<int32_t>(k & 1);
        const double pa = 1e-8 + static_cast<double>(p) * g.width;
        const double pb = pa + g.width;
        const double mid = 0.5 * (pa + pb), half = 0.5 * (pb - pa);
        const double u = side == 0 ? mid - half * c_gl_x[j] : mid + half * c_gl_x[j];
        const double wi = c_gl_w[j];
        const double inv_u = 1.0 / u;
        double sn, cs;
        sincos(u * g.lk, &sn, &cs);
        const Cx c2 = g.cf(cx(u, 0.0));
        s2 += half * wi * ((cs * c2.im - sn * c2.re) * inv_u);
        if (g.phi_abs >= 1e-14) {
            const Cx c1 = g.cf(cx(u, -1.0));
            const double n1_re = cs * c1.re + sn * c1.im;
            const double n1_im = cs * c1.im - sn * c1.re;
            const double d_re = n1_im * inv_u, d_im = -n1_re * inv_u;
            s1 += half * wi * ((d_re * g.phi_mi.re + d_im * g.phi_mi.im) * g.inv_phi_abs2);
        }
    }
    return Sums{s1, s2};
}

// Bound by the FP64 pipe.  Three CTAs per SM (162 registers): the two values of
// a node are independent chains, and what the compiler interleaves of them
// hides more latency than more warps do (four, five and six CTAs per SM ran 3,
// 3 and 5% longer; M = beta - d by subtraction 6% shorter, but k2 t magnifies
// its rounding: with the exact M prices are 5.6e-16 from an 80-bit evaluation,
// the general form's 1.0e-15).  65536 options x 1024 nodes end to end 6.6 ->
// 1.77 ms; the general form for every option 3.2-6.2 ms by its parameters.
template <int WARPS>
__global__ void __launch_bounds__(128, 3)
    heston_cf_kernel(const double* __restrict__ in, int32_t m, double* __restrict__ out) {
    __shared__ Fp64Tables tab;
    __shared__ Sums smem[WARPS == 1 ? 1 : 128];
    fp64_load_tables(tab);
    __syncthreads();
    const int32_t i = WARPS == 1 ? (int32_t)(blockIdx.x * 4 + (threadIdx.x >> 5)) : (int32_t)blockIdx.x;
    if (i >= m) return;
    const bool writer = (threadIdx.x & (WARPS == 1 ? 31 : 127)) == 0;
    const FourierIn o = load_columns(in, m, i);
    double price;
    bool simulate = shared_checks(o, price) && o.kappa > 0.0 && o.theta >= 0.0 && o.sigma > 0.0 &&
                    o.rho > -1.0 && o.rho < 1.0;
    if (simulate && o.t <= 1e-12) {
        price = intrinsic_(o.spot, o.strike, o.option_type);
        simulate = false;
    }
    if (simulate && (o.count < 16 || !(o.limit > 1e-6))) {
        // heston.cpp:22-24 compares limit <= 1e-6: a NaN limit integrates to NaN
        simulate = o.count >= 16 && isnan(o.limit);
        price = nan_();
    }
    if (!simulate) {
        if (writer) out[i] = price;
        return;
    }
    const int64_t panels = ((int64_t)o.count + 63) / 64;  // >= 1
    const double width = (o.limit - 1e-8) / static_cast<double>(panels);
    const int64_t nodes = panels * 64;
    HestonFast f2, f1;
    Sums s;
    bool nan_phi = false;
    const double drift = (o.r - o.q) * o.t;
    bool bounded = o.limit >= 1.0 && panels < (1 << 24) && fast_constants(o, o.limit, f2, f1);
    if (bounded) {
        // log phi(-i): below log(1e-14) = -32.24 the price is NaN, near exp's
        // range phi(-i) and the quotient by it overflow.  The bounded route forms
        // neither: both ends are the general form's.
        const double log_phi = fp64_log(o.spot, tab) + drift;
        bounded = log_phi >= -32.2 && log_phi <= 700.0;
    }
    if (bounded) {
        // of log(S/K), not log S - log K: u magnifies the difference's rounding
        f2.phase = f1.phase = log(o.spot / o.strike) + drift;
        const double half = 0.5 * width;
        s = tree_sum<WARPS>(
            [&](int v) {
                const int j = (v >> 1) & 31;
                const double x = (v & 1) == 0 ? -c_gl_x[j] : c_gl_x[j];
                double s1 = 0.0, s2 = 0.0;
                double pd = (double)(v >> 6) + 0.5;  // panel + 1/2
                for (int32_t k = v; k < (int32_t)nodes; k += 128, pd += 2.0) {
                    const double u = fma(half, x, fma(pd, width, 1e-8));
                    const double u2 = u * u, inv_u = fp64_rcp(u);
                    double er, ei, sn, cs;
                    f2(u, u2, tab, er, ei);
                    fp64_sincos(ei, tab, sn, cs);
                    s2 = fma(fp64_exp<false>(er, tab) * sn, inv_u, s2);
                    f1(u, u2, tab, er, ei);
                    fp64_sincos(ei, tab, sn, cs);
                    s1 = fma(fp64_exp<false>(er, tab) * sn, inv_u, s1);
                }
                const double w = half * c_gl_w[j];
                return Sums{s1 * w, s2 * w};
            },
            smem);
    } else {
        CfGeneral g;
        cf_general_setup(o, g);
        g.width = width;
        g.nodes = nodes;
        nan_phi = !(g.phi_abs >= 1e-14);
        s = tree_sum<WARPS>([&](int v) { return cf_general_nodes(g, v); }, smem);
    }
    if (writer) {
        const double kPi = 3.1415926535897932384626433832795;
        double p2 = 0.5 + s.b / kPi;
        double p1 = 0.5 + s.a / kPi;
        p2 = fmin(1.0, fmax(0.0, p2));
        p1 = fmin(1.0, fmax(0.0, p1));
        if (nan_phi || !isfinite(p1) || !isfinite(p2)) {
            price = nan_();
        } else {
            const double call = o.spot * exp(-o.q * o.t) * p1 - o.strike * exp(-o.r * o.t) * p2;
            price = o.option_type == 0 ? call : call - o.spot * exp(-o.q * o.t) + o.strike * exp(-o.r * o.t);
        }
        out[i] = price;
    }
}


// ---------------------------------------------------------------------------
// COS expansion.  Complex arithmetic in the reference's expression order
// (std::complex products and real-complex mixes), so the terms agree with the
// reference's to rounding.
// ---------------------------------------------------------------------------
__device__ __forceinline__ Cx cmul(Cx a, Cx b) {
    return cx(a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re);
}
// real - complex as std::complex does it: (x - re, 0 - im)
__device__ __forceinline__ Cx rsub(double x, Cx a) { return cx(x - a.re, 0.0 - a.im); }
__device__ __forceinline__ Cx scale(Cx a, double s) { return cx(a.re * s, a.im * s); }

struct HestonLogCf {
    double spot_log, r, q, v0, kappa, theta, sigma, rho;
    // charfn_concepts.h:57-77: phi(u, t) of log S_t
    __device__ __noinline__ Cx operator()(Cx u, double t) const {
        const Cx iu = cmul(cx(0.0, 1.0), u);
        const Cx rs_iu = scale(iu, rho * sigma);
        const Cx a = rsub(kappa, rs_iu);
        const Cx b = scale(iu + cmul(u, u), sigma * sigma);
        const Cx d = csqrt_(cmul(a, a) + b);
        const Cx amd = a - d;
        const Cx g = amd / (a + d);
        const Cx edt = cexp_(scale(cx(-d.re, -d.im), t));
        const Cx lg = clog_(rsub(1.0, cmul(g, edt)) / rsub(1.0, g));
        const Cx C = scale(scale(amd, t) - scale(lg, 2.0), kappa * theta / (sigma * sigma));
        const Cx D = cmul(cx(amd.re / (sigma * sigma), amd.im / (sigma * sigma)), rsub(1.0, edt)) /
                     rsub(1.0, cmul(g, edt));
        return cexp_(scale(iu, spot_log) + scale(scale(iu, r - q), t) + C + scale(D, v0));
    }
};

// Virtual thread v's terms with the general characteristic function.
struct CosGeneral {
    HestonLogCf phi;
    double t, a, c, dd, inv, exp_c, exp_d, strike;
    int32_t terms;
};
__device__ __noinline__ double cos_general_terms(const CosGeneral& g, int v) {
    const double kPi = 3.1415926535897932384626433832795;
    double s = 0.0;
    for (int64_t k = v; k < g.terms; k += 128) {  // 64-bit: no wrap
        const double u = static_cast<double>(k) * kPi * g.inv;
        double chi, psi;
        if (k == 0) {
            chi = g.exp_d - g.exp_c;
            psi = g.dd - g.c;
        } else {
            double sd, cd, sc, cc;
            sincos(u * (g.dd - g.a), &sd, &cd);
            sincos(u * (g.c - g.a), &sc, &cc);
            chi = ((cd * g.exp_d - cc * g.exp_c) + u * (sd * g.exp_d - sc * g.exp_c)) / (1.0 + u * u);
            psi = (sd - sc) / u;
        }
        const double u_k = 2.0 * g.inv * (chi - g.strike * psi);
        const Cx f = g.phi(cx(u, 0.0), g.t);
        // Re(phi * exp(-i u a)) = Re(phi * (cos ua, -sin ua))
        double sa, ca;
        sincos(u * g.a, &sa, &ca);
        const double f_k = f.re * ca - f.im * (-sa);
        const double weight = (k == 0) ? 0.5 : 1.0;
        s += weight * f_k * u_k;
    }
    return s;
}

// Eight terms a lane at the default 256: the option's logarithms and
// exponentials, taken once per lane, weigh as much as a term.  Five CTAs per SM
// (65536 options x 256 terms end to end, which the copy of the columns bounds:
// 0.56-0.62 ms by host; three, four and six CTAs 4-7% more; the general form
// packed on the host 3.66; 3.1e-14 from an 80-bit evaluation, before 7.7e-14).
template <int WARPS>
__global__ void __launch_bounds__(128, 5)
    heston_cos_kernel(const double* __restrict__ in, int32_t m, double* __restrict__ out) {
    __shared__ Fp64Tables tab;
    __shared__ Sums smem[WARPS == 1 ? 1 : 128];
    fp64_load_tables(tab);
    __syncthreads();
    const int32_t i = WARPS == 1 ? (int32_t)(blockIdx.x * 4 + (threadIdx.x >> 5)) : (int32_t)blockIdx.x;
    if (i >= m) return;
    const bool writer = (threadIdx.x & (WARPS == 1 ? 31 : 127)) == 0;
    const FourierIn o = load_columns(in, m, i);
    const double kPi = 3.1415926535897932384626433832795;
    double price;
    bool simulate = shared_checks(o, price) && isfinite(o.limit);
    if (simulate && o.t <= 1e-12) {
        price = intrinsic_(o.spot, o.strike, o.option_type);
        simulate = false;
    }
    // cos_method.cpp:47-55: truncation interval from max(v0, theta)
    const double log_spot = log(o.spot);
    const double eff_var = (o.v0 < o.theta) ? o.theta : o.v0;
    const double c1 = log_spot + (o.r - o.q - 0.5 * eff_var) * o.t;
    const double c2 = eff_var * o.t;
    const double span = o.limit * sqrt((c2 < 0.0) ? 0.0 : c2);
    const double a = c1 - span, b = c1 + span;
    if (simulate && (o.count < 8 || o.limit <= 0.0 || !(b > a + 1e-12))) {  // cos_method.h:22
        price = nan_();
        simulate = false;
    }
    if (!simulate) {
        if (writer) out[i] = price;
        return;
    }
    const double lk = log(o.strike);
    const double cm = lk < a ? a : lk;   // std::min(std::max(log K, a), b)
    const double c = b < cm ? b : cm;
    Sums s{0.0, 0.0};
    const bool summed = c < b;
    if (summed) {
        const double inv = 1.0 / (b - a);
        const double exp_d = exp(b), exp_c = exp(c);
        HestonFast f, unused;
        if (o.kappa > 0.0 && o.sigma > 0.0 && isfinite(exp_d) && o.count < (1 << 24) && b - a >= 1e-3 &&
            fast_constants(o, (double)o.count * kPi * inv, f, unused)) {
            // log S + (r - q) t - a and c - a without a's own rounding, which
            // u would magnify
            f.phase = fma(0.5, c2, span);
            const double ca = c == lk ? fma(-(o.r - o.q - 0.5 * eff_var), o.t, log(o.strike / o.spot)) + span
                                      : c - a;
            // sin(u (b - a)) = sin(k pi) = 0 and its cosine +-1: chi and psi
            // need the sine and cosine at c only
            const double pi_inv = kPi * inv;
            s = tree_sum<WARPS>(
                [&](int v) {
                    double sum = 0.0;
                    const double flip = (v & 1) == 0 ? exp_d : -exp_d;
                    for (int32_t k = v; k < o.count; k += 128) {
                        const double u = (double)k * pi_inv, u2 = u * u;
                        double coef;
                        if (k == 0) {
                            coef = 0.5 * ((exp_d - exp_c) - o.strike * (b - c));
                        } else {
                            double sc, cc;
                            fp64_sincos(u * ca, tab, sc, cc);
                            const double v1 = 1.0 + u2;
                            const double r = fp64_rcp(u * v1);  // 1/(1+u^2) = r u, 1/u = r (1+u^2)
                            const double num = fma(-exp_c, fma(u, sc, cc), flip);
                            coef = r * fma(num, u, o.strike * sc * v1);
                        }
                        double er, ei, sn, cs;
                        f(u, u2, tab, er, ei);
                        fp64_sincos(ei, tab, sn, cs);
                        sum = fma(fp64_exp<false>(er, tab) * cs, coef, sum);
                    }
                    return Sums{2.0 * inv * sum, 0.0};
                },
                smem);
        } else {
            CosGeneral g;
            g.phi.spot_log = log_spot;
            g.phi.r = o.r;
            g.phi.q = o.q;
            g.phi.v0 = o.v0;
            g.phi.kappa = o.kappa;
            g.phi.theta = o.theta;
            g.phi.sigma = o.sigma;
            g.phi.rho = o.rho;
            g.t = o.t;
            g.a = a;
            g.c = c;
            g.dd = b;
            g.inv = inv;
            g.exp_c = exp_c;
            g.exp_d = exp_d;
            g.strike = o.strike;
            g.terms = o.count;
            s = tree_sum<WARPS>([&](int v) { return Sums{cos_general_terms(g, v), 0.0}; }, smem);
        }
    }
    if (writer) {
        double call = summed ? exp(-o.r * o.t) * s.a : 0.0;
        call = (0.0 < call) ? call : 0.0;  // std::max(0.0, call): NaN -> 0
        out[i] = o.option_type == 0 ? call
                                    : call - o.spot * exp(-o.q * o.t) + o.strike * exp(-o.r * o.t);
    }
}

// 64-point Gauss-Legendre nodes (the 32 positive ones) and weights.
void gl64(double* x, double* w) {
    const int n = 64;
    for (int i = 0; i < 32; ++i) {
        double z = std::cos(M_PI * (i + 0.75) / (n + 0.5));
        double dp = 0.0;
        for (int it = 0; it < 100; ++it) {
            double p0 = 1.0, p1 = z;
            for (int k = 2; k <= n; ++k) {
                const double pk = ((2.0 * k - 1.0) * z * p1 - (k - 1.0) * p0) / k;
                p0 = p1;
                p1 = pk;
            }
            dp = n * (z * p1 - p0) / (z * z - 1.0);
            const double dz = p1 / dp;
            z -= dz;
            if (std::fabs(dz) < 1e-16) break;
        }
        x[31 - i] = z;
        w[31 - i] = 2.0 / ((1.0 - z * z) * dp * dp);
    }
}

constexpr int kMaxDev = 64;
std::mutex g_cf_mu;
bool g_cf_ready[kMaxDev] = {};

}  // namespace

namespace {

// The Gauss-Legendre table of the current device, uploaded on first use and
// waited for: the kernels run on non-blocking streams, which the default
// stream's copies are not ordered before.
cudaError_t ensure_gl_table() {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDev) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_cf_mu);
    if (!g_cf_ready[dev]) {
        double x[32], w[32];
        gl64(x, w);
        if ((e = cudaMemcpyToSymbol(c_gl_x, x, sizeof x)) != cudaSuccess) return e;
        if ((e = cudaMemcpyToSymbol(c_gl_w, w, sizeof w)) != cudaSuccess) return e;
        if ((e = cudaStreamSynchronize(cudaStreamLegacy)) != cudaSuccess) return e;
        g_cf_ready[dev] = true;
    }
    return cudaSuccess;
}

// From here on one warp takes an option, whose per-option work is then done once
// instead of four times; below, four warps share it, which divides a lone
// quote's chain of nodes by four.  The sums are the same bits.  Where the two
// meet depends on the work an option has; one and four warps, us a call:
//   CF 256 nodes    592: 49.5 51.6   1776: 63.8 72.7   2960: 82.7 85.2   4736: 108 120
//     1024          148: 59.7 47.5    888: 82.8 71.6   2960: 133  134    4736: 188 197
//     2048          148: 84.5 48.6   1184: 111  110    2960: 207  209    8192: 507 515
//   COS 64 terms    592: 45.1 45.2    888: 49.3 57.5   2960: 57.5 68.4   4736: 73.4 92.2
//     256           592: 50.5 50.7   1776: 63.2 63.5   2960: 68.7 76.7   4736: 88.0 98.8
//     512           592: 88.3 57.7   1776: 100  75.6   2960: 108  84.7   8192: 188 178
constexpr int32_t kWarpPerOption = 2960;

cudaError_t launch_fourier(FourierMethod method, const double* d_in, int32_t m, double* d_out,
                           bool warp_per_option, cudaStream_t st) {
    if (cudaError_t e = injected_fault(kFaultLaunch)) return e;
    const unsigned grid = (unsigned)(warp_per_option ? (m + 3) / 4 : m);
    if (method == FourierMethod::kCos) {
        if (warp_per_option)
            heston_cos_kernel<1><<<grid, 128, 0, st>>>(d_in, m, d_out);
        else
            heston_cos_kernel<4><<<grid, 128, 0, st>>>(d_in, m, d_out);
    } else {
        if (warp_per_option)
            heston_cf_kernel<1><<<grid, 128, 0, st>>>(d_in, m, d_out);
        else
            heston_cf_kernel<4><<<grid, 128, 0, st>>>(d_in, m, d_out);
    }
    return cudaGetLastError();
}

// Per-thread, per-device staging for the host-buffer entry points.
struct FourierScratch {
    DevBuf d_in, d_out;
    PinnedBuf h_in, h_out;
    cudaStream_t st[2] = {nullptr, nullptr};
    ~FourierScratch() {
        for (cudaStream_t s : st)
            if (s) {
                cudaStreamSynchronize(s);
                cudaStreamDestroy(s);
            }
        d_in.release();
        d_out.release();
        h_in.release();
        h_out.release();
    }
};

constexpr size_t kFourierRow = kFourierF64 * sizeof(double) + 2 * sizeof(int32_t);

// Options per upload: a chunk's copy into pinned memory (0.75 MB) hides behind
// the pricing of the one before it; two streams let a chunk's last CTAs share
// the chip with the next chunk's first.
constexpr int32_t kFourierChunk = 8192;

}  // namespace

cudaError_t heston_fourier_price_host(FourierMethod method, const FourierColumns& c, int32_t n,
                                      double* out) {
    NvtxRange range("qk.heston_cf");
    if (n <= 0) return cudaSuccess;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    thread_local std::map<int, std::unique_ptr<FourierScratch>> scratch;
    auto& sp = scratch[dev];
    if (!sp) sp.reset(new FourierScratch());
    FourierScratch& s = *sp;
    for (cudaStream_t& st : s.st)
        if (!st && (e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking)) != cudaSuccess) {
            st = nullptr;
            return e;
        }
    const size_t pb = sizeof(double) * static_cast<size_t>(n);
    if ((e = s.d_in.ensure(kFourierRow * static_cast<size_t>(n))) != cudaSuccess) return e;
    if ((e = s.d_out.ensure(pb)) != cudaSuccess) return e;
    if ((e = s.h_in.ensure(kFourierRow * static_cast<size_t>(n))) != cudaSuccess) return e;
    if ((e = s.h_out.ensure(pb)) != cudaSuccess) return e;
    if (method == FourierMethod::kCf && (e = ensure_gl_table()) != cudaSuccess) return e;
    double* d_out = static_cast<double*>(s.d_out.p);
    double* h_out = static_cast<double*>(s.h_out.p);
    int k = 0;
    for (int64_t i0 = 0; i0 < n && e == cudaSuccess; i0 += kFourierChunk, k ^= 1) {
        const int32_t m = (int32_t)std::min<int64_t>(kFourierChunk, n - i0);
        const size_t at = kFourierRow * static_cast<size_t>(i0), bytes = kFourierRow * static_cast<size_t>(m);
        char* h = static_cast<char*>(s.h_in.p) + at;
        char* d = static_cast<char*>(s.d_in.p) + at;
        for (const double* col : c.f64) {
            std::memcpy(h, col + i0, sizeof(double) * static_cast<size_t>(m));
            h += sizeof(double) * static_cast<size_t>(m);
        }
        for (const int32_t* col : {c.option_type, c.count}) {
            std::memcpy(h, col + i0, sizeof(int32_t) * static_cast<size_t>(m));
            h += sizeof(int32_t) * static_cast<size_t>(m);
        }
        cudaStream_t st = s.st[k];
        e = cudaMemcpyAsync(d, static_cast<char*>(s.h_in.p) + at, bytes, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess)
            e = launch_fourier(method, reinterpret_cast<const double*>(d), m, d_out + i0,
                               n >= kWarpPerOption, st);
        if (e == cudaSuccess) e = injected_fault(kFaultCopy);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(h_out + i0, d_out + i0, sizeof(double) * static_cast<size_t>(m),
                                cudaMemcpyDeviceToHost, st);
    }
    // also after an error: nothing of this call is in flight when it returns
    for (cudaStream_t st : s.st) {
        const cudaError_t es = cudaStreamSynchronize(st);
        if (e == cudaSuccess) e = es;
    }
    if (e != cudaSuccess) return e;
    std::memcpy(out, s.h_out.p, pb);
    return cudaSuccess;
}

}  // namespace qkb
