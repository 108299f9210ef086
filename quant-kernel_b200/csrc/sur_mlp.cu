// sur_mlp.cu -- training and inference of the Heston price surrogate.
//
// One optimiser step on a minibatch of B rows (B % 128 == 0) is two launches:
//   mlp_train_kernel  (sur_gemm.cu) gather, forward, head, loss gradient,
//                     backward, and each 128 rows' slab of the weight gradients
//   update_kernel     sums the slabs, the bias and head gradients and the loss in
//                     a fixed order, Adam with cosine-decayed lr, the FP32
//                     master, the bf16 weights and transposed weights the next
//                     step reads; the last block advances the step
// All reductions run in a fixed order: training is deterministic.
#include "sur_mlp.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <numeric>
#include <random>
#include <vector>

#include "mc_device.cuh"
#include "mc_plan.h"
#include "qk_fault.h"
#include "sur_gemm.cuh"

namespace qkb {

namespace {

constexpr int kPredChunk = 65536;
// A chunk's error word before its results, which keep their alignment.
constexpr size_t kOutHead = 256;

#define QK_TRY(x)                                \
    do {                                         \
        cudaError_t e_ = (x);                    \
        if (e_ != cudaSuccess) return e_;        \
    } while (0)

template <typename T>
cudaError_t dalloc(T** p, size_t count) {
    if (*p) cudaFree(*p);
    *p = nullptr;
    return cudaMalloc(reinterpret_cast<void**>(p), sizeof(T) * std::max<size_t>(count, 1));
}

template <typename T>
void dfree(T*& p) {
    if (p) cudaFree(p);
    p = nullptr;
}

// He-normal weights from the Philox/Box-Muller stream (seed, parameter index),
// zero biases, zero layer-1 padding columns, and a zero output layer: the
// untrained model is its base, and the first steps grow the residual from 0.
__global__ void init_params_kernel(float* P, uint64_t seed) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= SurLayout::total) return;
    double z[4];
    normals4_f64(static_cast<uint32_t>(i), 7u, static_cast<uint32_t>(seed), static_cast<uint32_t>(seed >> 32), z);
    const float z0 = static_cast<float>(z[0]);
    float v = 0.0f;
    if (i < SurLayout::b1) {
        const int col = (i - SurLayout::W1) % kSurInPad;
        v = col < kSurIn ? z0 * sqrtf(2.0f / kSurIn) : 0.0f;
    } else if ((i >= SurLayout::W2 && i < SurLayout::b2) || (i >= SurLayout::W3 && i < SurLayout::b3)) {
        v = z0 * sqrtf(2.0f / kSurHid);
    }
    P[i] = v;
}

// The residual's base: the Black-Scholes call / S at the Heston model's mean
// variance over [0, T],
//   vbar = theta + (v0 - theta) (1 - exp(-kappa T)) / (kappa T)
// (the expectation of (1/T) int_0^T v_t dt), from f = (S/K, T, r, q, v0,
// kappa, theta, ...).  The host and the device evaluate the same FP64
// expression with their own exp/log/erfc; rounded to FP32 the two agree.
__host__ __device__ inline double sur_base(const double* f) {
    const double m = f[0], T = f[1], r = f[2], q = f[3], v0 = f[4], kappa = f[5], theta = f[6];
    const double x = kappa * T;
    const double w = (x > 1e-12) ? -expm1(-x) / x : 1.0;
    double vbar = theta + (v0 - theta) * w;
    if (!(vbar > 0.0)) vbar = 0.0;
    const double sd = sqrt(vbar * T);
    const double dq = exp(-q * T);
    const double dk = exp(-r * T) / m;
    if (!(sd > 1e-12)) {  // no variance left: the discounted forward payoff
        const double fwd = dq - dk;
        return fwd > 0.0 ? fwd : 0.0;
    }
    const double inv_sqrt2 = 0.70710678118654752440;
    const double d1 = (log(m) + (r - q) * T) / sd + 0.5 * sd;
    return dq * (0.5 * erfc(-d1 * inv_sqrt2)) - dk * (0.5 * erfc(-(d1 - sd) * inv_sqrt2));
}

// The normalised coordinate of feature value x in [lo, hi], as bf16 bits.
__host__ __device__ inline unsigned short sur_norm_bits(double x, double lo, double hi) {
    const double u = hi > lo ? 2.0 * (x - lo) / (hi - lo) - 1.0 : 0.0;
    return __bfloat16_as_ushort(__float2bfloat16_rn(static_cast<float>(u)));
}

// Device features: one thread per row computes its nine normalised values
// and base; the block then writes its 256 rows of 128 bytes as consecutive
// 16-byte chunks (columns 9..63 are zero).
constexpr int kFeatRows = 256;
__global__ void __launch_bounds__(kFeatRows)
features_kernel(const double* __restrict__ f, int64_t n, SurBox box, int32_t kind,
                __nv_bfloat16* __restrict__ rows, float* __restrict__ base) {
    __shared__ uint4 stage[kFeatRows][2];
    const int t = threadIdx.x;
    const int64_t row0 = static_cast<int64_t>(blockIdx.x) * kFeatRows;
    const int64_t i = row0 + t;
    unsigned short b[16] = {};
    if (i < n) {
        double x[kSurIn];
#pragma unroll
        for (int c = 0; c < kSurIn; ++c) x[c] = f[i * kSurIn + c];
#pragma unroll
        for (int c = 0; c < kSurIn; ++c) b[c] = sur_norm_bits(x[c], box.lo[c], box.hi[c]);
        if (base) base[i] = kind == kSurBaseBsmMeanVar ? static_cast<float>(sur_base(x)) : 0.0f;
    }
    uint4 c0, c1;
    c0.x = b[0] | (static_cast<uint32_t>(b[1]) << 16);
    c0.y = b[2] | (static_cast<uint32_t>(b[3]) << 16);
    c0.z = b[4] | (static_cast<uint32_t>(b[5]) << 16);
    c0.w = b[6] | (static_cast<uint32_t>(b[7]) << 16);
    c1.x = b[8];
    c1.y = c1.z = c1.w = 0u;
    stage[t][0] = c0;
    stage[t][1] = c1;
    __syncthreads();
    uint4* out = reinterpret_cast<uint4*>(rows);
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int k = 0; k < 8; ++k) {  // 256 rows x 8 chunks, 8 per thread
        const int idx = k * kFeatRows + t;
        const int r = idx >> 3, c = idx & 7;
        const int64_t row = row0 + r;
        if (row < n) out[row * 8 + c] = c < 2 ? stage[r][c] : zero;
    }
}

// The host pricing call, read straight from its pinned slot: ten double
// columns (spot, strike, t, r, q, v0, kappa, theta, sigma, rho), then
// option_type, n each, coalesced.  One thread per option decides its route --
// 0: the network, 1: Monte Carlo (outside the box; NaN until priced), 2: entry
// checks of heston_monte_carlo.cpp:18-26 -- and writes the network's row (its
// first 32 bytes, all that the fused kernel reads) and base; other routes get
// a row of zeros.  fix holds what quote_price_kernel needs: (spot, S e^-qT, K
// e^-rT) for a put, (spot, 0, 0) for a call, (0, -result, 0) for routes 1, 2,
// whose price the network's output does not enter, whatever it is.
// Bound by the copy into the slot and PCIe (84 bytes an option): on the host,
// the checks, bf16 rows and base took 180 ns an option on one thread (20,000
// quotes 3.70 ms a call, now 0.21; 200,000 34 ms, now 1.27).
__global__ void __launch_bounds__(kFeatRows)
quote_features_kernel(const double* __restrict__ in, int64_t n, SurBox box, int32_t kind,
                      __nv_bfloat16* __restrict__ rows, float* __restrict__ base,
                      double* __restrict__ fix, int32_t* __restrict__ out_route) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * kFeatRows + threadIdx.x;
    if (i >= n) return;
    double c[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) c[k] = in[k * n + i];
    const int32_t ot = reinterpret_cast<const int32_t*>(in + 10 * n)[i];
    const double spot = c[0], strike = c[1], t = c[2];
    int32_t to = 2;
    unsigned short b[16] = {};
    float base_i = 0.0f;
    double f0 = 0.0, f1 = 0.0, f2 = 0.0;
    if (!(ot == 0 || ot == 1) || spot <= 0.0 || strike <= 0.0 || t < 0.0 || c[5] < 0.0 ||
        c[6] < 0.0 || c[7] < 0.0 || c[8] < 0.0 || c[9] < -1.0 || c[9] > 1.0) {
        f1 = __longlong_as_double(0x7FF8000000000000ll);
    } else if (t <= 1e-12) {
        const double d = ot == 0 ? spot - strike : strike - spot;
        f1 = (0.0 < d) ? -d : 0.0;
    } else {
        const double x[kSurIn] = {spot / strike, t, c[3], c[4], c[5], c[6], c[7], c[8], c[9]};
        bool inside = true;
#pragma unroll
        for (int k = 0; k < kSurIn; ++k) inside = inside && x[k] >= box.lo[k] && x[k] <= box.hi[k];
        to = inside ? 0 : 1;
        if (!inside) {
            f1 = __longlong_as_double(0x7FF8000000000000ll);
        } else {
#pragma unroll
            for (int k = 0; k < kSurIn; ++k) b[k] = sur_norm_bits(x[k], box.lo[k], box.hi[k]);
            if (kind == kSurBaseBsmMeanVar) base_i = static_cast<float>(sur_base(x));
            f0 = spot;
            if (ot == 1) {
                f1 = spot * exp(-c[4] * t);
                f2 = strike * exp(-c[3] * t);
            }
        }
    }
    out_route[i] = to;
    base[i] = base_i;
    fix[i] = f0;
    fix[n + i] = f1;
    fix[2 * n + i] = f2;
    uint4* row = reinterpret_cast<uint4*>(rows + i * kSurInPad);
    row[0] = make_uint4(b[0] | (static_cast<uint32_t>(b[1]) << 16), b[2] | (static_cast<uint32_t>(b[3]) << 16),
                        b[4] | (static_cast<uint32_t>(b[5]) << 16), b[6] | (static_cast<uint32_t>(b[7]) << 16));
    row[1] = make_uint4(b[8], 0u, 0u, 0u);
}

// The call from price / S, puts by put-call parity, straight into the pinned
// slot (coalesced), with the network's error word.
__global__ void __launch_bounds__(kFeatRows)
quote_price_kernel(const double* __restrict__ fix, int64_t n, const float* __restrict__ y,
                   double* __restrict__ out, const int* __restrict__ err, int* __restrict__ out_err) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * kFeatRows + threadIdx.x;
    if (i >= n) return;
    if (i == 0) *out_err = *err;
    const double spot = fix[i], network = static_cast<double>(y[i]);
    const double call = spot != 0.0 ? spot * network : 0.0;  // 0: not the network's
    out[i] = call - fix[n + i] + fix[2 * n + i];
}

// ----------------------------------------------------------------------------
// The update.  Block kinds, by blockIdx.x:
//   [0, 128)     8 columns of db1, db2, db3 (sums of dZ over the batch) or dw4
//                (sum of h3 dy), two a warp: 32 residue chains a column (lane =
//                row mod 32, in row order), merged in a fixed shuffle tree
//   128          db4 = sum dy and the loss (256 strided chains, a tree)
//   [129, ...)   four weights a thread: their slabs in order
// each followed by Adam on what it summed.  Bound by reading the slabs and dZ
// back from L2 (50 MB at batch 8192).  Every array is read in the layout the
// training pass writes (16-byte chunks, rows contiguous).
// ----------------------------------------------------------------------------
constexpr int kUpdThreads = 128;
constexpr int kBiasBlocks = 128;
constexpr int kWeightDepth = 32;
constexpr size_t kUpdSmem = sizeof(uint4) * kWeightDepth * kUpdThreads;
constexpr int kW1Quads = kSurHid * 16 / 4, kWQuads = kSurHid * kSurHid / 4;

struct UpdateArgs {
    const uint4* dz[3];              // dZ1, dZ2, dZ3
    const uint4* h3;
    const float *y, *target, *dy;    // [B]
    const float4 *dw1, *dw2, *dw3;   // slabs
    int batch;
    float *P, *M, *V, *G;            // flat layout; G is written without update only
    __nv_bfloat16 *W1b, *W2b, *W3b, *W2Tb, *W3Tb;
    float* loss_hist;
    int loss_cap;
    int update;                      // 0: gradients only
    SurState* st;
    unsigned* blocks_done;
};

// add(k, value) for k = 0 .. n - 1 in order, value k the 16 bytes at addr(k),
// through a ring of DEPTH asynchronous copies per thread (slot k of thread t at
// buf[k % DEPTH][t] of T threads).  As register loads the compiler kept four
// in flight and the chain waited on L2 at every fourth addition.
template <int T, int DEPTH, class Addr, class Add>
__device__ __forceinline__ void stream_sum(uint4* buf, int t, int n, const Addr& addr, const Add& add) {
    constexpr int kGroup = 16, kAhead = DEPTH / kGroup;
    auto issue = [&](int g) {
#pragma unroll
        for (int i = 0; i < kGroup; ++i) {
            const int k = g * kGroup + i;
            if (k < n) {
                const uint32_t dst =
                    static_cast<uint32_t>(__cvta_generic_to_shared(buf + (k % DEPTH) * T + t));
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(addr(k)) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int g = 0; g < kAhead; ++g) issue(g);
    for (int g = 0; g * kGroup < n; ++g) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kAhead - 1) : "memory");
#pragma unroll
        for (int i = 0; i < kGroup; ++i) {
            const int k = g * kGroup + i;
            if (k < n) add(k, buf[(k % DEPTH) * T + t]);
        }
        issue(g + kAhead);
    }
}

// Adam with this step's constants.
struct Adam {
    float lr, b1, b2, eps, c1, c2;
    __device__ __forceinline__ explicit Adam(const SurState& st) {
        const int t = st.step + 1;
        const float span = static_cast<float>(max(st.total_steps - st.step_begin, 1));
        const float prog = fminf(static_cast<float>(st.step - st.step_begin) / span, 1.0f);
        lr = st.lr0 * 0.5f * (1.0f + cosf(3.14159265358979f * prog));
        b1 = st.beta1;
        b2 = st.beta2;
        eps = st.eps;
        c1 = 1.0f - powf(st.beta1, static_cast<float>(t));
        c2 = 1.0f - powf(st.beta2, static_cast<float>(t));
    }
    __device__ __forceinline__ void operator()(float g, float& p, float& m, float& v) const {
        m = b1 * m + (1.0f - b1) * g;
        v = b2 * v + (1.0f - b2) * g * g;
        const float mh = m / c1;
        const float vh = v / c2;
        p -= lr * mh / (sqrtf(vh) + eps);
    }
};

// `failed`: the training pass did not complete, its sums are not gradients (read
// at the kernel's start, ahead of the sums: at the update it cost 0.4 us a step).
__device__ __forceinline__ void update_one(const UpdateArgs& a, bool failed, int idx, float g) {
    if (!a.update) {
        a.G[idx] = g;
        return;
    }
    if (failed) return;
    float p = a.P[idx], m = a.M[idx], v = a.V[idx];
    Adam(*a.st)(g, p, m, v);
    a.P[idx] = p;
    a.M[idx] = m;
    a.V[idx] = v;
}

__device__ __forceinline__ void update_columns(const UpdateArgs& a, bool failed, int block) {
    const int lane = threadIdx.x & 31, pair = threadIdx.x >> 5;
    const int which = block >> 5, chunk = block & 31;
    const uint32_t* x = reinterpret_cast<const uint32_t*>((which < 3 ? a.dz[which] : a.h3) + chunk * 128 + lane) + pair;
    const float* w = which < 3 ? nullptr : a.dy + lane;
    const int n = a.batch / 32;
    // row 32 m + lane is row 32 (m % 4) + lane of tile m / 4
    auto at = [&](int m) { return x + (static_cast<size_t>(m >> 2) * 32 * 128 + (m & 3) * 32) * 4; };
    float s0 = 0.0f, s1 = 0.0f;
    auto add = [&](uint32_t u, float wv) {
        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u));
        s0 = fmaf(f.x, wv, s0);
        s1 = fmaf(f.y, wv, s1);
    };
    // 32 loads ahead of the additions (n is a multiple of 4)
    int m = 0;
    for (; m + 32 <= n; m += 32) {
        uint32_t u[32];
#pragma unroll
        for (int k = 0; k < 32; ++k) u[k] = __ldg(at(m + k));
        if (w) {
            float wv[32];
#pragma unroll
            for (int k = 0; k < 32; ++k) wv[k] = __ldg(w + 32 * (m + k));
#pragma unroll
            for (int k = 0; k < 32; ++k) add(u[k], wv[k]);
        } else {
#pragma unroll
            for (int k = 0; k < 32; ++k) add(u[k], 1.0f);
        }
    }
    for (; m < n; m += 4) {
        uint32_t u[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) u[k] = __ldg(at(m + k));
#pragma unroll
        for (int k = 0; k < 4; ++k) add(u[k], w ? __ldg(w + 32 * (m + k)) : 1.0f);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        s0 += __shfl_down_sync(0xffffffffu, s0, off);
        s1 += __shfl_down_sync(0xffffffffu, s1, off);
    }
    s1 = __shfl_sync(0xffffffffu, s1, 0);
    if (lane < 2) {
        const int off = which == 0 ? SurLayout::b1 : which == 1 ? SurLayout::b2
                      : which == 2 ? SurLayout::b3 : SurLayout::w4;
        update_one(a, failed, off + chunk * 8 + pair * 2 + lane, lane == 0 ? s0 : s1);
    }
}

__device__ __forceinline__ void update_loss(const UpdateArgs& a, bool failed, float* s1, float* s2) {
    // chains t and t + 128 of 256
    const int t = threadIdx.x;
    float d1[2] = {}, d2[2] = {};
#pragma unroll 8
    for (int i = t; i < a.batch; i += 256) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int k = i + h * 128;
            if (k < a.batch) {
                d1[h] += a.dy[k];
                const float d = a.y[k] - a.target[k];
                d2[h] = fmaf(d, d, d2[h]);
            }
        }
    }
    s1[t] = d1[0];
    s2[t] = d2[0];
    s1[t + 128] = d1[1];
    s2[t + 128] = d2[1];
    __syncthreads();
    for (int off = 128; off > 0; off >>= 1) {
        if (t < off) {
            s1[t] += s1[t + off];
            s2[t] += s2[t + off];
        }
        __syncthreads();
    }
    if (t == 0) {
        const int k = a.st->step;
        if (k >= 0 && k < a.loss_cap) a.loss_hist[k] = s2[0] / static_cast<float>(a.batch);
        update_one(a, failed, SurLayout::b4, s1[0]);
    }
}

__device__ __forceinline__ void update_weights(const UpdateArgs& a, bool failed, int e, uint4* ring) {
    if (e >= kW1Quads + 2 * kWQuads) return;
    // W1's slabs hold the first 16 columns; the padding's gradient is zero and
    // leaves it zero
    const int which = e < kW1Quads ? 0 : (e < kW1Quads + kWQuads ? 1 : 2);
    const int local = which == 0 ? e : (which == 1 ? e - kW1Quads : e - kW1Quads - kWQuads);
    const float4* slab = (which == 0 ? a.dw1 : (which == 1 ? a.dw2 : a.dw3)) + local;
    const size_t stride = which == 0 ? kW1Quads : kWQuads;
    float4 g = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    stream_sum<kUpdThreads, kWeightDepth>(
        ring, threadIdx.x, a.batch / 128, [&](int k) { return slab + k * stride; },
        [&](int, const uint4& v) {
            g.x += __uint_as_float(v.x);
            g.y += __uint_as_float(v.y);
            g.z += __uint_as_float(v.z);
            g.w += __uint_as_float(v.w);
        });
    // [half][chunk of 4 columns][row of 128]
    const int half = local / (which == 0 ? 4 * 128 : 64 * 128);
    const int row = half * 128 + (local & 127), c = ((local >> 7) & (which == 0 ? 3 : 63)) * 4;
    const int at = row * (which == 0 ? kSurInPad : kSurHid) + c;
    const int idx = (which == 0 ? SurLayout::W1 : which == 1 ? SurLayout::W2 : SurLayout::W3) + at;
    if (!a.update) {
        *reinterpret_cast<float4*>(a.G + idx) = g;
        return;
    }
    if (failed) return;
    float4 p = *reinterpret_cast<float4*>(a.P + idx);
    float4 m = *reinterpret_cast<float4*>(a.M + idx);
    float4 v = *reinterpret_cast<float4*>(a.V + idx);
    const Adam adam(*a.st);
    adam(g.x, p.x, m.x, v.x);
    adam(g.y, p.y, m.y, v.y);
    adam(g.z, p.z, m.z, v.z);
    adam(g.w, p.w, m.w, v.w);
    *reinterpret_cast<float4*>(a.P + idx) = p;
    *reinterpret_cast<float4*>(a.M + idx) = m;
    *reinterpret_cast<float4*>(a.V + idx) = v;
    __nv_bfloat162 b[2] = {__floats2bfloat162_rn(p.x, p.y), __floats2bfloat162_rn(p.z, p.w)};
    __nv_bfloat16* wb = which == 0 ? a.W1b : which == 1 ? a.W2b : a.W3b;
    *reinterpret_cast<uint2*>(wb + at) = *reinterpret_cast<uint2*>(b);
    if (which != 0) {
        __nv_bfloat16* wt = (which == 1 ? a.W2Tb : a.W3Tb) + c * kSurHid + row;  // rows contiguous in a warp
        wt[0] = b[0].x;
        wt[kSurHid] = b[0].y;
        wt[2 * kSurHid] = b[1].x;
        wt[3 * kSurHid] = b[1].y;
    }
}

__global__ void __launch_bounds__(kUpdThreads) update_kernel(const UpdateArgs a) {
    extern __shared__ uint4 ring[];
    const int b = blockIdx.x;
    // what the training pass wrote is read from here on
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    const bool failed = a.st->err != 0;
    if (b < kBiasBlocks) {
        update_columns(a, failed, b);
    } else if (b == kBiasBlocks) {
        update_loss(a, failed, reinterpret_cast<float*>(ring), reinterpret_cast<float*>(ring) + 256);
    } else {
        update_weights(a, failed, (b - kBiasBlocks - 1) * kUpdThreads + threadIdx.x, ring);
    }
    if (!a.update) return;
    // every block has read the step; the last one advances it
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(a.blocks_done, 1u) == gridDim.x - 1) {
            *a.blocks_done = 0u;
            if (!failed) a.st->step += 1;
        }
    }
}

// bf16 weights and transposes from the FP32 master (after init and loads).
__global__ void refresh_kernel(const float* __restrict__ P, __nv_bfloat16* W1b, __nv_bfloat16* W2b,
                               __nv_bfloat16* W3b, __nv_bfloat16* W2Tb, __nv_bfloat16* W3Tb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kSurHid * kSurInPad) W1b[i] = __float2bfloat16_rn(P[SurLayout::W1 + i]);
    if (i < kSurHid * kSurHid) {
        const int r = i >> 8, c = i & 255;
        const __nv_bfloat16 w2 = __float2bfloat16_rn(P[SurLayout::W2 + i]);
        const __nv_bfloat16 w3 = __float2bfloat16_rn(P[SurLayout::W3 + i]);
        W2b[i] = w2;
        W3b[i] = w3;
        W2Tb[c * kSurHid + r] = w2;
        W3Tb[c * kSurHid + r] = w3;
    }
}

// Host memory to the device, after the default stream's earlier work (a
// caller's inference there) and done when it returns: cudaMemcpy alone returns
// when the source has been read, and its transfer is not ordered before the
// kernels of a non-blocking stream -- they met half of the parameters before it.
cudaError_t put(void* dst, const void* src, size_t bytes) {
    QK_TRY(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice));
    return cudaStreamSynchronize(cudaStreamLegacy);
}

bool tmap(CUtensorMap* m, const void* base, int64_t rows, int64_t cols, int box_rows) {
    return make_tmap_bf16(m, base, static_cast<uint64_t>(rows), static_cast<uint64_t>(cols),
                          static_cast<uint32_t>(box_rows));
}

struct DeviceGuard {
    int prev = -1;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (dev >= 0 && prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
    }
};

}  // namespace

struct SurModel::StepLaunch {
    TrainMaps maps;
    TrainArgs train;
    UpdateArgs update;
};

// ----------------------------------------------------------------------------
SurModel::~SurModel() {
    if (device_ < 0) return;
    DeviceGuard g(device_);
    float* fl[] = {P_, M_, V_, G_, Tall_, Tb_, y_, dy_, dW1p_, dW2p_, dW3p_, loss_hist_, Pbase_};
    for (float* p : fl)
        if (p) cudaFree(p);
    __nv_bfloat16* bl[] = {W1b_, W2b_, W3b_, W2Tb_, W3Tb_, Xall_, Z1_, H1_, Z2_, H3_, dZ3_, dZ2_, dZ1_,
                           PX_, PH1_, PH2_};
    for (__nv_bfloat16* p : bl)
        if (p) cudaFree(p);
    if (Perr_) cudaFree(Perr_);
    if (perm_) cudaFree(perm_);
    if (state_) cudaFree(state_);
    if (blocks_done_) cudaFree(blocks_done_);
    if (d_in_) cudaFree(d_in_);
    if (uploaded_) cudaEventDestroy(uploaded_);
    if (stream_) cudaStreamDestroy(stream_);
}

cudaError_t SurModel::init(uint64_t seed, const SurBox& box) {
    QK_TRY(cudaGetDevice(&device_));
    box_ = box;
    QK_TRY(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    QK_TRY(cudaEventCreateWithFlags(&uploaded_, cudaEventDisableTiming));
    QK_TRY(dalloc(&P_, SurLayout::total));
    QK_TRY(dalloc(&M_, SurLayout::total));
    QK_TRY(dalloc(&V_, SurLayout::total));
    QK_TRY(dalloc(&G_, SurLayout::total));
    QK_TRY(dalloc(&W1b_, kSurHid * kSurInPad));
    QK_TRY(dalloc(&W2b_, kSurHid * kSurHid));
    QK_TRY(dalloc(&W3b_, kSurHid * kSurHid));
    QK_TRY(dalloc(&W2Tb_, kSurHid * kSurHid));
    QK_TRY(dalloc(&W3Tb_, kSurHid * kSurHid));
    QK_TRY(dalloc(&state_, 1));
    QK_TRY(dalloc(&blocks_done_, 1));
    QK_TRY(cudaMemsetAsync(blocks_done_, 0, sizeof(unsigned), stream_));
    SurState s{};
    s.beta1 = 0.9f;
    s.beta2 = 0.999f;
    s.eps = 1e-8f;
    s.lr0 = 1e-3f;
    s.steps_per_epoch = 1;
    s.total_steps = 1;
    QK_TRY(cudaMemcpyAsync(state_, &s, sizeof s, cudaMemcpyHostToDevice, stream_));
    init_params_kernel<<<(SurLayout::total + 255) / 256, 256, 0, stream_>>>(P_, seed);
    QK_TRY(cudaGetLastError());
    QK_TRY(cudaMemsetAsync(M_, 0, sizeof(float) * SurLayout::total, stream_));
    QK_TRY(cudaMemsetAsync(V_, 0, sizeof(float) * SurLayout::total, stream_));
    QK_TRY(refresh_bf16(stream_));
    return cudaStreamSynchronize(stream_);
}

void SurModel::normalise(const double* f, int64_t n, __nv_bfloat16* out) const {
    for (int64_t i = 0; i < n; ++i) {
        __nv_bfloat16* row = out + i * kSurInPad;
        for (int c = 0; c < kSurInPad; ++c) row[c] = __float2bfloat16_rn(0.0f);
        for (int c = 0; c < kSurIn; ++c)
            row[c] = __ushort_as_bfloat16(sur_norm_bits(f[i * kSurIn + c], box_.lo[c], box_.hi[c]));
    }
}

void SurModel::base_host(const double* f, int64_t n, float* out) const {
    for (int64_t i = 0; i < n; ++i)
        out[i] = base_kind_ == kSurBaseBsmMeanVar ? static_cast<float>(sur_base(f + i * kSurIn)) : 0.0f;
}

cudaError_t SurModel::features_device(const double* f, int64_t n, __nv_bfloat16* rows, float* base,
                                      cudaStream_t st) {
    DeviceGuard g(device_);
    if (n <= 0 || (reinterpret_cast<uintptr_t>(rows) & 15u) != 0 ||
        (reinterpret_cast<uintptr_t>(f) & 7u) != 0 || (reinterpret_cast<uintptr_t>(base) & 3u) != 0)
        return cudaErrorInvalidValue;
    const int64_t blocks = (n + kFeatRows - 1) / kFeatRows;
    if (blocks > 0x7fffffff) return cudaErrorInvalidValue;
    features_kernel<<<static_cast<unsigned>(blocks), kFeatRows, 0, st ? st : stream_>>>(
        f, n, box_, base_kind_, rows, base);
    return cudaGetLastError();
}

cudaError_t SurModel::refresh_bf16(cudaStream_t st) {
    refresh_kernel<<<kSurHid * kSurHid / 256, 256, 0, st>>>(P_, W1b_, W2b_, W3b_, W2Tb_, W3Tb_);
    return cudaGetLastError();
}

cudaError_t SurModel::set_dataset(const double* features, const double* target, int64_t n) {
    DeviceGuard g(device_);
    std::vector<__nv_bfloat16> rows(static_cast<size_t>(n) * kSurInPad);
    normalise(features, n, rows.data());
    // the network learns target - base
    std::vector<float> t(static_cast<size_t>(n));
    for (int64_t i = 0; i < n; ++i) {
        const double b = base_kind_ == kSurBaseBsmMeanVar ? sur_base(features + i * kSurIn) : 0.0;
        t[i] = static_cast<float>(target[i] - b);
    }
    QK_TRY(dalloc(&Xall_, static_cast<size_t>(n) * kSurInPad));
    QK_TRY(dalloc(&Tall_, static_cast<size_t>(n)));
    QK_TRY(dalloc(&perm_, static_cast<size_t>(n)));
    QK_TRY(put(Xall_, rows.data(), rows.size() * sizeof(__nv_bfloat16)));
    QK_TRY(put(Tall_, t.data(), t.size() * sizeof(float)));
    std::vector<int32_t> id(static_cast<size_t>(n));
    std::iota(id.begin(), id.end(), 0);
    QK_TRY(put(perm_, id.data(), id.size() * sizeof(int32_t)));
    n_data_ = n;
    return cudaSuccess;
}

cudaError_t SurModel::ensure_batch_buffers(int B) {
    if (B == batch_) return cudaSuccess;
    batch_ = 0;
    const size_t BH = static_cast<size_t>(B) * kSurHid;
    const int S = B / 128;
    __nv_bfloat16** act[] = {&Z1_, &H1_, &Z2_, &H3_, &dZ3_, &dZ2_, &dZ1_};
    for (auto p : act) QK_TRY(dalloc(p, BH));
    QK_TRY(dalloc(&Tb_, B));
    QK_TRY(dalloc(&y_, B));
    QK_TRY(dalloc(&dy_, B));
    QK_TRY(dalloc(&dW1p_, static_cast<size_t>(S) * kSurHid * 16));
    QK_TRY(dalloc(&dW2p_, static_cast<size_t>(S) * kSurHid * kSurHid));
    QK_TRY(dalloc(&dW3p_, static_cast<size_t>(S) * kSurHid * kSurHid));
    batch_ = B;
    return cudaSuccess;
}

// What every step of a call launches: the step's kernels read the step
// counter and the schedule from state_.
cudaError_t SurModel::prepare_steps(bool update, StepLaunch* s) {
    TrainMaps& m = s->maps;
    if (!(make_tmap_bf16_k16(&m.w1, W1b_, kSurHid, kSurInPad, 256) &&
          tmap(&m.w2, W2b_, kSurHid, kSurHid, 256) && tmap(&m.w3, W3b_, kSurHid, kSurHid, 256) &&
          tmap(&m.w3t, W3Tb_, kSurHid, kSurHid, 256) && tmap(&m.w2t, W2Tb_, kSurHid, kSurHid, 256)))
        return cudaErrorInvalidValue;
    TrainArgs& t = s->train;
    t = TrainArgs{};
    t.xall = Xall_;
    t.x_stride = kSurInPad;
    t.tall = Tall_;
    t.perm = perm_;
    t.step = &state_->step;
    t.steps_per_epoch = &state_->steps_per_epoch;
    t.batch = batch_;
    t.loss_scale = 2.0f / static_cast<float>(batch_);
    t.b1 = P_ + SurLayout::b1;
    t.b2 = P_ + SurLayout::b2;
    t.b3 = P_ + SurLayout::b3;
    t.w4 = P_ + SurLayout::w4;
    t.b4 = P_ + SurLayout::b4;
    t.z1 = reinterpret_cast<uint4*>(Z1_);
    t.z2 = reinterpret_cast<uint4*>(Z2_);
    t.h1 = reinterpret_cast<uint4*>(H1_);
    t.h3 = reinterpret_cast<uint4*>(H3_);
    t.dz3 = reinterpret_cast<uint4*>(dZ3_);
    t.dz2 = reinterpret_cast<uint4*>(dZ2_);
    t.dz1 = reinterpret_cast<uint4*>(dZ1_);
    t.y_out = y_;
    t.dy_out = dy_;
    t.target_out = Tb_;
    t.dw1 = reinterpret_cast<float4*>(dW1p_);
    t.dw2 = reinterpret_cast<float4*>(dW2p_);
    t.dw3 = reinterpret_cast<float4*>(dW3p_);
    t.err = &state_->err;
    UpdateArgs& u = s->update;
    u = UpdateArgs{};
    u.dz[0] = reinterpret_cast<const uint4*>(dZ1_);
    u.dz[1] = reinterpret_cast<const uint4*>(dZ2_);
    u.dz[2] = reinterpret_cast<const uint4*>(dZ3_);
    u.h3 = reinterpret_cast<const uint4*>(H3_);
    u.y = y_;
    u.target = Tb_;
    u.dy = dy_;
    u.dw1 = reinterpret_cast<const float4*>(dW1p_);
    u.dw2 = reinterpret_cast<const float4*>(dW2p_);
    u.dw3 = reinterpret_cast<const float4*>(dW3p_);
    u.batch = batch_;
    u.P = P_;
    u.M = M_;
    u.V = V_;
    u.G = G_;
    u.W1b = W1b_;
    u.W2b = W2b_;
    u.W3b = W3b_;
    u.W2Tb = W2Tb_;
    u.W3Tb = W3Tb_;
    u.loss_hist = loss_hist_;
    u.loss_cap = loss_cap_;
    u.update = update ? 1 : 0;
    u.st = state_;
    u.blocks_done = blocks_done_;
    return cudaSuccess;
}

cudaError_t SurModel::run_step(const StepLaunch& s, cudaStream_t st) {
    static DeviceOnce once;
    QK_TRY(allow_shared(once, update_kernel, kUpdSmem));
    QK_TRY(launch_mlp_train(s.maps, s.train, st));
    constexpr int kQuads = kW1Quads + 2 * kWQuads;
    return launch_dependent(update_kernel, kBiasBlocks + 1 + (kQuads + kUpdThreads - 1) / kUpdThreads, kUpdThreads,
                            kUpdSmem, st, s.update);
}

cudaError_t SurModel::train(int epochs, int batch, float lr0, uint64_t shuffle_seed,
                            float* out_loss_last, float* out_epoch_loss) {
    DeviceGuard g(device_);
    if (batch <= 0 || batch % 128 != 0 || n_data_ < batch || epochs <= 0) return cudaErrorInvalidValue;
    QK_TRY(ensure_batch_buffers(batch));
    const int spe = static_cast<int>(n_data_ / batch);
    const int total = spe * epochs;
    SurState s{};
    QK_TRY(cudaMemcpy(&s, state_, sizeof s, cudaMemcpyDeviceToHost));
    const int step0 = s.step;
    if (loss_cap_ < step0 + total) {
        // half as much again, so that a caller training epoch by epoch does
        // not reallocate on every call
        const int cap = step0 + total + (step0 + total) / 2;
        loss_cap_ = 0;
        QK_TRY(dalloc(&loss_hist_, static_cast<size_t>(cap)));
        loss_cap_ = cap;
    }
    s.total_steps = step0 + total;
    s.step_begin = step0;
    s.steps_per_epoch = spe;
    s.batch = batch;
    s.lr0 = lr0;
    s.err = 0;
    // steps_per_epoch and batch change the gather: keep the step counter and
    // make epoch boundaries relative to it
    std::mt19937_64 rng(shuffle_seed);
    std::vector<int32_t> perm(static_cast<size_t>(n_data_));
    std::iota(perm.begin(), perm.end(), 0);
    // the gather reads perm[(step % spe) * batch + i]: the permutation goes up
    // rotated, in two pieces, so that the epoch starts at its beginning whatever
    // step0 % spe is.  The copies run on the stream, after the epoch before; the
    // next shuffle waits for them and overlaps this epoch.
    const int64_t head = static_cast<int64_t>(spe - step0 % spe) * batch;
    const int64_t all = static_cast<int64_t>(spe) * batch;
    auto upload = [&](int64_t to, int64_t from, int64_t count) -> cudaError_t {
        if (count == 0) return cudaSuccess;
        return cudaMemcpyAsync(perm_ + to, perm.data() + from, static_cast<size_t>(count) * sizeof(int32_t),
                               cudaMemcpyHostToDevice, stream_);
    };
    auto enqueue_epochs = [&]() -> cudaError_t {
        QK_TRY(cudaMemcpyAsync(state_, &s, sizeof s, cudaMemcpyHostToDevice, stream_));
        QK_TRY(arm_timeout(&state_->err));
        StepLaunch step;
        QK_TRY(prepare_steps(true, &step));
        for (int e = 0; e < epochs; ++e) {
            if (e > 0) QK_TRY(cudaEventSynchronize(uploaded_));
            std::shuffle(perm.begin(), perm.end(), rng);
            QK_TRY(upload(all - head, 0, head));
            QK_TRY(upload(0, head, all - head));
            if (e + 1 < epochs) QK_TRY(cudaEventRecord(uploaded_, stream_));
            for (int j = 0; j < spe; ++j) QK_TRY(run_step(step, stream_));
        }
        return cudaSuccess;
    };
    const cudaError_t enqueued = enqueue_epochs();
    const cudaError_t ran = cudaStreamSynchronize(stream_);  // also after an error: perm and s go
    QK_TRY(enqueued);
    QK_TRY(ran);
    QK_TRY(cudaMemcpy(&s, state_, sizeof s, cudaMemcpyDeviceToHost));
    if (s.err != 0) {
        pipeline_code_ = s.err;
        return cudaErrorLaunchTimeout;
    }
    std::vector<float> hist(static_cast<size_t>(total));
    QK_TRY(cudaMemcpy(hist.data(), loss_hist_ + step0, hist.size() * sizeof(float), cudaMemcpyDeviceToHost));
    if (out_loss_last) *out_loss_last = hist.back();
    if (out_epoch_loss) {
        for (int e = 0; e < epochs; ++e) {
            double acc = 0.0;
            for (int j = 0; j < spe; ++j) acc += hist[static_cast<size_t>(e) * spe + j];
            out_epoch_loss[e] = static_cast<float>(acc / spe);
        }
    }
    return cudaSuccess;
}

cudaError_t SurModel::ensure_predict_buffers(int64_t rows, size_t in_row) {
    if (rows > pred_rows_) {
        pred_rows_ = 0;
        QK_TRY(dalloc(&PX_, static_cast<size_t>(rows) * kSurInPad));
        QK_TRY(dalloc(&Perr_, static_cast<size_t>(rows) + kOutHead / sizeof(int)));
        QK_TRY(cudaMemsetAsync(Perr_, 0, kOutHead, stream_));
        Py_ = reinterpret_cast<float*>(Perr_ + kOutHead / sizeof(int));
        QK_TRY(dalloc(&Pbase_, static_cast<size_t>(rows)));
        pred_rows_ = rows;
    }
    const size_t bytes = in_row * static_cast<size_t>(rows);
    if (bytes > d_in_bytes_) {
        d_in_bytes_ = 0;
        QK_TRY(dalloc(&d_in_, bytes / sizeof(double) + 1));
        d_in_bytes_ = bytes;
    }
    return cudaSuccess;
}

// Hidden activations of the layer-by-layer path.
cudaError_t SurModel::ensure_layered_buffers(int64_t rows) {
    if (rows <= layered_rows_) return cudaSuccess;
    layered_rows_ = 0;
    QK_TRY(dalloc(&PH1_, static_cast<size_t>(rows) * kSurHid));
    QK_TRY(dalloc(&PH2_, static_cast<size_t>(rows) * kSurHid));
    layered_rows_ = rows;
    return cudaSuccess;
}

cudaError_t SurModel::predict_device(const __nv_bfloat16* x, const float* base, int64_t n, float* y,
                                     cudaStream_t st, bool layered) {
    return network(x, base, n, y, &state_->err, st, layered);
}

cudaError_t SurModel::network(const __nv_bfloat16* x, const float* base, int64_t n, float* y, int* err,
                              cudaStream_t st, bool layered) {
    DeviceGuard g(device_);
    if (base_kind_ != kSurBaseNone && base == nullptr) return cudaErrorInvalidValue;
    if (!layered) {
        if (sm_count_ <= 0)
            QK_TRY(cudaDeviceGetAttribute(&sm_count_, cudaDevAttrMultiProcessorCount, device_));
        CUtensorMap tx, tw1, tw2, tw3;
        if (!(make_tmap_bf16_k16(&tx, x, static_cast<uint64_t>(n), kSurInPad, 128) &&
              make_tmap_bf16_k16(&tw1, W1b_, kSurHid, kSurInPad, 256) &&
              tmap(&tw2, W2b_, kSurHid, kSurHid, 256) && tmap(&tw3, W3b_, kSurHid, kSurHid, 256)))
            return cudaErrorInvalidValue;
        InferArgs ia{};
        ia.n = n;
        ia.b1 = P_ + SurLayout::b1;
        ia.b2 = P_ + SurLayout::b2;
        ia.b3 = P_ + SurLayout::b3;
        ia.w4 = P_ + SurLayout::w4;
        ia.b4 = P_ + SurLayout::b4;
        ia.base = base_kind_ != kSurBaseNone ? base : nullptr;
        ia.y = y;
        ia.err = err;
        return launch_mlp_infer(tx, tw1, tw2, tw3, ia, sm_count_, st);
    }
    QK_TRY(ensure_layered_buffers(std::min<int64_t>(n, kPredChunk)));
    for (int64_t off = 0; off < n; off += kPredChunk) {
        const int64_t m = std::min<int64_t>(kPredChunk, n - off);
        CUtensorMap tx, tw1, th1, tw2, th2, tw3;
        bool ok = tmap(&tx, x + off * kSurInPad, m, kSurInPad, 128) && tmap(&tw1, W1b_, kSurHid, kSurInPad, 128) &&
                  tmap(&th1, PH1_, m, kSurHid, 128) && tmap(&tw2, W2b_, kSurHid, kSurHid, 128) &&
                  tmap(&th2, PH2_, m, kSurHid, 128) && tmap(&tw3, W3b_, kSurHid, kSurHid, 256);
        if (!ok) return cudaErrorInvalidValue;
        GemmArgs f{};
        f.err = err;
        f.M = static_cast<int>(m); f.N = kSurHid; f.K = kSurInPad; f.k_per_split = kSurInPad;
        f.bias = P_ + SurLayout::b1; f.h_out = PH1_;
        QK_TRY(launch_umma_gemm(kEpiFwd, 128, tx, tw1, f, 1, st));
        f.K = kSurHid; f.k_per_split = kSurHid; f.bias = P_ + SurLayout::b2; f.h_out = PH2_;
        QK_TRY(launch_umma_gemm(kEpiFwd, 128, th1, tw2, f, 1, st));
        GemmArgs l{};
        l.err = err;
        l.M = static_cast<int>(m); l.N = kSurHid; l.K = kSurHid; l.k_per_split = kSurHid;
        l.bias = P_ + SurLayout::b3; l.w4 = P_ + SurLayout::w4; l.b4 = P_ + SurLayout::b4;
        l.y_out = y + off;
        l.base = base_kind_ != kSurBaseNone ? base + off : nullptr;
        QK_TRY(launch_umma_gemm(kEpiLast, 256, th2, tw3, l, 1, st));
    }
    return cudaSuccess;
}

namespace {

// Two pinned slots of the calling thread (pinning 2 MB takes milliseconds, so
// a new model's first call must not pay for its own): each holds at most one
// chunk, a call drains both before it returns, and they go with the thread.
struct HostStage {
    PinnedBuf in[2], out[2];
    cudaEvent_t done[2] = {nullptr, nullptr};
    cudaError_t ensure(int slot, size_t in_bytes, size_t out_bytes) {
        QK_TRY(in[slot].ensure(in_bytes));
        QK_TRY(out[slot].ensure(out_bytes));
        if (!done[slot]) QK_TRY(cudaEventCreateWithFlags(&done[slot], cudaEventDisableTiming));
        return cudaSuccess;
    }
    ~HostStage() {
        for (int s = 0; s < 2; ++s) {
            in[s].release();
            out[s].release();
            if (done[s]) cudaEventDestroy(done[s]);
        }
    }
};

HostStage& thread_host_stage(int device) {
    thread_local std::map<int, std::unique_ptr<HostStage>> stages;
    auto& p = stages[device];
    if (!p) p.reset(new HostStage());
    return *p;
}

}  // namespace

// Host calls run in chunks of kPredChunk options through two pinned slots: a
// chunk's inputs are copied into its slot while the GPU works on the chunk
// before it, and a chunk's results leave its slot when the slot comes up
// again.  fill(h_in, off, m) copies inputs in, enqueue(h_in, h_out, m) queues
// the chunk's work on stream_, its results ending in h_out after kOutHead bytes
// that start with the error word, drain(results, off, m) copies them to the
// caller.  A chunk whose word is set has no results: the call fails.
template <class Fill, class Enqueue, class Drain>
cudaError_t SurModel::run_chunked(int64_t n, size_t in_row, size_t out_row, const Fill& fill,
                                  const Enqueue& enqueue, const Drain& drain) {
    const int64_t chunk = std::min<int64_t>(n, kPredChunk);
    QK_TRY(ensure_predict_buffers(chunk, in_row));
    HostStage& stage = thread_host_stage(device_);
    for (int s = 0; s < (n > chunk ? 2 : 1); ++s)
        QK_TRY(stage.ensure(s, in_row * static_cast<size_t>(chunk),
                            kOutHead + out_row * static_cast<size_t>(chunk)));
    struct Pending {
        int64_t off = 0, m = 0;
    } pending[2];
    cudaError_t e = cudaSuccess;
    auto finish = [&](int s) -> cudaError_t {
        if (pending[s].m == 0) return cudaSuccess;
        cudaError_t es = cudaEventSynchronize(stage.done[s]);
        if (es == cudaSuccess) {
            const char* h = static_cast<const char*>(stage.out[s].p);
            if (const int code = *reinterpret_cast<const int*>(h)) {
                pipeline_code_ = code;
                es = cudaErrorLaunchTimeout;
            } else {
                drain(h + kOutHead, pending[s].off, pending[s].m);
            }
        }
        pending[s].m = 0;
        return es;
    };
    int s = 0;
    for (int64_t off = 0; off < n && e == cudaSuccess; off += chunk, s ^= 1) {
        e = finish(s);
        if (e != cudaSuccess) break;
        const int64_t m = std::min<int64_t>(chunk, n - off);
        fill(static_cast<char*>(stage.in[s].p), off, m);
        e = enqueue(static_cast<char*>(stage.in[s].p), static_cast<char*>(stage.out[s].p), m);
        if (e == cudaSuccess) e = cudaEventRecord(stage.done[s], stream_);
        if (e == cudaSuccess) pending[s] = {off, m};
    }
    for (int k = 0; k < 2; ++k, s ^= 1) {
        const cudaError_t es = finish(s);
        if (e == cudaSuccess) e = es;
    }
    if (e != cudaSuccess) {
        cudaStreamSynchronize(stream_);  // nothing of the call stays in flight
        cudaMemsetAsync(Perr_, 0, kOutHead, stream_);
    }
    return e;
}

cudaError_t SurModel::predict(const double* features, int64_t n, double* out) {
    DeviceGuard g(device_);
    const size_t row = kSurIn * sizeof(double);
    return run_chunked(
        n, row, sizeof(float),
        [&](char* h, int64_t off, int64_t m) {
            std::memcpy(h, features + off * kSurIn, row * static_cast<size_t>(m));
        },
        [&](char* h_in, char* h_out, int64_t m) -> cudaError_t {
            QK_TRY(cudaMemcpyAsync(d_in_, h_in, row * static_cast<size_t>(m), cudaMemcpyHostToDevice, stream_));
            QK_TRY(features_device(d_in_, m, PX_, Pbase_, stream_));
            QK_TRY(arm_timeout(Perr_));
            QK_TRY(network(PX_, Pbase_, m, Py_, Perr_, stream_, false));
            return cudaMemcpyAsync(h_out, Perr_, kOutHead + sizeof(float) * static_cast<size_t>(m),
                                   cudaMemcpyDeviceToHost, stream_);
        },
        [&](const char* h, int64_t off, int64_t m) {
            const float* y = reinterpret_cast<const float*>(h);
            for (int64_t i = 0; i < m; ++i) out[off + i] = y[i];
        });
}

cudaError_t SurModel::price_quotes(const double* const (&cols)[10], const int32_t* option_type,
                                   int64_t n, double* out, int32_t* route, SurOutside* outside) {
    DeviceGuard g(device_);
    const size_t in_row = 10 * sizeof(double) + sizeof(int32_t);
    const size_t out_row = sizeof(double) + sizeof(int32_t);
    return run_chunked(
        n, in_row, out_row,
        [&](char* h, int64_t off, int64_t m) {
            for (const double* c : cols) {
                std::memcpy(h, c + off, sizeof(double) * static_cast<size_t>(m));
                h += sizeof(double) * static_cast<size_t>(m);
            }
            std::memcpy(h, option_type + off, sizeof(int32_t) * static_cast<size_t>(m));
        },
        [&](char* h_in, char* h_out, int64_t m) -> cudaError_t {
            const unsigned blocks = static_cast<unsigned>((m + kFeatRows - 1) / kFeatRows);
            const double* in = reinterpret_cast<const double*>(h_in);
            double* price = reinterpret_cast<double*>(h_out + kOutHead);
            quote_features_kernel<<<blocks, kFeatRows, 0, stream_>>>(
                in, m, box_, base_kind_, PX_, Pbase_, d_in_, reinterpret_cast<int32_t*>(price + m));
            QK_TRY(cudaGetLastError());
            QK_TRY(arm_timeout(Perr_));
            QK_TRY(network(PX_, Pbase_, m, Py_, Perr_, stream_, false));
            quote_price_kernel<<<blocks, kFeatRows, 0, stream_>>>(d_in_, m, Py_, price, Perr_,
                                                                  reinterpret_cast<int*>(h_out));
            return cudaGetLastError();
        },
        [&](const char* h, int64_t off, int64_t m) {
            const int32_t* to = reinterpret_cast<const int32_t*>(h + sizeof(double) * static_cast<size_t>(m));
            // a vector loop counts, the one below runs only where there are
            // some: alone it took 20,000 quotes from 207 to 230 us
            int64_t far = 0;
            for (int64_t i = 0; i < m; ++i) far += to[i] == 1;
            if (far > 0) {
                const size_t at = outside->index.size();
                outside->index.resize(at + static_cast<size_t>(far));
                outside->option_type.resize(at + static_cast<size_t>(far));
                int32_t* index = outside->index.data() + at;
                for (int64_t i = 0, k = 0; k < far; ++i)
                    if (to[i] == 1) index[k++] = static_cast<int32_t>(off + i);
                for (int64_t k = 0; k < far; ++k) outside->option_type[at + k] = option_type[index[k]];
                for (int c = 0; c < 10; ++c) {
                    outside->cols[c].resize(at + static_cast<size_t>(far));
                    for (int64_t k = 0; k < far; ++k) outside->cols[c][at + k] = cols[c][index[k]];
                }
            }
            std::memcpy(out + off, h, sizeof(double) * static_cast<size_t>(m));
            if (route) std::memcpy(route + off, to, sizeof(int32_t) * static_cast<size_t>(m));
        });
}

cudaError_t SurModel::gradients(const double* features, const double* target, int n, double* grads,
                                double* loss) {
    DeviceGuard g(device_);
    if (n <= 0 || n % 128 != 0) return cudaErrorInvalidValue;
    QK_TRY(set_dataset(features, target, n));
    QK_TRY(ensure_batch_buffers(n));
    SurState s{};
    QK_TRY(cudaMemcpy(&s, state_, sizeof s, cudaMemcpyDeviceToHost));
    if (loss_cap_ < s.step + 1) {
        QK_TRY(dalloc(&loss_hist_, static_cast<size_t>(s.step + 1)));
        loss_cap_ = s.step + 1;
    }
    s.batch = n;
    s.steps_per_epoch = 1;
    s.err = 0;
    QK_TRY(put(state_, &s, sizeof s));
    QK_TRY(arm_timeout(&state_->err));
    StepLaunch step;
    QK_TRY(prepare_steps(false, &step));
    QK_TRY(run_step(step, stream_));
    QK_TRY(cudaStreamSynchronize(stream_));
    QK_TRY(cudaMemcpy(&s, state_, sizeof s, cudaMemcpyDeviceToHost));
    if (s.err != 0) {
        pipeline_code_ = s.err;
        return cudaErrorLaunchTimeout;
    }
    std::vector<float> G(SurLayout::total);
    QK_TRY(cudaMemcpy(G.data(), G_, G.size() * sizeof(float), cudaMemcpyDeviceToHost));
    float l = 0.0f;
    QK_TRY(cudaMemcpy(&l, loss_hist_ + s.step, sizeof(float), cudaMemcpyDeviceToHost));
    if (loss) *loss = l;
    int k = 0;
    for (int r = 0; r < kSurHid; ++r)
        for (int c = 0; c < kSurIn; ++c) grads[k++] = G[SurLayout::W1 + r * kSurInPad + c];
    for (int i = SurLayout::b1; i <= SurLayout::b4; ++i) grads[k++] = G[i];
    return cudaSuccess;
}

cudaError_t SurModel::parameters(double* out) const {
    std::vector<float> P(SurLayout::total);
    QK_TRY(cudaMemcpy(P.data(), P_, P.size() * sizeof(float), cudaMemcpyDeviceToHost));
    int k = 0;
    for (int r = 0; r < kSurHid; ++r)
        for (int c = 0; c < kSurIn; ++c) out[k++] = P[SurLayout::W1 + r * kSurInPad + c];
    for (int i = SurLayout::b1; i <= SurLayout::b4; ++i) out[k++] = P[i];
    return cudaSuccess;
}

cudaError_t SurModel::set_parameters(const double* in) {
    DeviceGuard g(device_);
    std::vector<float> P(SurLayout::total, 0.0f);
    int k = 0;
    for (int r = 0; r < kSurHid; ++r)
        for (int c = 0; c < kSurIn; ++c) P[SurLayout::W1 + r * kSurInPad + c] = static_cast<float>(in[k++]);
    for (int i = SurLayout::b1; i <= SurLayout::b4; ++i) P[i] = static_cast<float>(in[k++]);
    QK_TRY(put(P_, P.data(), P.size() * sizeof(float)));
    QK_TRY(refresh_bf16(stream_));
    return cudaStreamSynchronize(stream_);
}

int SurModel::steps_done() const {
    SurState s{};
    if (cudaMemcpy(&s, state_, sizeof s, cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    return s.step;
}

int SurModel::take_pipeline_code() {
    const int code = pipeline_code_;
    pipeline_code_ = 0;
    return code;
}

// The injected form of a wait that ran out in the kernels of the next launch.
cudaError_t SurModel::arm_timeout(int* err) {
    if (injected_fault(kFaultTimeout) == cudaSuccess) return cudaSuccess;
    return cudaMemsetAsync(err, 1, sizeof(int), stream_);
}

// Checkpoint: "QKSURv02", layout size, base kind, the box, the state, P, M, V
// (FP32).  "QKSURv01" files (no base kind: a network without a base) load too.
cudaError_t SurModel::save(const char* path) {
    DeviceGuard g(device_);
    SurState s{};
    QK_TRY(cudaMemcpy(&s, state_, sizeof s, cudaMemcpyDeviceToHost));
    std::vector<float> buf(static_cast<size_t>(SurLayout::total) * 3);
    QK_TRY(cudaMemcpy(buf.data(), P_, SurLayout::total * sizeof(float), cudaMemcpyDeviceToHost));
    QK_TRY(cudaMemcpy(buf.data() + SurLayout::total, M_, SurLayout::total * sizeof(float), cudaMemcpyDeviceToHost));
    QK_TRY(cudaMemcpy(buf.data() + 2 * SurLayout::total, V_, SurLayout::total * sizeof(float), cudaMemcpyDeviceToHost));
    FILE* f = std::fopen(path, "wb");
    if (!f) return cudaErrorInvalidValue;
    const char magic[8] = {'Q', 'K', 'S', 'U', 'R', 'v', '0', '2'};
    const int32_t total = SurLayout::total;
    bool ok = std::fwrite(magic, 1, 8, f) == 8 && std::fwrite(&total, sizeof total, 1, f) == 1 &&
              std::fwrite(&base_kind_, sizeof base_kind_, 1, f) == 1 &&
              std::fwrite(&box_, sizeof box_, 1, f) == 1 && std::fwrite(&s, sizeof s, 1, f) == 1 &&
              std::fwrite(buf.data(), sizeof(float), buf.size(), f) == buf.size();
    ok = (std::fclose(f) == 0) && ok;
    return ok ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t SurModel::load(const char* path) {
    DeviceGuard g(device_);
    FILE* f = std::fopen(path, "rb");
    if (!f) return cudaErrorInvalidValue;
    char magic[8];
    int32_t total = 0, kind = kSurBaseNone;
    SurBox box{};
    SurState s{};
    std::vector<float> buf(static_cast<size_t>(SurLayout::total) * 3);
    bool ok = std::fread(magic, 1, 8, f) == 8;
    const bool v2 = ok && std::memcmp(magic, "QKSURv02", 8) == 0;
    ok = ok && (v2 || std::memcmp(magic, "QKSURv01", 8) == 0) &&
         std::fread(&total, sizeof total, 1, f) == 1 && total == SurLayout::total &&
         (!v2 || std::fread(&kind, sizeof kind, 1, f) == 1) &&
         (kind == kSurBaseNone || kind == kSurBaseBsmMeanVar) &&
         std::fread(&box, sizeof box, 1, f) == 1 && std::fread(&s, sizeof s, 1, f) == 1 &&
         std::fread(buf.data(), sizeof(float), buf.size(), f) == buf.size();
    std::fclose(f);
    if (!ok) return cudaErrorInvalidValue;
    box_ = box;
    base_kind_ = kind;
    s.err = 0;
    QK_TRY(put(state_, &s, sizeof s));
    QK_TRY(put(P_, buf.data(), SurLayout::total * sizeof(float)));
    QK_TRY(put(M_, buf.data() + SurLayout::total, SurLayout::total * sizeof(float)));
    QK_TRY(put(V_, buf.data() + 2 * SurLayout::total, SurLayout::total * sizeof(float)));
    QK_TRY(refresh_bf16(stream_));
    return cudaStreamSynchronize(stream_);
}

}  // namespace qkb
