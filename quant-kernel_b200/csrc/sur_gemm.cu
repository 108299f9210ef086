// sur_gemm.cu -- tcgen05 / TMEM / TMA BF16 GEMM with fused MLP epilogues.
// See sur_gemm.cuh for the structure.
#include "sur_gemm.cuh"

#include <cudaTypedefs.h>

#include <mutex>

namespace qkb {

namespace {

constexpr int kStages = 4;
constexpr int kBM = 128;
constexpr int kBK = 64;                       // 64 bf16 = 128 B = one swizzle row
constexpr uint32_t kSpinLimit = 1u << 25;     // bounded mbarrier polls (seconds)
constexpr uint32_t kABytes = kBM * kBK * 2;   // 16 KiB
constexpr int kSurHidden = 256;               // hidden width of the surrogate MLP

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// One lane of a converged warp.  tcgen05 and TMA instructions take their
// operands from uniform registers: under this predicate the compiler knows
// that one lane is active.
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
    return e != 0;
}

// Whether the phase has completed, without waiting.
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait: false after kSpinLimit polls (each poll may suspend briefly).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kSpinLimit; ++i)
        if (mbar_try(bar, parity)) return true;
    return false;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 B apart (SBO), leading offset unused for swizzled K-major (1),
// descriptor version 1 (sm_100), layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t desc_sw128(uint32_t addr) {
    return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>(1) << 16) |
           (static_cast<uint64_t>(1024 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
           (static_cast<uint64_t>(2) << 61);
}

// The same for 32-byte rows (K = 16 bf16): 32-byte swizzle, 8-row groups 256
// B apart, layout type 6 (SWIZZLE_32B).
__device__ __forceinline__ uint64_t desc_sw32(uint32_t addr) {
    return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>(1) << 16) |
           (static_cast<uint64_t>(256 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
           (static_cast<uint64_t>(6) << 61);
}

// Instruction descriptor, kind::f16: D fp32, A and B bf16, both K-major,
// N >> 3 at bit 17, M >> 4 at bit 24.
template <int BN>
__device__ __forceinline__ constexpr uint32_t idesc_bf16() {
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(BN >> 3) << 17) |
           (static_cast<uint32_t>(kBM >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ void fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// 32 consecutive fp32 columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// sigmoid(z) = (1 + tanh(z / 2)) / 2 with the MUFU tanh (one special-function
// op; |error| ~ 2^-11, below the bf16 rounding every activation gets next).
__device__ __forceinline__ float tanh_approx(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float sigmoidf_(float z) { return fmaf(0.5f, tanh_approx(0.5f * z), 0.5f); }

// SiLU straight from the accumulator: hz = z / 2 = fma(acc, 1/2, bias / 2) is
// exact (halving commutes with the rounding of acc + bias), so tanh(hz) is the
// sigmoid's tanh(z / 2), and silu(z) = z sigma(z) = hz + hz tanh(hz): two FMAs
// around one MUFU op.  Returns silu; hz and t = tanh(hz) for the caller.
__device__ __forceinline__ float silu_from_acc(float acc, float half_bias, float& hz, float& t) {
    hz = fmaf(acc, 0.5f, half_bias);
    t = tanh_approx(hz);
    return fmaf(hz, t, hz);
}

// silu_from_acc on two adjacent columns, the two FMAs as packed f32x2
// operations (each lane rounded as the scalar fmaf: the same bits).
__device__ __forceinline__ float2 silu2_from_acc(float2 acc, float2 half_bias) {
    const float2 hz = __ffma2_rn(acc, make_float2(0.5f, 0.5f), half_bias);
    const float2 t = make_float2(tanh_approx(hz.x), tanh_approx(hz.y));
    return __ffma2_rn(hz, t, hz);
}

// 32 bf16 values to 64 contiguous bytes.
__device__ __forceinline__ void store_bf16x32(__nv_bfloat16* dst, const float (&v)[32]) {
    uint4* d = reinterpret_cast<uint4*>(dst);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        __nv_bfloat162 p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = __floats2bfloat162_rn(v[q * 8 + 2 * j], v[q * 8 + 2 * j + 1]);
        d[q] = *reinterpret_cast<uint4*>(p);
    }
}

// Eight epilogue warps: warp w reads TMEM lanes 32 (w % 4) .. + 31 (its tile
// rows) and the column half w / 4 of the tile (chunks of 32 columns
// [c_lo, c_hi)); every element's arithmetic is the same as with one warp per
// lane quarter, so the split changes no bits.
template <int BN, int EPI>
__device__ __forceinline__ void epilogue(const GemmArgs& a, uint32_t tmem, int m0, int n0,
                                         float (*part_s)[kBM]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int q = warp & 3, half = warp >> 2;
    const int row = m0 + q * 32 + lane;
    const bool live = row < a.M;
    const uint32_t tbase = tmem + (static_cast<uint32_t>(q * 32) << 16);
    constexpr int kChunks = BN / 32;
    const int c_lo = half * (kChunks / 2), c_hi = c_lo + kChunks / 2;
    float v[32];
    if (EPI == kEpiF32) {
#pragma unroll 1
        for (int c = c_lo; c < c_hi; ++c) {
            tmem_ld32(tbase + c * 32, v);
            if (live) {
                float4* dst = reinterpret_cast<float4*>(
                    a.c_f32 + (static_cast<size_t>(blockIdx.z) * a.M + row) * a.N + n0 + c * 32);
#pragma unroll
                for (int q = 0; q < 8; ++q) dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            }
        }
    } else if (EPI == kEpiFwd) {
#pragma unroll 1
        for (int c = c_lo; c < c_hi; ++c) {
            tmem_ld32(tbase + c * 32, v);
            const int col0 = n0 + c * 32;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                float hz, t;
                v[j] = silu_from_acc(v[j], 0.5f * __ldg(a.bias + col0 + j), hz, t);
            }
            if (live) store_bf16x32(a.h_out + static_cast<size_t>(row) * a.N + col0, v);
        }
    } else {  // kEpiLast: BN == N (the whole hidden row is in this CTA)
        // head dot product as four partial sums, group g over the columns
        // 64 kb + 16 g + j (kb = 0..3, j = 0..15, in that order), combined in
        // order -- the summation of the fused inference kernel, whose warp g
        // owns those columns.  This warp's half takes groups 2 half, 2 half + 1.
        float p0 = 0.0f, p1 = 0.0f;
#pragma unroll 1
        for (int kb = 0; kb < 4; ++kb) {
            const int col0 = kb * 64 + half * 32;  // groups 2 half (16 cols), 2 half + 1 (16)
            tmem_ld32(tbase + col0, v);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                float hz, t;
                const float h = silu_from_acc(v[j], 0.5f * __ldg(a.bias + col0 + j), hz, t);
                p0 = fmaf(h, __ldg(a.w4 + col0 + j), p0);
            }
#pragma unroll
            for (int j = 16; j < 32; ++j) {
                float hz, t;
                const float h = silu_from_acc(v[j], 0.5f * __ldg(a.bias + col0 + j), hz, t);
                p1 = fmaf(h, __ldg(a.w4 + col0 + j), p1);
            }
        }
        part_s[2 * half][q * 32 + lane] = p0;
        part_s[2 * half + 1][q * 32 + lane] = p1;
        __syncthreads();  // all eight warps run the epilogue
        const int r = q * 32 + lane;
        float y = ((part_s[0][r] + part_s[1][r]) + part_s[2][r]) + part_s[3][r];
        y += __ldg(a.b4);
        if (live && half == 0) a.y_out[row] = a.base ? y + __ldg(a.base + row) : y;
    }
}

constexpr int kGemmThreads = 256;  // warp 0: TMA, warp 1: MMA; all 8 warps: epilogue

template <int BN, int EPI>
__global__ void __launch_bounds__(kGemmThreads, 1)
    umma_gemm_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
                     const GemmArgs a) {
    constexpr uint32_t kBBytes = BN * kBK * 2;
    constexpr uint32_t kStage = kABytes + kBBytes;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    __shared__ __align__(8) uint64_t full_bar[kStages];
    __shared__ __align__(8) uint64_t empty_bar[kStages];
    __shared__ __align__(8) uint64_t acc_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    __shared__ float part_s[4][kBM];  // head partial sums (kEpiLast)

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * kBM, n0 = blockIdx.y * BN;
    const int kb0 = blockIdx.z * (a.k_per_split / kBK);
    int krem = a.K - blockIdx.z * a.k_per_split;
    if (krem > a.k_per_split) krem = a.k_per_split;
    const int nkb = krem > 0 ? krem / kBK : 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(smem_u32(&full_bar[s]), 1);
            mbar_init(smem_u32(&empty_bar[s]), 1);
        }
        mbar_init(smem_u32(&acc_bar), 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_slot)),
                     "r"(static_cast<uint32_t>(BN))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot;

    int last_round[kStages];
#pragma unroll
    for (int s = 0; s < kStages; ++s) last_round[s] = -1;

    if (warp == 0 && lane == 0) {
        // TMA producer
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = kb % kStages;
            const int round = kb / kStages;
            if (round > 0 && !mbar_wait(smem_u32(&empty_bar[s]), (round - 1) & 1)) {
                abort_flag = 1;
                atomicExch(a.err, 1);
                break;
            }
            if (abort_flag) break;
            const uint32_t sa = smem_u32(smem + s * kStage);
            mbar_expect_tx(smem_u32(&full_bar[s]), kStage);
            const int kx = (kb0 + kb) * kBK;
            tma_load_2d(sa, &ta, kx, m0, smem_u32(&full_bar[s]));
            tma_load_2d(sa + kABytes, &tb, kx, n0, smem_u32(&full_bar[s]));
            last_round[s] = round;
        }
    } else if (warp == 1 && lane == 0) {
        // MMA issuer
        constexpr uint32_t idesc = idesc_bf16<BN>();
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = kb % kStages;
            if (!mbar_wait(smem_u32(&full_bar[s]), (kb / kStages) & 1)) {
                abort_flag = 1;
                atomicExch(a.err, 2);
                break;
            }
            if (abort_flag) break;
            fence_after();
            const uint32_t sa = smem_u32(smem + s * kStage);
#pragma unroll
            for (int kk = 0; kk < kBK / 16; ++kk)
                umma_bf16(tmem, desc_sw128(sa + kk * 32), desc_sw128(sa + kABytes + kk * 32), idesc,
                          (kb | kk) != 0 ? 1u : 0u);
            umma_commit(smem_u32(&empty_bar[s]));
        }
        umma_commit(smem_u32(&acc_bar));  // arrives once every issued MMA has completed
    }
    __syncwarp();

    // Epilogue: accumulator ready (bounded wait), then TMEM -> registers -> global.
    const bool acc_ok = mbar_wait(smem_u32(&acc_bar), 0);
    __syncwarp();
    fence_after();
    if (!acc_ok) {
        if (threadIdx.x == 0) atomicExch(a.err, 3);
        abort_flag = 1;
    }
    __syncthreads();
    if (!abort_flag && nkb > 0) epilogue<BN, EPI>(a, tmem, m0, n0, part_s);

    // Teardown: the producer drains its own loads (bounded), then TMEM is freed.
    if (warp == 0 && lane == 0 && abort_flag) {
        for (int s = 0; s < kStages; ++s)
            if (last_round[s] >= 0) mbar_wait(smem_u32(&full_bar[s]), last_round[s] & 1);
    }
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(static_cast<uint32_t>(BN))
                     : "memory");
    }
}


// ----------------------------------------------------------------------------
// Fused MLP inference.  One persistent CTA per SM walks its 128-row tiles two
// at a time, ping-pong: tile slot s (0, 1) owns TMEM accumulator s (256 fp32
// columns), a 64 KiB shared buffer of activations and a 4 KiB one of input
// rows.  While the epilogue warps work on one slot's layer, the tensor core
// computes the other slot's.  Four warp roles:
//   warp 16 (one lane)  weight producer: W1's first 16 columns once (8 KiB,
//                       resident), then the 32 KiB k-blocks of W2 and W3 in
//                       the order the MMA issuer takes them (per tile pair:
//                       W2[0..3] for A, for B, W3[0..3] for A, for B) through
//                       a 2-slot ring;
//   warp 17 (one lane)  MMA issuer: per tile pair A, B: layer 2 of A, of B,
//                       layer 3 of A, of B, each once the epilogue has written
//                       the slot's previous layer.  Layer 1 (one K = 16 MMA:
//                       the 9 features and their zero padding; the rows'
//                       columns 16..63 are zeros too and would add exact
//                       zeros) of the next A goes in among the k-blocks of B's
//                       layer 3, of the next B among those of A's layer 2, as
//                       soon as the head has read the slot's accumulator;
//   warp 18 (one lane)  input loader: a slot's next input rows (their first
//                       16 columns, 32-byte swizzled) once its previous tile's
//                       layer 1 has read the buffer;
//   warps 0-15          epilogue: layer 2 of A, of B, the head of A, layer 1
//                       of the next A, the head of B, layer 1 of the next B;
//                       warp w reads TMEM lanes 32 (w % 4) .. + 31 (its tile
//                       rows) and, in each 64-column block kb, columns 64 kb +
//                       16 (w / 4) .. + 15; bias + SiLU, BF16 into the slot's
//                       buffer in the 128-byte-swizzled K-major layout the
//                       next layer's MMA reads as its A operand; the head sums
//                       partial chains and writes the prices.
// Every hand-off is an mbarrier with a bounded wait (no CTA-wide barrier
// inside the loop), so a timeout anywhere ends every role with an error code.
// Barriers per slot: xfull (input rows landed), xfree (layer 1 has read them),
// accfull (a layer's MMAs complete: three phases per tile), hdone (all 16
// epilogue warps finished a layer of the slot: three phases per tile), pready
// (the head's partial sums, one phase per tile).  Hazards, each closed by the
// chain: an accumulator is rewritten only after hdone reports the epilogue
// read it; a buffer of activations is rewritten by the epilogue only after
// accfull reports that the MMAs which read it completed; the head's partial
// sums are double-buffered by slot.
// The arithmetic and summation order are those of the layer-by-layer GEMMs
// (kEpiFwd, kEpiLast), so the results are the same bits.
//
// Bound by the chain of a slot (epilogue, hand-off, MMAs) and the ring, whose
// two blocks take 1.8k cycles to come round: 10.5k cycles a tile, 6.3k of them
// in the epilogue, whose tanh needs 6.1k.  With layer 1 after both heads and
// the issuing lane chosen by its number, a million rows took 355 us, now 335
// (100,000: 42.1 with their features, now 40.4).  Pairs of CTAs that share the
// weight blocks (cta_group::2) took 395: beside the faster MMAs the epilogue
// slows from 2.1k to 3k cycles a layer.
// ----------------------------------------------------------------------------
constexpr int kIWSlots = 2;
constexpr uint32_t kWBlock = 256 * kBK * 2;        // 32 KiB: 256 rows x 64 bf16
constexpr uint32_t kHBytes = 4 * kABytes;          // 64 KiB: 128 rows x 256 bf16
constexpr int kTileSlots = 2;
// Layer 1 reads only K = 16 (the 9 features and their zero padding): input
// rows of 32 bytes, and W1's first 16 columns held resident for the launch.
constexpr uint32_t kXBytes = kBM * 16 * 2;         // 4 KiB: 128 rows x 16 bf16
constexpr uint32_t kW1Bytes = 256 * 16 * 2;        // 8 KiB: 256 rows x 16 bf16
constexpr size_t kInferSmem = kTileSlots * (kHBytes + kXBytes) + kIWSlots * kWBlock + kW1Bytes + 1024;
constexpr int kInferEpiWarps = 16;                 // 4 per TMEM lane quarter
constexpr int kInferThreads = (kInferEpiWarps + 3) * 32;
constexpr int kProducerWarp = kInferEpiWarps, kMmaWarp = kInferEpiWarps + 1,
              kXWarp = kInferEpiWarps + 2;

// 16 consecutive fp32 columns of this thread's TMEM lane (no wait).
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// 16 activations (columns col0 .. col0 + 15 of tile row r, col0 % 16 == 0)
// into the layout a 128-byte-swizzle TMA load would produce: k-block
// col / 64, row r at 128 r, 16-byte chunk c at (c ^ (r & 7)) * 16.
__device__ __forceinline__ void store_h16_sw128(uint8_t* hbuf, int r, int col0, const float (&v)[16]) {
    uint8_t* row = hbuf + (col0 >> 6) * kABytes + r * 128;
    const int c0 = (col0 & 63) >> 3;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        __nv_bfloat162 p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = __floats2bfloat162_rn(v[q * 8 + 2 * j], v[q * 8 + 2 * j + 1]);
        *reinterpret_cast<uint4*>(row + (((c0 + q) ^ (r & 7)) << 4)) = *reinterpret_cast<uint4*>(p);
    }
}

__global__ void __launch_bounds__(kInferThreads, 1)
    mlp_infer_kernel(const __grid_constant__ CUtensorMap tx, const __grid_constant__ CUtensorMap tw1,
                     const __grid_constant__ CUtensorMap tw2, const __grid_constant__ CUtensorMap tw3,
                     const InferArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    uint8_t* hbufs = smem;  // [kTileSlots][kHBytes]: a slot's activations
    uint8_t* wbuf = smem + kTileSlots * kHBytes;
    uint8_t* w1s = wbuf + kIWSlots * kWBlock;  // W1 [256][16], resident
    uint8_t* xbufs = w1s + kW1Bytes;           // [kTileSlots][kXBytes]: a slot's input rows
    __shared__ __align__(8) uint64_t w1full;
    __shared__ __align__(8) uint64_t xfull[kTileSlots], xfree[kTileSlots], accfull[kTileSlots];
    __shared__ __align__(8) uint64_t hdone[kTileSlots], pready[kTileSlots];
    __shared__ __align__(8) uint64_t wfull[kIWSlots], wempty[kIWSlots], drain;
    __shared__ __align__(16) float sb1[kSurHidden], sb2[kSurHidden], sb3[kSurHidden], sw4[kSurHidden];
    __shared__ float part[kTileSlots][4][kBM];  // head partial sums per slot and column group
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t n_tiles = (a.n + kBM - 1) / kBM;
    // this CTA's tiles i = 0, 1, ...: tile blockIdx.x + i gridDim.x, slot i % 2,
    // the slot's use u = i / 2; tiles 2p and 2p + 1 form pair p
    const int64_t my_tiles =
        blockIdx.x < n_tiles ? (n_tiles - 1 - static_cast<int64_t>(blockIdx.x)) / gridDim.x + 1 : 0;

    if (tid < kSurHidden) {
        sb1[tid] = 0.5f * a.b1[tid];  // halved biases for silu_from_acc (exact)
        sb2[tid] = 0.5f * a.b2[tid];
        sb3[tid] = 0.5f * a.b3[tid];
        sw4[tid] = a.w4[tid];
    }
    if (tid == 0) {
        for (int s = 0; s < kTileSlots; ++s) {
            mbar_init(smem_u32(&xfull[s]), 1);
            mbar_init(smem_u32(&xfree[s]), 1);
            mbar_init(smem_u32(&accfull[s]), 1);
            mbar_init(smem_u32(&hdone[s]), kInferEpiWarps);
            mbar_init(smem_u32(&pready[s]), kInferEpiWarps);
        }
        for (int s = 0; s < kIWSlots; ++s) {
            mbar_init(smem_u32(&wfull[s]), 1);
            mbar_init(smem_u32(&wempty[s]), 1);
        }
        mbar_init(smem_u32(&drain), 1);
        mbar_init(smem_u32(&w1full), 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {  // one accumulator of 256 fp32 columns per tile slot
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot;
    auto fail = [&](int code) {
        abort_flag = 1;
        atomicExch(a.err, code);
    };

    // bookkeeping for the teardown drain
    int last_round[kIWSlots] = {-1, -1};
    int64_t x_last[kTileSlots] = {-1, -1};
    bool w1_issued = false;
    bool leader = false;  // this warp's elected lane

    if (warp == kProducerWarp) {
        if (elect_one()) {
            leader = true;
            uint32_t wl = 0;
            auto load_w = [&](const CUtensorMap* m, int kx) -> bool {
                const uint32_t s = wl % kIWSlots, round = wl / kIWSlots;
                if (round > 0 && !mbar_wait(smem_u32(&wempty[s]), (round - 1) & 1)) return false;
                mbar_expect_tx(smem_u32(&wfull[s]), kWBlock);
                tma_load_2d(smem_u32(wbuf + s * kWBlock), m, kx, 0, smem_u32(&wfull[s]));
                last_round[s] = static_cast<int>(round);
                ++wl;
                return true;
            };
            if (my_tiles > 0) {  // W1's first 16 columns, once
                mbar_expect_tx(smem_u32(&w1full), kW1Bytes);
                tma_load_2d(smem_u32(w1s), &tw1, 0, 0, smem_u32(&w1full));
                w1_issued = true;
            }
            for (int64_t i0 = 0; i0 < my_tiles; i0 += 2) {
                if (abort_flag) break;
                const int nt = (my_tiles - i0) >= 2 ? 2 : 1;
                // the MMA issuer's order: layers 2 and 3 for tile A, then tile B
                bool ok = true;
                for (int k = 0; ok && k < nt; ++k)
                    for (int kb = 0; ok && kb < 4; ++kb) ok = load_w(&tw2, kb * kBK);
                for (int k = 0; ok && k < nt; ++k)
                    for (int kb = 0; ok && kb < 4; ++kb) ok = load_w(&tw3, kb * kBK);
                if (!ok) {
                    fail(22);
                    break;
                }
            }
        }
    } else if (warp == kXWarp) {
        if (elect_one()) {
            leader = true;
            for (int64_t i = 0; i < my_tiles; ++i) {
                if (abort_flag) break;
                const int s = static_cast<int>(i & 1);
                const int64_t u = i >> 1;
                // layer 1 of the slot's previous tile, the buffer's reader, has
                // completed (one xfree phase per tile)
                if (u > 0 && !mbar_wait(smem_u32(&xfree[s]), static_cast<uint32_t>((u - 1) & 1))) {
                    fail(21);
                    break;
                }
                mbar_expect_tx(smem_u32(&xfull[s]), kXBytes);
                const int64_t t = blockIdx.x + i * gridDim.x;
                tma_load_2d(smem_u32(xbufs + s * kXBytes), &tx, 0, static_cast<int>(t * kBM),
                            smem_u32(&xfull[s]));
                x_last[s] = u;
            }
        }
    } else if (warp == kMmaWarp) {
        if (elect_one()) {
            leader = true;
            constexpr uint32_t idesc = idesc_bf16<256>();
            uint32_t wc = 0;
            // one k-block of W from the ring into accumulator acc
            auto mma_kblock = [&](uint32_t acc, uint32_t sa, bool first) -> bool {
                const uint32_t s = wc % kIWSlots;
                if (!mbar_wait(smem_u32(&wfull[s]), (wc / kIWSlots) & 1)) return false;
                fence_after();
                const uint32_t sb = smem_u32(wbuf + s * kWBlock);
#pragma unroll
                for (int kk = 0; kk < kBK / 16; ++kk)
                    umma_bf16(acc, desc_sw128(sa + kk * 32), desc_sw128(sb + kk * 32), idesc,
                              (first && kk == 0) ? 0u : 1u);
                umma_commit(smem_u32(&wempty[s]));
                ++wc;
                return true;
            };
            bool ok = my_tiles == 0 || mbar_wait(smem_u32(&w1full), 0u);
            if (!ok) fail(25);
            const uint64_t dw1 = desc_sw32(smem_u32(w1s));
            // layer 1 of tile i, one K = 16 MMA, once its input rows have landed
            // and the head of the slot's previous tile has read the accumulator;
            // where wait is false only if both have happened
            auto layer1 = [&](int64_t i, bool wait) -> bool {
                const int s = static_cast<int>(i & 1);
                const int64_t u = i >> 1;
                const uint32_t xp = static_cast<uint32_t>(u & 1), hp = static_cast<uint32_t>((3 * u - 1) & 1);
                if (wait) {
                    ok = ok && mbar_wait(smem_u32(&xfull[s]), xp) && (u == 0 || mbar_wait(smem_u32(&hdone[s]), hp));
                    if (!ok) return false;
                } else if (!mbar_test(smem_u32(&xfull[s]), xp) || (u > 0 && !mbar_test(smem_u32(&hdone[s]), hp))) {
                    return false;
                }
                fence_after();
                umma_bf16(tmem + s * 256, desc_sw32(smem_u32(xbufs + s * kXBytes)), dw1, idesc, 0u);
                umma_commit(smem_u32(&xfree[s]));
                umma_commit(smem_u32(&accfull[s]));
                return true;
            };
            // layer l (1, 2) of tile i, once every epilogue warp has written its
            // activations and read its accumulator; layer 1 of tile `next` goes
            // in between as soon as it can
            auto layer = [&](int64_t i, int l, int64_t next) {
                const int s = static_cast<int>(i & 1);
                bool pending = next < my_tiles;
                if (pending) pending = !layer1(next, false);
                ok = ok && mbar_wait(smem_u32(&hdone[s]), static_cast<uint32_t>((3 * (i >> 1) + l - 1) & 1));
                fence_after();
                for (int kb = 0; ok && kb < 4; ++kb) {
                    if (pending) pending = !layer1(next, false);
                    ok = mma_kblock(tmem + s * 256, smem_u32(hbufs + s * kHBytes + kb * kABytes), kb == 0);
                }
                if (ok) umma_commit(smem_u32(&accfull[s]));
                if (ok && pending) layer1(next, true);
            };
            if (ok && my_tiles > 0 && !layer1(0, true)) fail(24);
            for (int64_t i = 0; ok && i < my_tiles; i += 2) {
                if (abort_flag) break;
                const bool two = i + 1 < my_tiles;
                layer(i, 1, i + 1);
                if (two) layer(i + 1, 1, my_tiles);
                layer(i, 2, my_tiles);
                if (two) layer(i + 1, 2, i + 2);
                if (!ok) fail(24);
            }
        }
    } else {
        // epilogue warps; lane 0 polls each barrier and broadcasts the
        // outcome, so a warp's lanes always take the same path; then every
        // lane observes the completed phase itself (its own acquire: the
        // phase cannot advance again before this warp's next arrival)
        auto warp_wait = [&](uint32_t bar, uint32_t parity) -> bool {
            bool done = false;
            if (lane == 0) done = mbar_wait(bar, parity);
            done = __shfl_sync(0xFFFFFFFFu, done ? 1 : 0, 0) != 0;
            if (done) done = __all_sync(0xFFFFFFFFu, mbar_try(bar, parity)) != 0;
            return done;
        };
        const int q = warp & 3, g = warp >> 2;
        const int r = q * 32 + lane;
        const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
        const float b4 = __ldg(a.b4);
        bool ok = true;
        // layer 1 of the first two tiles, then pair by pair: layer 2 of A and
        // of B, the head of A, layer 1 of the next A, the head of B, layer 1 of
        // the next B (bit pairs of `kLayers`, bits of `kSlots`, lowest first)
        constexpr uint32_t kLayers = 1u | 1u << 2 | 2u << 4 | 0u << 6 | 2u << 8 | 0u << 10;
        constexpr uint32_t kSlots = 0u | 1u << 1 | 0u << 2 | 0u << 3 | 1u << 4 | 1u << 5;
        for (int64_t i0 = -2; ok && i0 < my_tiles; i0 += 2) {
            for (int e = 0; ok && e < 6; ++e) {
                const int l = (kLayers >> (2 * e)) & 3, s = (kSlots >> e) & 1;
                const int64_t i = i0 + s + (l == 0 ? 2 : 0);
                if (i < 0 || i >= my_tiles) continue;
                const int64_t u = i >> 1;
                const uint32_t acc = tmem + s * 256 + lane_off;
                ok = warp_wait(smem_u32(&accfull[s]), static_cast<uint32_t>((3 * u + l) & 1));
                fence_after();
                if (!ok) {
                    if (lane == 0) fail(26);
                    break;
                }
                if (l < 2) {
                    const float* bias = l == 0 ? sb1 : sb2;
                    uint8_t* hbuf = hbufs + s * kHBytes;
#pragma unroll
                    for (int kb = 0; kb < 4; ++kb) {
                        const int col0 = kb * 64 + g * 16;
                        uint32_t uu[16];
                        tmem_ld16_async(acc + col0, uu);
                        tmem_wait_ld();
                        float v[16];
#pragma unroll
                        for (int j = 0; j < 16; j += 4) {
                            const float4 b = *reinterpret_cast<const float4*>(bias + col0 + j);
                            const float2 h0 = silu2_from_acc(
                                make_float2(__uint_as_float(uu[j]), __uint_as_float(uu[j + 1])),
                                make_float2(b.x, b.y));
                            const float2 h1 = silu2_from_acc(
                                make_float2(__uint_as_float(uu[j + 2]), __uint_as_float(uu[j + 3])),
                                make_float2(b.z, b.w));
                            v[j] = h0.x;
                            v[j + 1] = h0.y;
                            v[j + 2] = h1.x;
                            v[j + 3] = h1.y;
                        }
                        store_h16_sw128(hbuf, r, col0, v);
                    }
                    // the shared stores to the tensor core's (async) proxy,
                    // the TMEM reads before the hand-off
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&hdone[s]));
                } else {
                    // head: this warp's chain over columns 64 kb + 16 g + j
                    float p = 0.0f;
#pragma unroll
                    for (int kb = 0; kb < 4; ++kb) {
                        const int col0 = kb * 64 + g * 16;
                        uint32_t uu[16];
                        tmem_ld16_async(acc + col0, uu);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 16; j += 4) {
                            const float4 b = *reinterpret_cast<const float4*>(sb3 + col0 + j);
                            const float4 w = *reinterpret_cast<const float4*>(sw4 + col0 + j);
                            const float2 h0 = silu2_from_acc(
                                make_float2(__uint_as_float(uu[j]), __uint_as_float(uu[j + 1])),
                                make_float2(b.x, b.y));
                            const float2 h1 = silu2_from_acc(
                                make_float2(__uint_as_float(uu[j + 2]), __uint_as_float(uu[j + 3])),
                                make_float2(b.z, b.w));
                            p = fmaf(h0.x, w.x, p);
                            p = fmaf(h0.y, w.y, p);
                            p = fmaf(h1.x, w.z, p);
                            p = fmaf(h1.y, w.w, p);
                        }
                    }
                    // the accumulator is read: the slot's next tile may start
                    // its layer 1
                    fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&hdone[s]));
                    part[s][g][r] = p;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_u32(&pready[s]));
                    if (g == 0) {
                        ok = warp_wait(smem_u32(&pready[s]), static_cast<uint32_t>(u & 1));
                        if (!ok) {
                            if (lane == 0) fail(27);
                            break;
                        }
                        const float y =
                            (((part[s][0][r] + part[s][1][r]) + part[s][2][r]) + part[s][3][r]) + b4;
                        const int64_t row = (blockIdx.x + i * gridDim.x) * kBM + r;
                        if (row < a.n) a.y[row] = a.base ? y + __ldg(a.base + row) : y;
                    }
                }
            }
        }
    }

    // Teardown.  After an abort: the producer and the input loader wait
    // (bounded) for the loads they issued, the MMA issuer for its MMAs (a
    // commit on `drain`), then the accumulators are freed.
    fence_before();
    __syncthreads();
    if (abort_flag) {
        if (warp == kProducerWarp && leader) {
            for (int s = 0; s < kIWSlots; ++s)
                if (last_round[s] >= 0) mbar_wait(smem_u32(&wfull[s]), last_round[s] & 1);
            if (w1_issued) mbar_wait(smem_u32(&w1full), 0u);
        } else if (warp == kXWarp && leader) {
            for (int s = 0; s < kTileSlots; ++s)
                if (x_last[s] >= 0) mbar_wait(smem_u32(&xfull[s]), static_cast<uint32_t>(x_last[s] & 1));
        } else if (warp == kMmaWarp && leader) {
            umma_commit(smem_u32(&drain));
            mbar_wait(smem_u32(&drain), 0);
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u)
                     : "memory");
    }
}

// ----------------------------------------------------------------------------
// Fused training pass: one CTA takes 128 rows of the minibatch through the
// gather, the three layers, the head, the backward layers and the three weight
// gradients of its rows (one split-K slab each), in one launch.  The slabs,
// dZ, H3 and dy go to global memory for the update kernel, which sums them in a
// fixed order.
//
// A step was 14 launches of 6-22 us, each reading back what the one before it
// had written and its transpose; here the activations stay in shared memory
// and serve twice: as the K-major A operand of the next layer (row = M), and
// untransposed as the MN-major operands of the weight gradients (row = K),
// which the 128-byte-swizzled layout [64-column block][row][64 columns] is as
// it stands.  Batch 8192 runs 64 CTAs, each a chain of ten short MMA jobs and
// as many epilogues: latency bounds it, not a pipe (45 us, and 16 us for the
// update; the 14 launches took 129 us a step, the same losses and weights).
//
// Global arrays of the pass are laid out by chunk, [tile][16-byte chunk of a
// row][128 rows], so that a warp's stores (one row per lane) are contiguous:
// as rows they touched 32 lines each, and the stores were half of the kernel.
//
// Shared memory: P and Q (64 KiB each) hold H1, H2; then D3 in P and D2, H1
// (read back from this thread's own global copy), D1 as their readers
// complete; a 2-slot ring of 32 KiB weight blocks; X (128 x 16) and W1 (256 x
// 16).  TMEM: two accumulators of 256 columns.
// Roles: warp 16 streams weights, warp 17
// issues MMAs, warps 0-15 gather and run the epilogues (the lane and column
// split of mlp_infer_kernel).  Job j's completion arrives on full[j],
// hand-overs to the MMA warp on blk and done; each barrier is used once, and
// every wait is bounded.
//
//   job  MMA                              epilogue after it
//   0    X W1^T          -> acc0          z1, h1 -> P
//   1    P W2^T          -> acc1          z2, h2 -> Q
//   2    Q W3^T          -> acc0          head, dy, dz3 -> P
//   3    P W3            -> acc1
//   4    dW3 rows 0-127  -> acc0          slab out
//   5    dW3 rows 128-   -> acc0          h1 -> P, slab out, then (job 3) dz2 -> Q
//   6    Q W2            -> acc0
//   7    dW2 rows 0-127  -> acc1          slab out
//   8    dW2 rows 128-   -> acc1          (with job 6) dz1 -> Q, slab out
//   9    dW1             -> acc0          slab out
//
// A layer's MMAs start per 64-column block as the epilogue before it writes the
// block (blk), into the accumulator that epilogue is not reading.
// ----------------------------------------------------------------------------
constexpr int kTrainEpiWarps = 16;
constexpr int kTrainThreads = (kTrainEpiWarps + 2) * 32;
constexpr int kTrainJobs = 10, kTrainDone = 3, kTrainBlocked = 4;
constexpr size_t kTrainSmem = 2 * kHBytes + kIWSlots * kWBlock + kW1Bytes + kXBytes + 1024;

// MN-major shared-memory descriptors: rows of 128 (32) swizzled bytes along
// MN, one per k; 8-row groups SBO apart, blocks of 64 (16) columns LBO apart.
__device__ __forceinline__ uint64_t desc_mn_sw128(uint32_t addr) {
    return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) |
           (static_cast<uint64_t>(kABytes >> 4) << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) |
           (static_cast<uint64_t>(1) << 46) | (static_cast<uint64_t>(2) << 61);
}
__device__ __forceinline__ uint64_t desc_mn_sw32(uint32_t addr) {
    return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>(1) << 16) |
           (static_cast<uint64_t>(256 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
           (static_cast<uint64_t>(6) << 61);
}
constexpr uint32_t kIdescMn = (1u << 15) | (1u << 16);  // A and B MN-major

// Sixteen values as two 16-byte chunks, `stride` chunks apart.
__device__ __forceinline__ void store16_bf16(uint4* d, int stride, const float (&v)[16]) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        __nv_bfloat162 p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = __floats2bfloat162_rn(v[q * 8 + 2 * j], v[q * 8 + 2 * j + 1]);
        d[q * stride] = *reinterpret_cast<uint4*>(p);
    }
}
__device__ __forceinline__ void load16_bf16(const uint4* s, int stride, float (&v)[16]) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const uint4 u = s[q * stride];
        const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 f = __bfloat1622float2(p[j]);
            v[q * 8 + 2 * j] = f.x;
            v[q * 8 + 2 * j + 1] = f.y;
        }
    }
}

__global__ void __launch_bounds__(kTrainThreads, 1)
    mlp_train_kernel(const __grid_constant__ TrainMaps maps, const TrainArgs a) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                               ~static_cast<uintptr_t>(1023));
    uint8_t* bufp = smem;
    uint8_t* bufq = smem + kHBytes;
    uint8_t* wbuf = smem + 2 * kHBytes;
    uint8_t* w1s = wbuf + kIWSlots * kWBlock;
    uint8_t* xs = w1s + kW1Bytes;
    __shared__ __align__(8) uint64_t w1full, xready, pready, drain;
    __shared__ __align__(8) uint64_t full[kTrainJobs], done[kTrainDone], blk[kTrainBlocked][4];
    __shared__ __align__(8) uint64_t wfull[kIWSlots], wempty[kIWSlots];
    __shared__ __align__(16) float sb1[kSurHidden], sb2[kSurHidden], sb3[kSurHidden], sw4[kSurHidden];
    __shared__ float part[4][kBM];
    __shared__ float starget[kBM];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.x;
    if (tid == 0) {
        mbar_init(smem_u32(&w1full), 1);
        mbar_init(smem_u32(&xready), kTrainEpiWarps);
        mbar_init(smem_u32(&pready), kTrainEpiWarps);
        mbar_init(smem_u32(&drain), 1);
        for (int j = 0; j < kTrainJobs; ++j) mbar_init(smem_u32(&full[j]), 1);
        for (int e = 0; e < kTrainDone; ++e) mbar_init(smem_u32(&done[e]), kTrainEpiWarps);
        for (int e = 0; e < kTrainBlocked * 4; ++e) mbar_init(smem_u32(&blk[e >> 2][e & 3]), kTrainEpiWarps);
        for (int s = 0; s < kIWSlots; ++s) {
            mbar_init(smem_u32(&wfull[s]), 1);
            mbar_init(smem_u32(&wempty[s]), 1);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // what the previous kernel of the stream wrote is read from here on
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
    if (tid < kSurHidden) {
        sb1[tid] = 0.5f * a.b1[tid];  // halved biases for silu_from_acc (exact)
        sb2[tid] = 0.5f * a.b2[tid];
        sb3[tid] = 0.5f * a.b3[tid];
        sw4[tid] = a.w4[tid];
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = tmem_slot;
    auto fail = [&](int code) {
        abort_flag = 1;
        atomicExch(a.err, code);
    };
    int last_round[kIWSlots] = {-1, -1};
    bool w1_issued = false;
    bool elected = false;

    if (warp == kTrainEpiWarps) {
        if (elect_one()) {
            elected = true;
            mbar_expect_tx(smem_u32(&w1full), kW1Bytes);
            tma_load_2d(smem_u32(w1s), &maps.w1, 0, 0, smem_u32(&w1full));
            w1_issued = true;
            const CUtensorMap* order[4] = {&maps.w2, &maps.w3, &maps.w3t, &maps.w2t};
            bool ok = true;
            for (uint32_t wl = 0; ok && wl < 16; ++wl) {
                const uint32_t s = wl % kIWSlots, round = wl / kIWSlots;
                if (abort_flag) break;
                if (round > 0) ok = mbar_wait(smem_u32(&wempty[s]), (round - 1) & 1);
                if (!ok) {
                    fail(32);
                    break;
                }
                mbar_expect_tx(smem_u32(&wfull[s]), kWBlock);
                tma_load_2d(smem_u32(wbuf + s * kWBlock), order[wl >> 2],
                            static_cast<int>(wl & 3) * kBK, 0, smem_u32(&wfull[s]));
                last_round[s] = static_cast<int>(round);
            }
        }
    } else if (warp == kTrainEpiWarps + 1) {
        if (elect_one()) {
            elected = true;
            constexpr uint32_t idesc = idesc_bf16<256>(), idesc_mn = idesc | kIdescMn;
            constexpr uint32_t idesc_w1 = idesc_bf16<16>() | kIdescMn;
            const uint32_t acc0 = tmem, acc1 = tmem + 256;
            uint32_t wc = 0;
            bool ok = true;
            auto wait = [&](uint64_t* bar) {
                ok = ok && !abort_flag && mbar_wait(smem_u32(bar), 0);
                fence_after();
            };
            auto commit = [&](int j) {
                if (ok) umma_commit(smem_u32(&full[j]));
            };
            // a layer: buf [128 x 256] times the next four ring blocks, each
            // block as epilogue e hands it over
            auto layer = [&](const uint8_t* buf, uint32_t acc, int e) {
                for (int kb = 0; ok && kb < 4; ++kb) {
                    const uint32_t s = wc % kIWSlots;
                    wait(&blk[e][kb]);
                    if (ok) ok = mbar_wait(smem_u32(&wfull[s]), (wc / kIWSlots) & 1);
                    if (!ok) return;
                    fence_after();
                    const uint32_t sa = smem_u32(buf + kb * kABytes), sb = smem_u32(wbuf + s * kWBlock);
#pragma unroll
                    for (int kk = 0; kk < kBK / 16; ++kk)
                        umma_bf16(acc, desc_sw128(sa + kk * 32), desc_sw128(sb + kk * 32), idesc,
                                  (kb | kk) != 0 ? 1u : 0u);
                    umma_commit(smem_u32(&wempty[s]));
                    ++wc;
                }
            };
            // 128 rows of a weight gradient: D's columns 128 half .. + 127 by
            // H's 256 columns, over the CTA's 128 batch rows
            auto grad = [&](const uint8_t* d, int half, const uint8_t* h, uint32_t acc) {
                if (!ok) return;
                const uint32_t da = smem_u32(d + half * 2 * kABytes), hb = smem_u32(h);
#pragma unroll
                for (int k = 0; k < kBM / 16; ++k)
                    umma_bf16(acc, desc_mn_sw128(da + k * 2048), desc_mn_sw128(hb + k * 2048),
                              idesc_mn, k != 0 ? 1u : 0u);
            };
            wait(&w1full);
            wait(&xready);
            if (ok) umma_bf16(acc0, desc_sw32(smem_u32(xs)), desc_sw32(smem_u32(w1s)), idesc, 0u);
            commit(0);
            layer(bufp, acc1, 0);
            commit(1);
            layer(bufq, acc0, 1);
            commit(2);
            layer(bufp, acc1, 2);
            commit(3);
            grad(bufp, 0, bufq, acc0);
            commit(4);
            wait(&done[0]);
            grad(bufp, 1, bufq, acc0);
            commit(5);
            layer(bufq, acc0, 3);
            commit(6);
            grad(bufq, 0, bufp, acc1);
            commit(7);
            wait(&done[1]);
            grad(bufq, 1, bufp, acc1);
            commit(8);
            wait(&done[2]);
            for (int half = 0; ok && half < 2; ++half) {
                const uint32_t da = smem_u32(bufq + half * 2 * kABytes), xb = smem_u32(xs);
#pragma unroll
                for (int k = 0; k < kBM / 16; ++k)
                    umma_bf16(acc0 + half * 16, desc_mn_sw128(da + k * 2048),
                              desc_mn_sw32(xb + k * 512), idesc_w1, k != 0 ? 1u : 0u);
            }
            commit(9);
            if (!ok) fail(34);
        }
    } else {
        const int q = warp & 3, g = warp >> 2;
        const int r = q * 32 + lane;
        const size_t row = static_cast<size_t>(tile) * kBM + r;
        const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
        const uint32_t acc0 = tmem + lane_off, acc1 = tmem + 256 + lane_off;
        bool ok = true;
        // lane 0 polls and broadcasts; then every lane observes the phase itself
        auto wait = [&](uint64_t* bar) {
            if (!ok) return;
            bool got = false;
            if (lane == 0) got = mbar_wait(smem_u32(bar), 0);
            got = __shfl_sync(0xFFFFFFFFu, got ? 1 : 0, 0) != 0;
            if (got) got = __all_sync(0xFFFFFFFFu, mbar_try(smem_u32(bar), 0)) != 0;
            if (!got && lane == 0) fail(36);
            ok = got;
            fence_after();
        };
        // shared stores to the tensor core's proxy, TMEM reads before the hand-off
        auto arrive = [&](uint64_t* bar) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(bar));
        };
        auto col = [&](int kb) { return kb * 64 + g * 16; };
        // this thread's 16 columns of block kb of an accumulator
        auto acc16 = [&](uint32_t acc, int c, float (&v)[16]) {
            uint32_t u[16];
            tmem_ld16_async(acc + c, u);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(u[j]);
        };
        // [tile][half][chunk of 4 columns][128 rows]
        auto slab_out = [&](uint32_t acc, float4* slab, int half) {
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                float v[16];
                acc16(acc, col(kb), v);
                float4* d = slab + (static_cast<size_t>(tile * 2 + half) * 64 + (col(kb) >> 2)) * kBM + r;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    d[i * kBM] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            }
        };
        // this thread's two 8-column chunks of block kb
        auto chunk = [&](uint4* x, int kb) {
            return x + (static_cast<size_t>(tile) * 32 + (col(kb) >> 3)) * kBM + r;
        };
        // a hidden layer's backward epilogue: acc and the stored z -> dz in
        // buf, handed over per block where `bars` is not null
        auto backward = [&](uint32_t acc, uint4* z_in, uint8_t* buf, uint4* d_out, uint64_t* bars) {
            uint4 raw[4][2];  // every block's z in flight at once
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                raw[kb][0] = chunk(z_in, kb)[0];
                raw[kb][1] = chunk(z_in, kb)[kBM];
            }
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                const int c = col(kb);
                float v[16], z[16];
                load16_bf16(raw[kb], 1, z);
                acc16(acc, c, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float s = sigmoidf_(z[j]);
                    v[j] = v[j] * s * (1.0f + z[j] * (1.0f - s));
                }
                store_h16_sw128(buf, r, c, v);
                if (bars) arrive(bars + kb);
                store16_bf16(chunk(d_out, kb), kBM, v);
            }
        };

        // gather the tile's rows (first 16 columns, 32-byte swizzle) and targets
        if (tid < 2 * kBM) {
            const int i = tid >> 1, ch = tid & 1;
            const int64_t at = static_cast<int64_t>(*a.step % *a.steps_per_epoch) * a.batch +
                               static_cast<int64_t>(tile) * kBM + i;
            const int64_t src = a.perm[at];
            const uint4 x = *reinterpret_cast<const uint4*>(a.xall + src * a.x_stride + ch * 8);
            *reinterpret_cast<uint4*>(xs + i * 32 + ((ch ^ ((i >> 2) & 1)) << 4)) = x;
            if (ch == 0) {
                const float t = a.tall[src];
                starget[i] = t;
                a.target_out[static_cast<size_t>(tile) * kBM + i] = t;
            }
        }
        arrive(&xready);

        // layers 1 and 2 forward
#pragma unroll 1
        for (int l = 0; l < 2; ++l) {
            wait(&full[l]);
            if (!ok) break;
            const float* bias = l == 0 ? sb1 : sb2;
            uint4* z_out = l == 0 ? a.z1 : a.z2;
            uint8_t* buf = l == 0 ? bufp : bufq;
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                const int c = col(kb);
                float v[16], z[16];
                acc16(l == 0 ? acc0 : acc1, c, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float hz, t;
                    v[j] = silu_from_acc(v[j], bias[c + j], hz, t);
                    z[j] = 2.0f * hz;  // exact: the pre-activation acc + bias
                }
                store_h16_sw128(buf, r, c, v);
                arrive(&blk[l][kb]);
                store16_bf16(chunk(z_out, kb), kBM, z);
                if (l == 0) store16_bf16(chunk(a.h1, kb), kBM, v);
            }
        }
        // head: partial chains per column group, y, dy; then dz3
        wait(&full[2]);
        if (ok) {
            float p = 0.0f;
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                const int c = col(kb);
                float v[16];
                acc16(acc0, c, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float hz, t;
                    const float h = silu_from_acc(v[j], sb3[c + j], hz, t);
                    p = fmaf(h, sw4[c + j], p);
                }
            }
            part[g][r] = p;
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&pready));
            wait(&pready);
        }
        if (ok) {
            const float y = (((part[0][r] + part[1][r]) + part[2][r]) + part[3][r]) + __ldg(a.b4);
            const float dy = a.loss_scale * (y - starget[r]);
            if (g == 0) {
                a.y_out[row] = y;
                a.dy_out[row] = dy;
            }
#pragma unroll 1
            for (int kb = 0; kb < 4; ++kb) {
                const int c = col(kb);
                float v[16], h[16];
                acc16(acc0, c, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    float hz, t;
                    h[j] = silu_from_acc(v[j], sb3[c + j], hz, t);
                    const float z = 2.0f * hz, s = fmaf(0.5f, t, 0.5f);
                    v[j] = dy * sw4[c + j] * s * (1.0f + z * (1.0f - s));
                }
                store_h16_sw128(bufp, r, c, v);
                arrive(&blk[2][kb]);
                store16_bf16(chunk(a.dz3, kb), kBM, v);
                store16_bf16(chunk(a.h3, kb), kBM, h);
            }
        }
        wait(&full[4]);
        if (ok) {
            slab_out(acc0, a.dw3, 0);
            arrive(&done[0]);
        }
        wait(&full[3]);
        wait(&full[5]);  // every reader of P and Q is done
        if (ok) {
            // this thread's own copy of H1, back into P
            uint4 h[4][2];
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                h[kb][0] = chunk(a.h1, kb)[0];
                h[kb][1] = chunk(a.h1, kb)[kBM];
            }
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                const int c = col(kb), c0 = (c & 63) >> 3;
                uint8_t* d = bufp + (c >> 6) * kABytes + r * 128;
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    *reinterpret_cast<uint4*>(d + (((c0 + i) ^ (r & 7)) << 4)) = h[kb][i];
            }
            slab_out(acc0, a.dw3, 1);
            backward(acc1, a.z2, bufq, a.dz2, blk[3]);
        }
        wait(&full[7]);
        if (ok) {
            slab_out(acc1, a.dw2, 0);
            arrive(&done[1]);
        }
        wait(&full[6]);
        wait(&full[8]);
        if (ok) {
            backward(acc0, a.z1, bufq, a.dz1, nullptr);
            arrive(&done[2]);
            slab_out(acc1, a.dw2, 1);
        }
        wait(&full[9]);
        if (ok && g < 2) {  // group g takes rows 128 g .. of dW1, 16 columns
            float v[16];
            acc16(acc0, g * 16, v);
            float4* d = a.dw1 + static_cast<size_t>(tile * 2 + g) * 4 * kBM + r;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                d[i * kBM] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
    }

    // Teardown, as in mlp_infer_kernel.
    fence_before();
    __syncthreads();
    if (abort_flag) {
        if (warp == kTrainEpiWarps && elected) {
            for (int s = 0; s < kIWSlots; ++s)
                if (last_round[s] >= 0) mbar_wait(smem_u32(&wfull[s]), last_round[s] & 1);
            if (w1_issued) mbar_wait(smem_u32(&w1full), 0u);
        } else if (warp == kTrainEpiWarps + 1 && elected) {
            umma_commit(smem_u32(&drain));
            mbar_wait(smem_u32(&drain), 0);
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u)
                     : "memory");
    }
}

template <int BN, int EPI>
cudaError_t launch_t(const CUtensorMap& ta, const CUtensorMap& tb, const GemmArgs& a, int splits,
                     cudaStream_t st) {
    constexpr size_t smem = kStages * (kABytes + BN * kBK * 2) + 1024;
    static DeviceOnce once;
    const cudaError_t attr_err = allow_shared(once, umma_gemm_kernel<BN, EPI>, smem);
    if (attr_err != cudaSuccess) return attr_err;
    dim3 grid((a.M + kBM - 1) / kBM, a.N / BN, splits);
    umma_gemm_kernel<BN, EPI><<<grid, kGemmThreads, smem, st>>>(ta, tb, a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_mlp_infer(const CUtensorMap& tx, const CUtensorMap& tw1, const CUtensorMap& tw2,
                             const CUtensorMap& tw3, const InferArgs& a, int ctas, cudaStream_t st) {
    static DeviceOnce once;
    const cudaError_t attr_err = allow_shared(once, mlp_infer_kernel, kInferSmem);
    if (attr_err != cudaSuccess) return attr_err;
    if (a.n <= 0) return cudaSuccess;
    const int64_t tiles = (a.n + kBM - 1) / kBM;
    const int grid = static_cast<int>(tiles < ctas ? tiles : ctas);
    mlp_infer_kernel<<<grid, kInferThreads, kInferSmem, st>>>(tx, tw1, tw2, tw3, a);
    return cudaGetLastError();
}

cudaError_t launch_mlp_train(const TrainMaps& maps, const TrainArgs& a, cudaStream_t st) {
    static DeviceOnce once;
    const cudaError_t attr_err = allow_shared(once, mlp_train_kernel, kTrainSmem);
    if (attr_err != cudaSuccess) return attr_err;
    if (a.batch <= 0 || a.batch % kBM != 0) return cudaErrorInvalidValue;
    return launch_dependent(mlp_train_kernel, a.batch / kBM, kTrainThreads, kTrainSmem, st, maps, a);
}

bool make_tmap_bf16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols,
                    uint32_t box_rows) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    });
    if (!encode) return false;
    // Host-side checks of the TMA rules: 16-byte aligned base, row stride a
    // multiple of 16 bytes, a 64-element (128-byte) inner box.
    if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (cols * 2) % 16 != 0 || cols < 64) return false;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool make_tmap_bf16_k16(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols,
                        uint32_t box_rows) {
    if (!make_tmap_bf16(map, base, rows, cols, box_rows)) return false;  // also loads the encoder
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    });
    if (!encode || box_rows == 0 || box_rows > 256) return false;
    // 16 bf16 = 32 bytes: the inner box equals the 32-byte swizzle span
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {16, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t launch_umma_gemm(int epi, int bn, const CUtensorMap& ta, const CUtensorMap& tb,
                             const GemmArgs& a, int splits, cudaStream_t st) {
    if (a.K % kBK != 0 || a.k_per_split % kBK != 0 || a.N % bn != 0 || splits < 1)
        return cudaErrorInvalidValue;
    switch (bn) {
        case 64:
            if (epi == kEpiF32) return launch_t<64, kEpiF32>(ta, tb, a, splits, st);
            break;
        case 128:
            if (epi == kEpiF32) return launch_t<128, kEpiF32>(ta, tb, a, splits, st);
            if (epi == kEpiFwd) return launch_t<128, kEpiFwd>(ta, tb, a, splits, st);
            break;
        case 256:
            if (epi == kEpiF32) return launch_t<256, kEpiF32>(ta, tb, a, splits, st);
            if (epi == kEpiFwd) return launch_t<256, kEpiFwd>(ta, tb, a, splits, st);
            if (epi == kEpiLast) return launch_t<256, kEpiLast>(ta, tb, a, splits, st);
            break;
        default:
            break;
    }
    return cudaErrorInvalidValue;
}

}  // namespace qkb
