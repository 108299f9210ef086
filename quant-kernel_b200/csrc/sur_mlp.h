// sur_mlp.h -- the Heston price surrogate: MLP 9 -> 256 -> 256 -> 256 -> 1,
// SiLU, BF16 weights/activations, FP32 accumulation, FP32 master weights and
// Adam moments, trained and evaluated on the GPU with the tcgen05 GEMM.
//
// The network learns a residual: price / S = base(f) + MLP(normalised f),
// with base the Black-Scholes call / S at the Heston model's mean variance
// over [0, T] (see sur_base).  The base carries the bulk of the price
// surface, so the network's absolute error shrinks with the residual's scale.
#pragma once

#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <vector>

namespace qkb {

constexpr int kSurIn = 9;        // S/K, T, r, q, v0, kappa, theta, sigma, rho
constexpr int kSurInPad = 64;    // layer-1 K, zero-padded for the 64-wide k-block
constexpr int kSurHid = 256;
// Base of the residual (stored in checkpoints).
enum : int32_t { kSurBaseNone = 0, kSurBaseBsmMeanVar = 1 };

constexpr int kSurParams = kSurHid * kSurIn + kSurHid + 2 * (kSurHid * kSurHid + kSurHid) +
                           kSurHid + 1;  // 134,401 trainable values

// Internal flat layout of the FP32 master copy (W1 keeps its zero padding).
struct SurLayout {
    static constexpr int W1 = 0;
    static constexpr int b1 = W1 + kSurHid * kSurInPad;
    static constexpr int W2 = b1 + kSurHid;
    static constexpr int b2 = W2 + kSurHid * kSurHid;
    static constexpr int W3 = b2 + kSurHid;
    static constexpr int b3 = W3 + kSurHid * kSurHid;
    static constexpr int w4 = b3 + kSurHid;
    static constexpr int b4 = w4 + kSurHid;
    static constexpr int total = b4 + 4;  // padded to 16 bytes
};

// Training state on the device, read by a step's kernels: the launches of a
// call are alike, the step counter and the schedule advance here.
struct SurState {
    int step;          // completed optimiser steps
    int total_steps;   // cosine schedule length
    int steps_per_epoch;
    int batch;
    float lr0, beta1, beta2, eps;
    int err;           // error word of the training and device-inference kernels
    int step_begin;    // first step of the current schedule
    int pad[2];
};

struct SurBox {
    double lo[kSurIn];
    double hi[kSurIn];
};

// Options that the network does not price: their places and inputs.
struct SurOutside {
    std::vector<int32_t> index, option_type;
    std::vector<double> cols[10];
};

class SurModel {
public:
    SurModel() = default;
    ~SurModel();
    SurModel(const SurModel&) = delete;
    SurModel& operator=(const SurModel&) = delete;

    cudaError_t init(uint64_t seed, const SurBox& box);
    // Raw features (n x 9, the order of kSurIn) -> normalised bf16 rows.
    void normalise(const double* features, int64_t n, __nv_bfloat16* out_rows) const;
    // The residual's base (price / S, FP64 rounded to FP32) for each row; 0
    // for a model without one.
    void base_host(const double* features, int64_t n, float* out_base) const;
    // Device features (n x 9 FP64, DEVICE) -> normalised rows and base (DEVICE),
    // the same values as normalise and base_host, asynchronous on st.
    cudaError_t features_device(const double* features, int64_t n, __nv_bfloat16* rows,
                                float* base, cudaStream_t st);
    int32_t base_kind() const { return base_kind_; }

    cudaError_t set_dataset(const double* features, const double* target, int64_t n);
    cudaError_t train(int epochs, int batch, float lr0, uint64_t shuffle_seed, float* out_loss_last,
                      float* out_epoch_loss);
    // price / spot of calls for raw features, host in and out.
    cudaError_t predict(const double* features, int64_t n, double* out);
    // The host pricing call: columns spot, strike, t, r, q, v0, kappa, theta,
    // sigma, rho and option_type, n each.  route[i] (route may be null): 0 priced
    // by the network, 1 outside the box (out[i] is NaN), 2 decided by the entry
    // checks.  The options outside are copied to `outside` before anything is
    // written: out and route may be the caller's input columns.
    cudaError_t price_quotes(const double* const (&cols)[10], const int32_t* option_type, int64_t n,
                             double* out, int32_t* route, SurOutside* outside);
    // Device-resident inference on normalised bf16 rows [n][64] plus the
    // rows' base (required when base_kind() != kSurBaseNone): the fused kernel
    // (all three layers per 128-row tile in one persistent launch), or with
    // layered = true the layer-by-layer GEMMs it is tested against.
    cudaError_t predict_device(const __nv_bfloat16* x_rows, const float* base, int64_t n, float* y,
                               cudaStream_t st, bool layered = false);
    // One forward + backward without an update: loss and the 134,401 gradients.
    cudaError_t gradients(const double* features, const double* target, int n, double* grads,
                          double* loss);
    cudaError_t parameters(double* out) const;            // canonical order, 134,401
    cudaError_t set_parameters(const double* in);
    cudaError_t save(const char* path);
    cudaError_t load(const char* path);
    const SurBox& box() const { return box_; }
    int device() const { return device_; }
    int steps_done() const;
    // The error code a tensor-core kernel of the last failed call recorded (a
    // call that finds one returns cudaErrorLaunchTimeout), cleared by reading; 0
    // if none.
    int take_pipeline_code();

private:
    cudaError_t network(const __nv_bfloat16* x_rows, const float* base, int64_t n, float* y, int* err,
                        cudaStream_t st, bool layered);
    cudaError_t arm_timeout(int* err);
    cudaError_t ensure_batch_buffers(int batch);
    cudaError_t ensure_predict_buffers(int64_t rows, size_t in_row);
    cudaError_t ensure_layered_buffers(int64_t rows);
    template <class Fill, class Enqueue, class Drain>
    cudaError_t run_chunked(int64_t n, size_t in_row, size_t out_row, const Fill& fill,
                            const Enqueue& enqueue, const Drain& drain);
    struct StepLaunch;  // the arguments of a step's two kernels
    cudaError_t prepare_steps(bool update, StepLaunch* s);
    cudaError_t run_step(const StepLaunch& s, cudaStream_t st);
    cudaError_t refresh_bf16(cudaStream_t st);

    int device_ = -1;
    cudaStream_t stream_ = nullptr;
    cudaEvent_t uploaded_ = nullptr;  // an epoch's permutation has left the host
    SurBox box_{};
    int32_t base_kind_ = kSurBaseBsmMeanVar;
    // parameters, Adam moments, gradient
    float* P_ = nullptr;
    float* M_ = nullptr;
    float* V_ = nullptr;
    float* G_ = nullptr;
    __nv_bfloat16 *W1b_ = nullptr, *W2b_ = nullptr, *W3b_ = nullptr, *W2Tb_ = nullptr, *W3Tb_ = nullptr;
    SurState* state_ = nullptr;  // device
    // dataset
    __nv_bfloat16* Xall_ = nullptr;
    float* Tall_ = nullptr;
    int32_t* perm_ = nullptr;
    int64_t n_data_ = 0;
    // training batch buffers
    int batch_ = 0;
    float* Tb_ = nullptr;
    __nv_bfloat16 *Z1_ = nullptr, *H1_ = nullptr, *Z2_ = nullptr, *H3_ = nullptr;
    __nv_bfloat16 *dZ3_ = nullptr, *dZ2_ = nullptr, *dZ1_ = nullptr;
    float *y_ = nullptr, *dy_ = nullptr;
    float *dW1p_ = nullptr, *dW2p_ = nullptr, *dW3p_ = nullptr;
    unsigned* blocks_done_ = nullptr;  // update_kernel's block counter
    float* loss_hist_ = nullptr;
    int loss_cap_ = 0;
    // inference buffers
    int64_t pred_rows_ = 0;
    int sm_count_ = 0;
    __nv_bfloat16 *PX_ = nullptr, *PH1_ = nullptr, *PH2_ = nullptr;
    // a chunk's error word and, kOutHead bytes on, its outputs: one copy to the host
    int* Perr_ = nullptr;
    float* Py_ = nullptr;
    float* Pbase_ = nullptr;
    int pipeline_code_ = 0;
    // host calls: device room for one chunk's inputs
    double* d_in_ = nullptr;
    size_t d_in_bytes_ = 0;
    int64_t layered_rows_ = 0;
};

}  // namespace qkb
