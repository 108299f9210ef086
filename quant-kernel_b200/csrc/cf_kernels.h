// cf_kernels.h -- host interface of the batch Heston Fourier pricers: the
// characteristic-function price with Gauss-Legendre P1/P2 integration and the
// Fang-Oosterlee COS expansion (FP64).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace qkb {

enum class FourierMethod { kCf, kCos };

// The caller's columns, n values each.  f64: spot, strike, t, r, q, v0, kappa,
// theta, sigma, rho, and the integration limit (CF) or truncation width (COS);
// count: integration steps (CF) or terms (COS).
constexpr int kFourierF64 = 11;
struct FourierColumns {
    const double* f64[kFourierF64];
    const int32_t* option_type;
    const int32_t* count;
};

// Host columns in, host prices out: stages through the calling thread's pinned
// and device buffers on its own streams and waits for the result.  The
// reference's entry checks (heston.cpp:10-24, cos_method.cpp:38-53) run on the
// device; an option they decide gets NaN or its intrinsic value.
cudaError_t heston_fourier_price_host(FourierMethod method, const FourierColumns& c, int32_t n,
                                      double* out);

}  // namespace qkb
