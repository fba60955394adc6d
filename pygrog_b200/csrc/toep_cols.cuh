// toep_cols.cuh -- column passes of the 2-D Toeplitz normal operator
// (toep_cols.cu, toep_sub_cols.cu), launched by toep_fft.cu.
#pragma once

#include "fft_core.cuh"

namespace pgb {
namespace fft {

// Components of the subspace form: a block has F::T x 4 threads for each. 5 of
// them (640 threads at most) leave 96 registers a thread and next to no spills
// (12 to 24 bytes at L = 800, 960 and 1024). Built for 8 (64 registers, 0.4 to
// 2.5 KB spilled at L = 384 and more) the smaller ranks pay: 8 coils, L = 384,
// image 192 x 192, an application of 4 components 51 -> 96 us, of 5 72 -> 126
// (cuFFT: 182, 183).
constexpr int kSubMax = 5;

// The column transforms, the PSF and their inverse in place on the planes U
// (BC, n0, L1); PGB_ERR_UNSUPPORTED if the length L0 is not built.
int toep_cols(float2* U, const float* psf, int64_t BC, int n0, int L1, int L0, const float2* tw, cudaStream_t s);
// The same for K components, U (frames, K, C, n0, L1), BC = frames * C.
int toep_sub_cols(float2* U, const float* psf, int64_t BC, int C, int K, int n0, int L1, int L0, const float2* tw,
                  cudaStream_t s);

}  // namespace fft
}  // namespace pgb
