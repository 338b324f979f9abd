// Plane transforms of lengths that are not powers of two (fft_mr_impl.cuh).
#pragma once
#include "tg_common.cuh"

namespace tg {

constexpr int kMrMaxLength = 512;

// The lengths compiled: even, prime factors up to 7, not a power of two, at
// least two radices (so that the last pass follows a first).  Odd lengths,
// larger prime factors and lengths above 512 run the general kernels of fft.cu,
// which are several times slower (forward and backward, 300 planes FP32: 225x225
// 824 us, 224x224 95; 60 planes: 540x540 858, 500x500 170).  Nothing in the
// passes needs an even length: each length adds ten kernels, about 230 KB of
// library and some four seconds of compilation, and the 64 here are those that grids
// of spectral cases use.
constexpr bool mr_length(int L) {
  if (L < 18 || L > kMrMaxLength || L % 2 != 0 || (L & (L - 1)) == 0) return false;
  int n = L;
  for (int q = 2; q <= 7; ++q)
    while (n % q == 0) n /= q;
  return n == 1;
}

// The passes of dft_forward / dft_backward / dft_backward_adv; each returns
// false, with nothing launched, when its length is not one of these.
template <typename T>
bool mr_forward_x(const TransformDims& d, const FftPlan& px, const T* phys, void* work, int planes, cudaStream_t s,
                  const PhysProduct* prod);
template <typename T>
bool mr_forward_y(const TransformDims& d, const FftPlan& py, const void* work, double2* spec, int planes, double scale,
                  cudaStream_t s);
template <typename T>
bool mr_backward_y(const TransformDims& d, const FftPlan& py, const double2* spec, void* work, int planes,
                   cudaStream_t s, const SpecGather* gather);
template <typename T>
bool mr_backward_x(const TransformDims& d, const FftPlan& px, const void* work, T* phys, int planes, cudaStream_t s);
template <typename T>
bool mr_backward_adv(const TransformDims& d, const FftPlan& px, const void* work, const T* unl, T* out, int ncomp,
                     double su, double sv, double sw, cudaStream_t s);

}  // namespace tg
