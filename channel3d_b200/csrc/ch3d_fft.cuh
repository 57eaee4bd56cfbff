// ch3d_fft.cuh -- launchers of the generic-length Poisson transforms
// (ch3d_fft.cu); fft_generic_setup(...) once before the first launch.
#pragma once
#include "ch3d_dev.cuh"

namespace ch3d {

struct XShape {
  int LPB, LP, sh, threads;  // lines per block, padded line length, padding shift
  size_t smem;
};

// FP64 x plans stop at this radix, a pass more for some lengths but half the registers:
// 96 points as 4 x 4 x 6 76 us, as 8 x 12 82 us (192^3, forward); z transforms, whose
// passes move more between them, gain nothing (192 points as 12 x 16 34 us, as 4 x 6 x 8 43).
constexpr int kXRadix64 = 9;

cudaError_t fft_generic_setup(int device, bool fp32, const FFTPlanDev& planz);
size_t fft_generic_smem(const FFTPlanDev& planx, const FFTPlanDev& planz);
// mode: 0 div(u*)/pmAlpha of (a, b, c), 1 div(u), 2 source in a, 4 field in a
template <class T>
cudaError_t xfft_generic(const Geo<T>& g, const Metrics<T>& m, const T* a, const T* b, const T* c,
                         typename CplxOf<T>::type* spec, const FFTPlanDev& pl, const typename CplxOf<T>::type* tw,
                         const typename CplxOf<T>::type* twr, int mode, DevScalars* sc, T* pr, cudaStream_t st);
template <class T>
cudaError_t zfft_generic(const Geo<T>& g, typename CplxOf<T>::type* spec, const FFTPlanDev& pl,
                         const typename CplxOf<T>::type* tw, int inverse, const DevScalars* sc, cudaStream_t st);
template <class T>
cudaError_t xifft_generic(const Geo<T>& g, const typename CplxOf<T>::type* spec, T* phi, const FFTPlanDev& pl,
                          const typename CplxOf<T>::type* tw, const typename CplxOf<T>::type* twr, T normfft,
                          const DevScalars* sc, cudaStream_t st);

}  // namespace ch3d
