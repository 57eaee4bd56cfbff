// ch3d_fft.cu -- the Poisson transforms for line lengths without a
// register-resident plan (ch3d_rfft.cu), any product of 2 and 3, with the
// shared-memory passes of fft.cuh:
//   k_xfft_g   clcPrSrcOther (src/CFD_2nd/m_TScheme.f90:213-241) fused with the
//              forward x R2C transform (m_Poisson.f90:241-333, R2HC)
//   k_zfft_g   z transform of the spectrum, in place
//   k_xifft_g  inverse x C2R transform * normfft -> phi (m_Poisson.f90:1194-1200)
// The first pass forms or loads its points in registers and the last one
// stores them (k_xfft_g: after the real-to-complex split), so global memory is
// touched once and shared memory only between passes.  At 192^3 in FP64 the
// forward x transform takes 76 us (102 with radix 2 and 3 passes), z 34 each (55),
// the inverse x 35 (50), for 0.23, 0.11 and 0.11 GB: latency at 16 to 24 warps per
// SM, part of it the fetch of the unrolled butterflies' code.
#include "ch3d_fft.cuh"
#include <type_traits>

namespace ch3d {

// Position of point n of a line in shared memory: one gap per 2^sh points
// (against bank conflicts of the first pass's strided stores), none with sh = 31.
__device__ __forceinline__ int xpad(int n, int sh) { return n + (n >> sh); }

// The source of the forward transform, packed as z_n = src_2n + i src_2n+1:
// div(u)/pmAlpha (modes 0, 1), with its largest magnitude in dmax.
// SRC: 0 2nd-order divergence, 1 4th-order divergence, 2 the source (mode 2) or a
// field (mode 4) as it stands in the first array.
template <class T, int SRC> struct XSource {
  typedef typename CplxOf<T>::type CT;
  const Geo<T>& g;
  const Metrics<T>& m;
  const T* __restrict__ ux;
  const T* __restrict__ uy;
  const T* __restrict__ uz;
  T* __restrict__ pr;
  int mode;
  T sudtal;
  double dmax;
  // point n of line j + ny k
  __device__ __forceinline__ CT operator()(int line, int n) {
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const T rdx = g.rdx, rdz = g.rdz;
    const long long base = (long long)nx * line;
    const int i0 = 2 * n;
    T r0, r1;
    if constexpr (SRC == 2) {
      const CT s01 = __ldg(reinterpret_cast<const CT*>(ux + base + i0));  // (i0, i0+1): nx and i0 even
      r0 = s01.x; r1 = s01.y;
    } else {
      const int k = line / ny, j = line - k * ny;
      const T sucaj = m.rdyp[j + 1];
      if constexpr (SRC == 1) {
        const C4<T> c4(g);
        T d[2];
        div4_pair(g, c4, sucaj, ux, uy, uz, base, i0, j, k, d);
        r0 = d[0]; r1 = d[1];
      } else {
        const int i2 = i0 + 2 == nx ? 0 : i0 + 2;
        const long long basep = k + 1 == nz ? base - (long long)nx * ny * (nz - 1) : base + (long long)nx * ny;
        const CT u01 = __ldg(reinterpret_cast<const CT*>(ux + base + i0));
        const T u2 = __ldg(ux + base + i2);
        const CT v01 = __ldg(reinterpret_cast<const CT*>(uy + base + i0));
        // uy at j+1: the next row, above the top row the wall value or, periodic in y, row 0
        const CT v01p = j + 1 < ny ? __ldg(reinterpret_cast<const CT*>(uy + base + nx + i0))
                        : (g.bc.hi == 0 ? __ldg(reinterpret_cast<const CT*>(uy + base - (long long)(ny - 1) * nx + i0))
                                        : mk((T)g.bc.uy_hi, (T)g.bc.uy_hi));
        const CT w01 = __ldg(reinterpret_cast<const CT*>(uz + base + i0));
        const CT w01p = __ldg(reinterpret_cast<const CT*>(uz + basep + i0));
        r0 = (u01.y - u01.x) * rdx + (v01p.x - v01.x) * sucaj + (w01p.x - w01.x) * rdz;
        r1 = (u2 - u01.y) * rdx + (v01p.y - v01.y) * sucaj + (w01p.y - w01.y) * rdz;
        if (mode == 0 && g.implicit == 2) {  // clcPrSrc_FIMP: pressure += -xnu/2 div (m_TScheme.f90:271)
          const T xnuhm = -(T)0.5 * g.xnu;
          CT* p01 = reinterpret_cast<CT*>(pr + base + i0);
          const CT p = *p01;
          *p01 = mk(p.x + xnuhm * r0, p.y + xnuhm * r1);
        }
      }
    }
    dmax = fmax(dmax, fmax(fabs((double)r0), fabs((double)r1)));
    return mk(sudtal * r0, sudtal * r1);
  }
  // the block's largest |div| into sc->divmax1 (modes 0 to 2)
  __device__ __forceinline__ void finish(DevScalars* sc) {
    if (mode == 4) return;
    __shared__ double wred[16];
    for (int o = 16; o > 0; o >>= 1) dmax = fmax(dmax, __shfl_xor_sync(0xffffffffu, dmax, o));
    if ((threadIdx.x & 31) == 0) wred[threadIdx.x >> 5] = dmax;
    __syncthreads();
    if (threadIdx.x == 0) {
      double v = wred[0];
      for (int w = 1; w < (int)blockDim.x / 32; ++w) v = fmax(v, wred[w]);
      atomic_max_nonneg(&sc->divmax1, v);
    }
  }
};

// real-to-complex split of a line Z (0..M-1): X_k = (Z_k + conj Z_{M-k})/2 - i W_nx^k (Z_k - conj Z_{M-k})/2, k = 0..M
template <class CT> __device__ __forceinline__ CT r2c_split(CT a, CT zb, CT w) {
  const auto hf = a.x * 0 + (decltype(a.x))0.5;
  const CT b = cconj(zb);
  const CT e = mk(hf * (a.x + b.x), hf * (a.y + b.y));
  const CT dd = csub(a, b);
  const CT o = mk(hf * dd.y, -hf * dd.x);  // (a-b)/(2i)
  return cadd(e, cmul(w, o));
}
// and its inverse: Z_k = e + i o, conjugated for the forward-transform-based inverse
template <class CT> __device__ __forceinline__ CT c2r_unsplit(CT a, CT xb, CT w) {
  const CT b = cconj(xb);
  const CT e = cadd(a, b);
  const CT o = cmul(csub(a, b), cconj(w));
  return cconj(mk(e.x - o.y, e.y + o.x));
}

// Forward x transform of LPB lines per block.  FP64 forms the source of all lines in
// shared memory first: in the first pass's registers, next to the butterfly, it took
// 138 of them (12 warps per SM; 109 us at 192^3, now 76).  FP32 forms it there (80
// registers; 96 x 65 x 54 step 143 us, 148 with the source first).
template <class T, int SRC, int MAXR>
__global__ void __launch_bounds__(256) k_xfft_g(Geo<T> g, Metrics<T> m, const T* __restrict__ ux,
                                                const T* __restrict__ uy, const T* __restrict__ uz,
                                                typename CplxOf<T>::type* __restrict__ spec, FFTPlanDev pl,
                                                const typename CplxOf<T>::type* __restrict__ tw,
                                                const typename CplxOf<T>::type* __restrict__ twr, int LPB, int LP, int sh,
                                                unsigned long long mM, unsigned long long mM1, int mode,
                                                DevScalars* __restrict__ sc,
                                                T* __restrict__ pr) {
  typedef typename CplxOf<T>::type CT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (sc->status) return;
  const int M = g.nx / 2, nxh = g.nxh;
  const int line0 = blockIdx.x * LPB;
  const int nl = min(LPB, g.ny * g.nz - line0);
  CT* src = (CT*)smem_raw;
  CT* dst = src + (size_t)LPB * LP;
  XSource<T, SRC> form{g, m, ux, uy, uz, pr, mode, mode == 0 ? (T)(1.0 / sc->pmAlpha) : (T)1, 0.0};
  int p = 0;
  if constexpr (SRC == 2 || sizeof(T) == 4) {
    p = 1;
    fft_pass<CT, false, MAXR>(pl, 0, nl, 0ull, tw, [&](int l, int n) { return form(line0 + l, n); },
                              [&](int l, int n, CT v) { src[l * LP + xpad(n, sh)] = v; });
  } else {
#pragma unroll 2
    for (int t = threadIdx.x; t < nl * M; t += blockDim.x) {
      const int l = fdiv(t, mM), n = t - l * M;
      src[l * LP + xpad(n, sh)] = form(line0 + l, n);
    }
  }
  __syncthreads();
  for (; p < pl.npass; ++p) {
    fft_pass<CT, false, MAXR>(pl, p, nl, 0ull, tw, [&](int l, int n) { return src[l * LP + xpad(n, sh)]; },
                        [&](int l, int n, CT v) { dst[l * LP + xpad(n, sh)] = v; });
    __syncthreads();
    CT* t = src; src = dst; dst = t;
  }
  for (int t = threadIdx.x; t < nl * (M + 1); t += blockDim.x) {
    const int l = fdiv(t, mM1), kk = t - l * (M + 1);
    spec[(long long)nxh * (line0 + l) + kk] = r2c_split(src[l * LP + xpad(kk == M ? 0 : kk, sh)],
                                                        src[l * LP + xpad(kk == 0 ? 0 : M - kk, sh)], __ldg(twr + kk));
  }
  form.finish(sc);
}

// z transform of the spectrum, in place: layout (kx, j, kz), lines over kz.
// Block = up to TKX consecutive kx at one j; point n of line l at n * TKX + l.
template <class T, int MAXR>
__global__ void __launch_bounds__(256) k_zfft_g(Geo<T> g, typename CplxOf<T>::type* __restrict__ spec, FFTPlanDev pl,
                                                const typename CplxOf<T>::type* __restrict__ tw, int TKX,
                                                unsigned long long mT, unsigned long long mTail, int inverse,
                                                const DevScalars* __restrict__ sc) {
  typedef typename CplxOf<T>::type CT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (sc->status) return;
  const int nz = g.nz, nxh = g.nxh;
  const int kx0 = blockIdx.x * TKX, nl = min(TKX, nxh - kx0);
  const long long zs = (long long)nxh * g.ny;
  CT* const col = spec + kx0 + (long long)nxh * blockIdx.y;
  CT* src = (CT*)smem_raw;
  CT* dst = src + (size_t)TKX * nz;  // used from three passes on
  const unsigned long long mL = nl == TKX ? mT : mTail;
  auto ldg = [&](int l, int n) { const CT v = col[zs * n + l]; return inverse ? cconj(v) : v; };
  auto stg = [&](int l, int n, CT v) { col[zs * n + l] = inverse ? cconj(v) : v; };
  auto lds = [&](int l, int n) { return src[n * TKX + l]; };
  const int last = pl.npass - 1;
  if (last == 0) {
    fft_pass<CT, true, MAXR>(pl, 0, nl, mL, tw, ldg, stg);
    return;
  }
  fft_pass<CT, true, MAXR>(pl, 0, nl, mL, tw, ldg, [&](int l, int n, CT v) { src[n * TKX + l] = v; });
  __syncthreads();
  for (int p = 1; p < last; ++p) {
    fft_pass<CT, true, MAXR>(pl, p, nl, mL, tw, lds, [&](int l, int n, CT v) { dst[n * TKX + l] = v; });
    __syncthreads();
    CT* t = src; src = dst; dst = t;
  }
  fft_pass<CT, true, MAXR>(pl, last, nl, mL, tw, lds, stg);
}

// inverse x transform (complex-to-real, unnormalised as FFTW's HC2R) * normfft -> phi
template <class T, int MAXR>
__global__ void __launch_bounds__(256) k_xifft_g(Geo<T> g, const typename CplxOf<T>::type* __restrict__ spec,
                                                 T* __restrict__ phi, FFTPlanDev pl,
                                                 const typename CplxOf<T>::type* __restrict__ tw,
                                                 const typename CplxOf<T>::type* __restrict__ twr, int LPB, int LP,
                                                 int sh, T normfft, const DevScalars* __restrict__ sc) {
  typedef typename CplxOf<T>::type CT;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (sc->status) return;
  const int nx = g.nx, M = nx / 2, nxh = g.nxh;
  const int nlines = g.ny * g.nz;
  const int line0 = blockIdx.x * LPB;
  const int nl = min(LPB, nlines - line0);
  CT* src = (CT*)smem_raw;
  CT* dst = src + (size_t)LPB * LP;
  auto unsplit = [&](int l, int kk) {
    const CT* X = spec + (long long)nxh * (line0 + l);
    return c2r_unsplit(X[kk], X[M - kk], __ldg(twr + kk));
  };
  auto out = [&](int l, int n, CT v) {
    reinterpret_cast<CT*>(phi + (long long)nx * (line0 + l))[n] = mk(v.x * normfft, -v.y * normfft);
  };
  auto lds = [&](int l, int n) { return src[l * LP + xpad(n, sh)]; };
  const int last = pl.npass - 1;
  if (last == 0) {
    fft_pass<CT, false, MAXR>(pl, 0, nl, 0ull, tw, unsplit, out);
    return;
  }
  fft_pass<CT, false, MAXR>(pl, 0, nl, 0ull, tw, unsplit, [&](int l, int n, CT v) { src[l * LP + xpad(n, sh)] = v; });
  __syncthreads();
  for (int p = 1; p < last; ++p) {
    fft_pass<CT, false, MAXR>(pl, p, nl, 0ull, tw, lds, [&](int l, int n, CT v) { dst[l * LP + xpad(n, sh)] = v; });
    __syncthreads();
    CT* t = src; src = dst; dst = t;
  }
  fft_pass<CT, false, MAXR>(pl, last, nl, 0ull, tw, lds, out);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
constexpr int kFftSmemLimit = 200 * 1024;

// Radices compiled in.  FP64 kernels up to radix 9 have 72 to 74 registers, those with
// the 12- and 16-point butterflies 118 to 128 (64^3 step 145 / 141 us): x plans stop at
// 9, and z plans up to 9 have kernels of their own.  In FP32 (44 / 64) the smaller ones
// were no faster (96 x 65 x 54 143 / 146).
template <class T> constexpr int x_radices() { return sizeof(T) == 8 ? kXRadix64 : 16; }
template <class T, class F> static void with_z_radices(const FFTPlanDev& pl, F go) {
  if constexpr (sizeof(T) == 8)
    if (pl.npass == 0 || pl.radix[pl.npass - 1] <= 9) return go(std::integral_constant<int, 9>{});  // radices ascend
  go(std::integral_constant<int, 16>{});
}
// Shared-memory limits of the kernels that transforms with these plans use, each once
// per process and device (setting one loads the kernel).
template <class T> static cudaError_t setup_t(int device, const FFTPlanDev& planz) {
  static PerDevice xsite;  // per precision
  cudaError_t e = once_per_device(xsite, device, [] {
    constexpr int R = x_radices<T>();
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t r = cudaFuncSetAttribute(k_xfft_g<T, 0, R>, a, kFftSmemLimit);
    if (r == cudaSuccess) r = cudaFuncSetAttribute(k_xfft_g<T, 1, R>, a, kFftSmemLimit);
    if (r == cudaSuccess) r = cudaFuncSetAttribute(k_xfft_g<T, 2, R>, a, kFftSmemLimit);
    return r == cudaSuccess ? cudaFuncSetAttribute(k_xifft_g<T, R>, a, kFftSmemLimit) : r;
  });
  if (e != cudaSuccess) return e;
  with_z_radices<T>(planz, [&](auto R) {
    static PerDevice site;  // per precision and radix set
    e = once_per_device(site, device, [] {
      return cudaFuncSetAttribute(k_zfft_g<T, decltype(R)::value>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFftSmemLimit);
    });
  });
  return e;
}
cudaError_t fft_generic_setup(int device, bool fp32, const FFTPlanDev& planz) {
  return fp32 ? setup_t<float>(device, planz) : setup_t<double>(device, planz);
}

// Lines per x block: one round of 128 tasks in the first pass, at most 16 lines.
template <class T> static XShape x_shape(int M, int R0) {
  XShape s;
  s.LPB = 128 * R0 / M < 1 ? 1 : (128 * R0 / M > 16 ? 16 : 128 * R0 / M);
  s.sh = sizeof(T) == 8 ? 3 : 4;
  s.LP = M + (M >> s.sh);
  s.smem = (size_t)2 * s.LPB * s.LP * sizeof(typename CplxOf<T>::type);
  if (s.smem > (size_t)kFftSmemLimit) {  // very long lines: no padding
    s.sh = 31;
    s.LP = M;
    s.smem = (size_t)2 * s.LPB * s.LP * sizeof(typename CplxOf<T>::type);
  }
  s.threads = M / R0 > 128 ? 256 : 128;
  return s;
}

template <class T>
cudaError_t xfft_generic(const Geo<T>& g, const Metrics<T>& m, const T* a, const T* b, const T* c,
                         typename CplxOf<T>::type* spec, const FFTPlanDev& pl, const typename CplxOf<T>::type* tw,
                         const typename CplxOf<T>::type* twr, int mode, DevScalars* sc, T* pr, cudaStream_t st) {
  const XShape s = x_shape<T>(g.nx / 2, pl.radix[0]);
  const int nlines = g.ny * g.nz, grid = (nlines + s.LPB - 1) / s.LPB;
  auto go = [&](auto kern) {
    kern<<<grid, s.threads, s.smem, st>>>(g, m, a, b, c, spec, pl, tw, twr, s.LPB, s.LP, s.sh, fdiv_magic(g.nx / 2), fdiv_magic(g.nx / 2 + 1), mode, sc, pr);
  };
  constexpr int R = x_radices<T>();
  if (mode >= 2) go(k_xfft_g<T, 2, R>);
  else if (g.order == 4) go(k_xfft_g<T, 1, R>);
  else go(k_xfft_g<T, 0, R>);
  return cudaGetLastError();
}

// kx lines per z block: 128-byte segments per kz (FP32: 64-byte ones for long
// lines), fewer where shared memory asks for it
template <class T>
cudaError_t zfft_generic(const Geo<T>& g, typename CplxOf<T>::type* spec, const FFTPlanDev& pl,
                         const typename CplxOf<T>::type* tw, int inverse, const DevScalars* sc, cudaStream_t st) {
  typedef typename CplxOf<T>::type CT;
  const int nbuf = pl.npass <= 1 ? 0 : (pl.npass == 2 ? 1 : 2);
  int TKX = sizeof(T) == 8 || g.nz > 256 ? 8 : 16;
  while (TKX > 1 && (size_t)nbuf * TKX * g.nz * sizeof(CT) > (size_t)kFftSmemLimit / 2) TKX >>= 1;
  const int tail = g.nxh % TKX;
  auto go = [&](auto kern) {
    kern<<<dim3((g.nxh + TKX - 1) / TKX, g.ny), g.nz > 256 ? 256 : 128, (size_t)nbuf * TKX * g.nz * sizeof(CT), st>>>(
        g, spec, pl, tw, TKX, fdiv_magic(TKX), fdiv_magic(tail > 0 ? tail : 1), inverse, sc);
  };
  with_z_radices<T>(pl, [&](auto R) { go(k_zfft_g<T, R.value>); });
  return cudaGetLastError();
}

template <class T>
cudaError_t xifft_generic(const Geo<T>& g, const typename CplxOf<T>::type* spec, T* phi, const FFTPlanDev& pl,
                          const typename CplxOf<T>::type* tw, const typename CplxOf<T>::type* twr, T normfft,
                          const DevScalars* sc, cudaStream_t st) {
  const XShape s = x_shape<T>(g.nx / 2, pl.radix[0]);
  const int nlines = g.ny * g.nz;
  k_xifft_g<T, x_radices<T>()><<<(nlines + s.LPB - 1) / s.LPB, s.threads, s.smem, st>>>(g, spec, phi, pl, tw, twr, s.LPB, s.LP, s.sh, normfft, sc);
  return cudaGetLastError();
}

// Largest dynamic shared memory (bytes) a transform of an nx x nz plane's lines asks for in FP64
size_t fft_generic_smem(const FFTPlanDev& planx, const FFTPlanDev& planz) {
  const size_t sx = x_shape<double>(planx.n, planx.radix[0]).smem;
  const size_t sz = planz.npass <= 1 ? 0 : (size_t)(planz.npass == 2 ? 1 : 2) * planz.n * sizeof(double2);
  return sx > sz ? sx : sz;
}

#define CH3D_FFT_INST(T)                                                                                             \
  template cudaError_t xfft_generic<T>(const Geo<T>&, const Metrics<T>&, const T*, const T*, const T*,                \
                                       CplxOf<T>::type*, const FFTPlanDev&, const CplxOf<T>::type*,                   \
                                       const CplxOf<T>::type*, int, DevScalars*, T*, cudaStream_t);                   \
  template cudaError_t zfft_generic<T>(const Geo<T>&, CplxOf<T>::type*, const FFTPlanDev&, const CplxOf<T>::type*,    \
                                       int, const DevScalars*, cudaStream_t);                                         \
  template cudaError_t xifft_generic<T>(const Geo<T>&, const CplxOf<T>::type*, T*, const FFTPlanDev&,                 \
                                        const CplxOf<T>::type*, const CplxOf<T>::type*, T, const DevScalars*,         \
                                        cudaStream_t);
CH3D_FFT_INST(double)
CH3D_FFT_INST(float)

}  // namespace ch3d
