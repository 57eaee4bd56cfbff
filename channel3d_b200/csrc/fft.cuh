// fft.cuh -- batched mixed-radix Stockham FFT through shared memory.
//
// Replaces the FFTW r2r transforms of the Poisson solver
// (src/CFD_2nd/m_Poisson.f90:241-333, kinds R2HC/HC2R).  A block transforms
// several lines at once, one pass per radix (2, 3, 4, 6, 8, 9, 12 or 16): a
// pass reads one buffer and writes the other (Stockham auto-sort, natural
// order at the end); the first pass may read and the last one write global
// memory, so a line of up to 256 points takes two passes with one shared
// buffer and one barrier between them.  Twiddles come from a
// table W_N^q = exp(-2 pi i q / N), q = 0..N-1, built on the host in long
// double.  Inverse transforms use conj(FFT(conj(x))) and are unnormalised like
// FFTW's HC2R.
#pragma once
#include "ch3d_common.cuh"

namespace ch3d {

#define CH3D_MAX_PASSES 16


// Exact integer division by a runtime constant d: q = (n * m) >> 40 with
// m = floor(2^40 / d) + 1, exact whenever n * d < 2^40 (here n < 2^24 and
// d < 2^16).
__host__ __device__ inline unsigned long long fdiv_magic(unsigned d) { return ((1ull << 40) / d) + 1ull; }
__device__ __forceinline__ int fdiv(int n, unsigned long long m) {
  return (int)(((unsigned long long)(unsigned)n * m) >> 40);
}

struct FFTPlanDev {
  int n;                          // complex length
  int npass;
  int radix[CH3D_MAX_PASSES];
  int Ns[CH3D_MAX_PASSES];        // radix[0] * ... * radix[p-1]
  unsigned long long mNB[CH3D_MAX_PASSES];  // division by n / radix[p]
  unsigned long long mNs[CH3D_MAX_PASSES];  // division by radix[0] * ... * radix[p-1]
};

template <class CT, int R> struct Bfly;

template <class CT> struct Bfly<CT, 2> {
  static __device__ __forceinline__ void run(CT* v) {
    CT a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};

// forward radix-4: multiply by -i where W4 appears
template <class CT> struct Bfly<CT, 4> {
  static __device__ __forceinline__ void run(CT* v) {
    CT t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
    CT t2 = cadd(v[1], v[3]), t3 = csub(v[1], v[3]);
    CT mit3 = mk(t3.y, -t3.x);  // -i * t3
    v[0] = cadd(t0, t2);
    v[2] = csub(t0, t2);
    v[1] = cadd(t1, mit3);
    v[3] = csub(t1, mit3);
  }
};

// forward radix-3 with W3 = exp(-2 pi i / 3) = -1/2 - i sqrt(3)/2
template <class CT> struct Bfly<CT, 3> {
  static __device__ __forceinline__ void run(CT* v) {
    typedef decltype(v[0].x) RT;
    const RT s3 = (RT)0.86602540378443864676372317075293618;
    CT t1 = cadd(v[1], v[2]);
    CT t2 = csub(v[1], v[2]);
    CT m = mk(v[0].x - (RT)0.5 * t1.x, v[0].y - (RT)0.5 * t1.y);
    CT jt = mk(s3 * t2.y, -s3 * t2.x);  // -i*sqrt(3)/2 * t2
    v[0] = cadd(v[0], t1);
    v[1] = cadd(m, jt);
    v[2] = csub(m, jt);
  }
};

// forward radix-6 as 2 x 3: n = 3 n1 + n2, k = k1 + 2 k2, twiddle W6^(n2 k1)
template <class CT> struct Bfly<CT, 6> {
  static __device__ __forceinline__ void run(CT* v) {
    typedef decltype(v[0].x) RT;
    const RT s3 = (RT)0.86602540378443864676372317075293618, hf = (RT)0.5;
    CT y[3][2];
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) {
      y[n2][0] = cadd(v[n2], v[n2 + 3]);
      y[n2][1] = csub(v[n2], v[n2 + 3]);
    }
    y[1][1] = cmul(y[1][1], mk(hf, -s3));   // W6
    y[2][1] = cmul(y[2][1], mk(-hf, -s3));  // W6^2
#pragma unroll
    for (int k1 = 0; k1 < 2; ++k1) {
      CT w[3] = {y[0][k1], y[1][k1], y[2][k1]};
      Bfly<CT, 3>::run(w);
#pragma unroll
      for (int k2 = 0; k2 < 3; ++k2) v[k1 + 2 * k2] = w[k2];
    }
  }
};

// forward radix-8: two radix-4 transforms of the even and odd points, W8 = exp(-i pi/4)
template <class CT> struct Bfly<CT, 8> {
  static __device__ __forceinline__ void run(CT* v) {
    typedef decltype(v[0].x) RT;
    const RT h = (RT)0.70710678118654752440084436210484903928;  // sqrt(1/2)
    CT e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    Bfly<CT, 4>::run(e);
    Bfly<CT, 4>::run(o);
    const CT o1 = mk(h * (o[1].x + o[1].y), h * (o[1].y - o[1].x));   // W8^1 o1
    const CT o2 = mk(o[2].y, -o[2].x);                                // W8^2 o2 = -i o2
    const CT o3 = mk(h * (o[3].y - o[3].x), -h * (o[3].x + o[3].y));  // W8^3 o3
    v[0] = cadd(e[0], o[0]); v[4] = csub(e[0], o[0]);
    v[1] = cadd(e[1], o1);   v[5] = csub(e[1], o1);
    v[2] = cadd(e[2], o2);   v[6] = csub(e[2], o2);
    v[3] = cadd(e[3], o3);   v[7] = csub(e[3], o3);
  }
};

// forward radix-9 as 3 x 3: n = 3 n1 + n2, k = k1 + 3 k2, twiddle W9^(n2 k1)
template <class CT> struct Bfly<CT, 9> {
  static __device__ __forceinline__ void run(CT* v) {
    typedef decltype(v[0].x) RT;
    // cos and sin of 2 pi q / 9, q = 1, 2, 4
    const RT c1 = (RT)0.76604444311897803520239265055541667, s1 = (RT)0.64278760968653932632264340990726343;
    const RT c2 = (RT)0.17364817766693034885171662676931480, s2 = (RT)0.98480775301220805936674302458952302;
    const RT c4 = (RT)-0.93969262078590838405410927732473147, s4 = (RT)0.34202014332566873304409961468225958;
    CT y[3][3];
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < 3; ++n1) y[n2][n1] = v[3 * n1 + n2];
      Bfly<CT, 3>::run(y[n2]);
    }
    y[1][1] = cmul(y[1][1], mk(c1, -s1));
    y[1][2] = cmul(y[1][2], mk(c2, -s2));
    y[2][1] = cmul(y[2][1], mk(c2, -s2));
    y[2][2] = cmul(y[2][2], mk(c4, -s4));
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) {
      CT w[3] = {y[0][k1], y[1][k1], y[2][k1]};
      Bfly<CT, 3>::run(w);
#pragma unroll
      for (int k2 = 0; k2 < 3; ++k2) v[k1 + 3 * k2] = w[k2];
    }
  }
};

// multiply by the constant twiddle c + i s
template <class CT, class RT> __device__ __forceinline__ CT cmulk(CT a, RT c, RT s) {
  return mk(a.x * c - a.y * s, a.x * s + a.y * c);
}

// forward radix-12 as 4 x 3: n = 3 n1 + n2, k = k1 + 4 k2; radix-4 over n1,
// twiddle W12^(n2 k1), radix-3 over n2
template <class CT> struct Bfly<CT, 12> {
  static __device__ __forceinline__ void run(CT* v) {
    typedef decltype(v[0].x) RT;
    const RT s3 = (RT)0.86602540378443864676372317075293618;  // sqrt(3)/2
    const RT hf = (RT)0.5;
    CT y[3][4];
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < 4; ++n1) y[n2][n1] = v[3 * n1 + n2];
      Bfly<CT, 4>::run(y[n2]);
    }
    // W12^1 = (s3, -1/2), W12^2 = (1/2, -s3), W12^3 = -i, W12^4 = (-1/2, -s3), W12^6 = -1
    y[1][1] = cmulk(y[1][1], s3, -hf);
    y[1][2] = cmulk(y[1][2], hf, -s3);
    y[1][3] = mk(y[1][3].y, -y[1][3].x);
    y[2][1] = cmulk(y[2][1], hf, -s3);
    y[2][2] = cmulk(y[2][2], -hf, -s3);
    y[2][3] = mk(-y[2][3].x, -y[2][3].y);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      CT w[3] = {y[0][k1], y[1][k1], y[2][k1]};
      Bfly<CT, 3>::run(w);
#pragma unroll
      for (int k2 = 0; k2 < 3; ++k2) v[k1 + 4 * k2] = w[k2];
    }
  }
};

// forward radix-16 as 4 x 4: n = 4 n1 + n2, k = k1 + 4 k2, twiddle W16^(n2 k1)
template <class CT> struct Bfly<CT, 16> {
  static __device__ __forceinline__ void run(CT* v) {
    typedef decltype(v[0].x) RT;
    const RT c1 = (RT)0.92387953251128675612818318939678829, s1 = (RT)0.38268343236508977172845998403039887;  // pi/8
    const RT h = (RT)0.70710678118654752440084436210484903928;
    CT y[4][4];
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) {
#pragma unroll
      for (int n1 = 0; n1 < 4; ++n1) y[n2][n1] = v[4 * n1 + n2];
      Bfly<CT, 4>::run(y[n2]);
    }
    y[1][1] = cmulk(y[1][1], c1, -s1);
    y[1][2] = cmulk(y[1][2], h, -h);
    y[1][3] = cmulk(y[1][3], s1, -c1);
    y[2][1] = cmulk(y[2][1], h, -h);
    y[2][2] = mk(y[2][2].y, -y[2][2].x);
    y[2][3] = cmulk(y[2][3], -h, -h);
    y[3][1] = cmulk(y[3][1], s1, -c1);
    y[3][2] = cmulk(y[3][2], -h, -h);
    y[3][3] = cmulk(y[3][3], -c1, s1);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) {
      CT w[4] = {y[0][k1], y[1][k1], y[2][k1], y[3][k1]};
      Bfly<CT, 4>::run(w);
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) v[k1 + 4 * k2] = w[k2];
    }
  }
};

// One Stockham pass of radix R over `nlines` lines of length N with stride Ns:
// load(l, n) gives point n of line l, store(l, n, v) takes it; they may be
// shared or global memory.  Threads tid of nthr; LFAST selects the task order:
// line index fastest (lines interleaved in memory) or butterfly index fastest
// (lines contiguous).
template <class CT, int R, bool LFAST, class LD, class ST>
__device__ __forceinline__ void fft_pass_r(int N, int Ns, int nlines, const CT* __restrict__ tw, unsigned long long mNB,
                                           unsigned long long mNs, unsigned long long mL, LD load, ST store) {
  const int NB = N / R;
  const int total = nlines * NB;
  const int step = N / (Ns * R);
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    int l, b;
    if (LFAST) { b = fdiv(t, mL); l = t - b * nlines; }
    else { l = fdiv(t, mNB); b = t - l * NB; }
    const int kk = b - fdiv(b, mNs) * Ns;
    CT v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = load(l, b + r * NB);
    if (Ns > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], __ldg(tw + r * kk * step));
    }
    Bfly<CT, R>::run(v);
    const int idxD = (b - kk) * R + kk;
#pragma unroll
    for (int r = 0; r < R; ++r) store(l, idxD + r * Ns, v[r]);
  }
}
// pass p of the plan; mL: fdiv_magic(nlines), read for LFAST only.  MAXR: radices compiled in
// (9 or 16: the larger butterflies cost every pass of a kernel their registers)
template <class CT, bool LFAST, int MAXR, class LD, class ST>
__device__ __forceinline__ void fft_pass(const FFTPlanDev& pl, int p, int nlines, unsigned long long mL,
                                         const CT* __restrict__ tw, LD load, ST store) {
  const unsigned long long mNB = pl.mNB[p], mNs = pl.mNs[p];
  const int N = pl.n, Ns = pl.Ns[p];
  switch (pl.radix[p]) {
    case 2: fft_pass_r<CT, 2, LFAST>(N, Ns, nlines, tw, mNB, mNs, mL, load, store); break;
    case 3: fft_pass_r<CT, 3, LFAST>(N, Ns, nlines, tw, mNB, mNs, mL, load, store); break;
    case 4: fft_pass_r<CT, 4, LFAST>(N, Ns, nlines, tw, mNB, mNs, mL, load, store); break;
    case 6: fft_pass_r<CT, 6, LFAST>(N, Ns, nlines, tw, mNB, mNs, mL, load, store); break;
    case 8: fft_pass_r<CT, 8, LFAST>(N, Ns, nlines, tw, mNB, mNs, mL, load, store); break;
    case 9: fft_pass_r<CT, 9, LFAST>(N, Ns, nlines, tw, mNB, mNs, mL, load, store); break;
    case 12:
      if constexpr (MAXR >= 12) fft_pass_r<CT, 12, LFAST>(N, Ns, nlines, tw, mNB, mNs, mL, load, store);
      break;
    case 16:
      if constexpr (MAXR >= 16) fft_pass_r<CT, 16, LFAST>(N, Ns, nlines, tw, mNB, mNs, mL, load, store);
      break;
  }
}

}  // namespace ch3d
