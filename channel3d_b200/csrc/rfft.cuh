// rfft.cuh -- register-resident Stockham FFT for the Poisson transforms.
//
// A line of N complex points is owned by P threads; thread t holds the E =
// N / P points t + P m (m = 0..E-1) in registers.  In a Stockham pass of
// radix R (R | E) with stride NS, butterfly b = t + P q (q = 0..E/R-1) reads
// the points b + r N/R = t + P (q + r E/R): always the thread's own points.
// Its outputs go to (b - kk) R + kk + r NS (kk = b mod NS); while NS is not a
// multiple of P they belong to other threads and are exchanged through
// shared memory, once NS is a multiple of P they stay in the thread.  A plan
// therefore starts with radices whose product is P (one exchange after each)
// and ends with in-thread radices whose product is E.  The first pass reads
// the line straight from global memory and the result is left in the same
// t + P m order, so loads and stores are coalesced across the threads of a
// line.  Twiddles come from the W_N table of the generic transform (fft.cuh).
#pragma once
#include "fft.cuh"

namespace ch3d {

struct WarpSync {
  __device__ __forceinline__ void operator()() const { __syncwarp(); }
};
struct BlockSync {
  __device__ __forceinline__ void operator()() const { __syncthreads(); }
};

// Position of point p in a line's exchange buffer: p * ss, or with PAD one
// 16-byte gap after every 8 points (p + p / 8), which spreads the stride-R
// writes of the first pass over all shared-memory banks.
template <bool PAD> __device__ __forceinline__ int xpos(int p, int ss) { return PAD ? p + (p >> 3) : p * ss; }

// One pass (radix R, stride NS) over the thread's E points; sm: the line's
// exchange buffer (point p at xpos<PAD>(p, ss)).
template <class CT, int N, int P, int E, int NS, int R, bool PAD, class Sync>
__device__ __forceinline__ void rs_pass(CT (&v)[E], CT* sm, int ss, int t, const CT* __restrict__ tw, Sync sync) {
  static_assert(E % R == 0, "radix must divide the points per thread");
  constexpr int Q = E / R;
  constexpr int STEP = N / (NS * R);
  constexpr bool EXCH = NS % P != 0;
  CT o[E];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int b = t + P * q;
    const int kk = b % NS;
    CT x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = v[q + r * Q];
    if (NS > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) x[r] = cmul(x[r], __ldg(tw + r * kk * STEP));
    }
    Bfly<CT, R>::run(x);
    if (EXCH) {
      const int base = (b - kk) * R + kk;
#pragma unroll
      for (int r = 0; r < R; ++r) sm[xpos<PAD>(base + r * NS, ss)] = x[r];
    } else {
      constexpr int s = EXCH ? 1 : NS / P;
#pragma unroll
      for (int r = 0; r < R; ++r) o[(q - q % s) * R + q % s + r * s] = x[r];
    }
  }
  if (EXCH) {
    sync();
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = sm[xpos<PAD>(t + P * m, ss)];
    sync();
  } else {
#pragma unroll
    for (int m = 0; m < E; ++m) v[m] = o[m];
  }
}

template <class CT, int N, int P, int E, bool PAD, int NS, int... Rs> struct RRun;
template <class CT, int N, int P, int E, bool PAD, int NS> struct RRun<CT, N, P, E, PAD, NS> {
  template <class Sync> __device__ __forceinline__ static void run(CT (&)[E], CT*, int, int, const CT*, Sync) {
    static_assert(NS == N, "plan radices must multiply to N");
  }
};
template <class CT, int N, int P, int E, bool PAD, int NS, int R, int... Rs> struct RRun<CT, N, P, E, PAD, NS, R, Rs...> {
  template <class Sync>
  __device__ __forceinline__ static void run(CT (&v)[E], CT* sm, int ss, int t, const CT* __restrict__ tw, Sync sync) {
    rs_pass<CT, N, P, E, NS, R, PAD>(v, sm, ss, t, tw, sync);
    RRun<CT, N, P, E, PAD, NS * R, Rs...>::run(v, sm, ss, t, tw, sync);
  }
};

// A plan: N points, P threads per line, radices in pass order.  run<PAD>:
// PAD for a line-contiguous buffer of padded_len() points (ss unused),
// otherwise point p at sm[p * ss].
template <int N_, int P_, int... Rs> struct RPlan {
  static constexpr int N = N_, P = P_, E = N_ / P_;
  static constexpr int padded_len() { return N_ + N_ / 8; }
  template <bool PAD, class CT, class Sync>
  __device__ __forceinline__ static void run(CT (&v)[E], CT* sm, int ss, int t, const CT* __restrict__ tw, Sync sync) {
    RRun<CT, N, P, E, PAD, 1, Rs...>::run(v, sm, ss, t, tw, sync);
  }
};

}  // namespace ch3d
