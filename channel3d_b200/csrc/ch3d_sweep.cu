// ch3d_sweep.cu -- the Crank-Nicolson line solves of the 2nd- and 4th-order
// steps that do not run inside the column kernels: the periodic x, z and y
// sweeps (clcU1/2/3Hat_FIMP_010 and _000, src/CFD_2nd/m_TSchemeFIMP_inc.f90:
// 187-347, 559-729, 950-1128; clcU1/2/3Hat_PIMP_0, m_TSchemePIMP_inc.f90:435-461,
// 594-621, 745-771) and the y sweep between walls (clcU1/2/3Hat_PIMP, :392-740).
//
// The systems of one direction and component differ in the right-hand side
// only, so the coefficients of the elimination and the back substitution are
// those of the row table (walls) or the periodic factor block, the same for
// every line.  A line's rows stay in the registers of the threads that own its
// chunks: each chunk runs the first-order recurrences from zero, the chunks'
// end values are combined by a scan whose coefficient products a thread
// computes once and keeps for all the lines it solves, and the chunk repeats
// the recurrence from its true start value.  Right-hand side and solution
// cross global memory once each.  At 128^3 in FP64 (0.1 GB per sweep): x 28 us, z
// and y 37 each (one thread per line with staged loads, and the partitioned y solve:
// 44, 46 and 57); bound by the latency of load, two scans and store, 16 warps per SM.
#include "ch3d_march.cuh"

namespace ch3d {

// Exclusive scan of chunk maps d -> A d + B with fixed A over the chunks of a
// line, chunk q of CW in a warp (lane stride C) and warp after warp; UP from the
// first chunk, else from the last.
template <class R, int C, bool UP> struct FixedScan {
  static constexpr int CW = 32 / C;
  static constexpr int LOG = CW == 32 ? 5 : CW == 16 ? 4 : CW == 8 ? 3 : CW == 4 ? 2 : CW == 2 ? 1 : 0;
  R lv[LOG > 0 ? LOG : 1];  // factor of the value taken at each level
  R exA;                    // product over the chunks before this one in the warp
  int q;
  static __device__ __forceinline__ R from(R v, int o) {
    return UP ? __shfl_up_sync(0xffffffffu, v, o) : __shfl_down_sync(0xffffffffu, v, o);
  }
  // aggA: [warps], the warps' products
  __device__ __forceinline__ void init(R A, R* aggA, int lane, int warp) {
    q = UP ? lane / C : CW - 1 - lane / C;
    R f = A;
#pragma unroll
    for (int l = 0; l < LOG; ++l) {
      const R g = from(f, C << l);
      const bool take = q >= (1 << l);
      lv[l] = take ? f : (R)0;
      if (take) f *= g;
    }
    exA = C < 32 ? from(f, C % 32) : (R)1;
    if (q == 0) exA = (R)1;
    if (aggA && q == CW - 1) aggA[warp] = f;
  }
  // agg: [warps][C]; contains a block barrier when the line spans several warps
  __device__ __forceinline__ R run(R b, R* agg, const R* aggA, int warp, int nwarps, int c) const {
#pragma unroll
    for (int l = 0; l < LOG; ++l) {
      const R g = from(b, C << l);
      b += lv[l] * g;
    }
    R dx = (R)0;
    if (nwarps > 1) {
      if (q == CW - 1) agg[warp * C + c] = b;
      __syncthreads();
      for (int w = 0; w < nwarps - 1; ++w) {
        const int wq = UP ? w : nwarps - 1 - w;
        if (UP ? wq >= warp : wq <= warp) break;
        dx = agg[wq * C + c] + aggA[wq] * dx;
      }
    }
    if (C < 32) {
      const R e = from(b, C % 32);
      if (q > 0) dx = e + exA * dx;
    }
    return dx;
  }
};

// Rows of a periodic direction's factor block (ch3d_march.cuh).
struct PtriRows {
  const double* F;
  int n;
  __device__ __forceinline__ double pp(int j) const { return j == 0 ? 1.0 / F[3 * (n + 1) + 1] : F[j + 1]; }  // row 1 divides by b
  __device__ __forceinline__ double w(int j) const { return F[2 * (n + 1) + j + 1]; }
  __device__ __forceinline__ double a() const { return F[3 * (n + 1)]; }
  __device__ __forceinline__ double c() const { return F[3 * (n + 1) + 2]; }
  __device__ __forceinline__ double den() const { return F[3 * (n + 1) + 3]; }
};

// ---------------------------------------------------------------------------
// x sweep, periodic: a line per warp, RPT consecutive points per lane, in place.
// ---------------------------------------------------------------------------
template <class T, int RPT>
__global__ void __launch_bounds__(128) k_sweep_x(int nx, long long nlines, const double* __restrict__ pf, size_t pfs,
                                                 T* __restrict__ r0, T* __restrict__ r1, T* __restrict__ r2,
                                                 const DevScalars* __restrict__ sc) {
  typedef typename CplxOf<T>::type T2;
  if (sc->status) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const PtriRows F{pf + pfs * (sc->ns - 1), nx};
  const int i0 = lane * RPT;
  const T a = (T)F.a(), cc = (T)F.c(), rden = (T)(1.0 / F.den());
  T pp[RPT], w[RPT];
#pragma unroll
  for (int u = 0; u < RPT; ++u) {
    const bool ok = i0 + u < nx - 1;
    pp[u] = ok ? (T)F.pp(i0 + u) : (T)0;
    w[u] = ok ? (T)F.w(i0 + u) : (T)0;
  }
  FixedScan<T, 1, true> fu;
  FixedScan<T, 1, false> fd;
  {
    T A = (T)1, B = (T)1;
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      A *= i0 + u == 0 ? (T)0 : -a * pp[u];
      B *= -cc * pp[u];
    }
    fu.init(A, nullptr, lane, 0);
    fd.init(B, nullptr, lane, 0);
  }
  const int ln = (nx - 1) / RPT, l2 = (nx - 2) / RPT;  // lanes of points n and n-1
  T* const r = blockIdx.y == 0 ? r0 : (blockIdx.y == 1 ? r1 : r2);
  for (long long line = (long long)blockIdx.x * 4 + warp; line < nlines; line += (long long)gridDim.x * 4) {
    T* const g = r + line * nx;
    T v[RPT];
#pragma unroll
    for (int u = 0; u < RPT; u += 2) {
      T2 t = mk((T)0, (T)0);
      if (i0 + u < nx) t = *reinterpret_cast<const T2*>(g + i0 + u);  // nx and i0 even
      v[u] = t.x; v[u + 1] = t.y;
    }
    T last = (T)0;
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (i0 + u == nx - 1) last = v[u];
    last = __shfl_sync(0xffffffffu, last, ln);
    T b = (T)0;
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      v[u] *= pp[u];
      b = v[u] - (i0 + u == 0 ? (T)0 : a * pp[u]) * b;
    }
    T d = fu.run(b, nullptr, nullptr, 0, 1, 0);
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      d = v[u] - (i0 + u == 0 ? (T)0 : a * pp[u]) * d;
      v[u] = d;
    }
    b = (T)0;
#pragma unroll
    for (int u = RPT - 1; u >= 0; --u) b = v[u] - cc * pp[u] * b;
    d = fd.run(b, nullptr, nullptr, 0, 1, 0);
#pragma unroll
    for (int u = RPT - 1; u >= 0; --u) {
      d = v[u] - cc * pp[u] * d;
      v[u] = d;
    }
    // closure of point n, then f_j = f_n vecn2_j + arrmn_j
    T e2 = (T)0;
#pragma unroll
    for (int u = 0; u < RPT; ++u)
      if (i0 + u == nx - 2) e2 = v[u];
    const T e0 = __shfl_sync(0xffffffffu, v[0], 0);
    e2 = __shfl_sync(0xffffffffu, e2, l2);
    const T fn = (last - cc * e0 - a * e2) * rden;
#pragma unroll
    for (int u = 0; u < RPT; u += 2) {
      T2 t = mk(v[u] + fn * w[u], v[u + 1] + fn * w[u + 1]);
      if (i0 + u == nx - 1) t.x = fn;
      if (i0 + u + 1 == nx - 1) t.y = fn;
      if (i0 + u < nx) *reinterpret_cast<T2*>(g + i0 + u) = t;
    }
  }
}

// ---------------------------------------------------------------------------
// z and y sweeps: a block solves C consecutive i of one line set at a time,
// thread (i, chunk p) with RPT consecutive rows.  Rows are `rs` elements apart.
//   PER   periodic (factor block pf), else between walls (row table of the
//         substep; set 1 for uy, whose first row is held)
//   ADDU  write u* = u + solution, else the solution in place
// The line sets of component blockIdx.z start at (i0, o): blockIdx.y = o.
// ---------------------------------------------------------------------------
template <class T> struct SweepArgs {
  T *r0, *r1, *r2;
  const T *u0, *u1, *u2;
  T *s0, *s1, *s2;
  __device__ __forceinline__ T* r(int c) const { return c == 0 ? r0 : (c == 1 ? r1 : r2); }
  __device__ __forceinline__ const T* u(int c) const { return c == 0 ? u0 : (c == 1 ? u1 : u2); }
  __device__ __forceinline__ T* us(int c) const { return c == 0 ? s0 : (c == 1 ? s1 : s2); }
};

// shared memory of the scans, rounded to the staging's alignment
template <class R> __host__ __device__ constexpr size_t sweep_scan_bytes(int nwarps, int C) {
  return ((size_t)(2 * nwarps * C + 2 * nwarps + 2 * C) * sizeof(R) + 15) / 16 * 16;
}

template <class T, class R, int C, int RPT, int MAXT, int MINB, bool PER, bool ADDU>
__global__ void __launch_bounds__(MAXT, MINB) k_sweep(SweepArgs<T> A, int nx, int n, long long rs, long long os, int no,
                                                      const double* __restrict__ pf, size_t pfs, const R* __restrict__ tab, int addp,
                                                      const DevScalars* __restrict__ sc) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (sc->status) return;
  const int c = threadIdx.x % C, p = threadIdx.x / C, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5, comp = blockIdx.z;
  R* const aggU = reinterpret_cast<R*>(smem_raw);  // [warps][C] up, [warps][C] down, the products [2][warps], ends [2][C]
  R* const aggD = aggU + nwarps * C;
  R* const prod = aggD + nwarps * C;
  R* const ends = prod + 2 * nwarps;
  // the thread's rows of the next line set, [stage][rhs rows, u rows][threads]
  T* const stg = reinterpret_cast<T*>(smem_raw + sweep_scan_bytes<R>(nwarps, C)) + threadIdx.x;
  const int m = PER ? n - 1 : n;  // rows of the recurrences
  const int j0 = p * RPT;
  const int i = blockIdx.x * C + c;
  const bool in = i < nx;
  T* const r = A.r(comp);
  const T* const ub = A.u(comp);
  auto issue = [&](int o, int st) {
    if (in && o < no) {
      const long long base = i + os * o + rs * j0;
      T* const d = stg + (size_t)st * (ADDU ? 2 : 1) * RPT * blockDim.x;
#pragma unroll
      for (int u = 0; u < RPT; ++u)
        if (j0 + u < m) {
          cp_async_el(d + u * blockDim.x, r + base + rs * u);
          if (ADDU) cp_async_el(d + (RPT + u) * blockDim.x, ub + base + rs * u);
        }
    }
    cp_async_commit();
  };
  issue(blockIdx.y, 0);
  const PtriRows F{pf + pfs * (sc->ns - 1), n};
  const R a = PER ? (R)F.a() : (R)0, cc = PER ? (R)F.c() : (R)0, rden = PER ? (R)(1.0 / F.den()) : (R)0;
  const R* const tb = PER ? nullptr : tab + (size_t)(sc->ns - 1) * n * MT_W + (comp == 1 ? MT_A1 : MT_A0);
  R pp[RPT], s[RPT], cb[RPT], w[PER ? RPT : 1];
  R Au = (R)1, Ad = (R)1;
#pragma unroll
  for (int u = 0; u < RPT; ++u) {
    const int j = j0 + u;
    pp[u] = s[u] = cb[u] = (R)0;
    if (PER) w[u] = (R)0;
    if (j < m) {
      if constexpr (PER) {
        pp[u] = (R)F.pp(j);
        w[u] = (R)F.w(j);
        s[u] = j == 0 ? (R)0 : a * pp[u];
        cb[u] = cc * pp[u];
      } else {
        pp[u] = __ldg(tb + (size_t)j * MT_W + 1);
        s[u] = j == 0 ? (R)0 : __ldg(tb + (size_t)j * MT_W) * pp[u];
        cb[u] = __ldg(tb + (size_t)j * MT_W + 2);
      }
    }
    Au *= -s[u];
    Ad *= -cb[u];
  }
  FixedScan<R, C, true> fu;
  FixedScan<R, C, false> fd;
  fu.init(Au, prod, lane, warp);
  fd.init(Ad, prod + nwarps, lane, warp);
  __syncthreads();
  const R add = addp && comp == 0 ? (R)sc->dpmdxns : (R)0;
  int st = 0;
  for (int o = blockIdx.y; o < no; o += gridDim.y, st ^= 1) {  // uniform over the block
    const long long base = i + os * o;
    R v[RPT], last = (R)0, ulast = (R)0;
    if (PER && in) {
      last = (R)r[base + rs * (n - 1)] + add;
      if (ADDU) ulast = (R)__ldg(ub + base + rs * (n - 1));
    }
    issue(o + gridDim.y, st ^ 1);  // the next set's rows, while this one is solved
    cp_async_wait<1>();            // each thread reads only what it copied itself
    const T* const d0 = stg + (size_t)st * (ADDU ? 2 : 1) * RPT * blockDim.x;
#pragma unroll
    for (int u = 0; u < RPT; ++u) v[u] = in && j0 + u < m ? (R)d0[u * blockDim.x] + add : (R)0;
    if (!PER && comp == 1 && p == 0) v[0] = (R)0;  // duy_ym: uy_ym is constant (Update_uy_ym_CH)
    R b = (R)0;
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      v[u] *= pp[u];
      b = v[u] - s[u] * b;
    }
    R d = fu.run(b, aggU, prod, warp, nwarps, c);
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      d = v[u] - s[u] * d;
      v[u] = d;
    }
    b = (R)0;
#pragma unroll
    for (int u = RPT - 1; u >= 0; --u) b = v[u] - cb[u] * b;
    d = fd.run(b, aggD, prod + nwarps, warp, nwarps, c);
#pragma unroll
    for (int u = RPT - 1; u >= 0; --u) {
      d = v[u] - cb[u] * d;
      v[u] = d;
    }
    T* const out = ADDU ? A.us(comp) : r;
    if constexpr (PER) {
      if (p == 0) ends[c] = v[0];
#pragma unroll
      for (int u = 0; u < RPT; ++u)
        if (j0 + u == n - 2) ends[C + c] = v[u];
      __syncthreads();
      const R fn = (last - cc * ends[c] - a * ends[C + c]) * rden;
      if (in) {
        if (p == 0) out[base + rs * (n - 1)] = (T)(ADDU ? ulast + fn : fn);
#pragma unroll
        for (int u = 0; u < RPT; ++u)
          if (j0 + u < m) out[base + rs * (j0 + u)] = (T)((ADDU ? (R)d0[(RPT + u) * blockDim.x] : (R)0) + (v[u] + fn * w[u]));
      }
    } else if (in) {
#pragma unroll
      for (int u = 0; u < RPT; ++u)
        if (j0 + u < m) out[base + rs * (j0 + u)] = (T)((ADDU ? (R)d0[(RPT + u) * blockDim.x] : (R)0) + v[u]);
    }
    if (nwarps == 1) __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// One thread per line, for lines too long for the registers above: the
// recurrences in place in global memory (periodic: InversePTriFixedCoe).
// ---------------------------------------------------------------------------
template <class T, class R, bool PER, bool ADDU>
__global__ void __launch_bounds__(128) k_sweep_long(SweepArgs<T> A, int ni, long long is, int n, long long rs,
                                                    long long os, int no, const double* __restrict__ pf, size_t pfs,
                                                    const R* __restrict__ tab, int addp,
                                                    const DevScalars* __restrict__ sc) {
  if (sc->status) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x, comp = blockIdx.z;
  if (i >= ni) return;
  const PtriRows F{pf + pfs * (sc->ns - 1), n};
  const R a = PER ? (R)F.a() : (R)0, cc = PER ? (R)F.c() : (R)0;
  const R* const tb = PER ? nullptr : tab + (size_t)(sc->ns - 1) * n * MT_W + (comp == 1 ? MT_A1 : MT_A0);
  const R add = addp && comp == 0 ? (R)sc->dpmdxns : (R)0;
  const int m = PER ? n - 1 : n;
  for (int o = blockIdx.y; o < no; o += gridDim.y) {
    const long long base = i * is + os * o;
    T* const f = A.r(comp) + base;
    R d = (R)0, last = (R)0;
    if (PER) last = f[rs * (n - 1)] + add;
    for (int j = 0; j < m; ++j) {
      const R pp = PER ? (R)F.pp(j) : __ldg(tb + (size_t)j * MT_W + 1);
      const R s = j == 0 ? (R)0 : (PER ? a : __ldg(tb + (size_t)j * MT_W));
      const R v = !PER && comp == 1 && j == 0 ? (R)0 : (R)f[rs * j] + add;
      d = (v - s * d) * pp;
      f[rs * j] = (T)d;
    }
    d = (R)0;
    R el = (R)0;
    for (int j = m - 1; j >= 0; --j) {
      const R cb = PER ? cc * (R)F.pp(j) : __ldg(tb + (size_t)j * MT_W + 2);
      d = f[rs * j] - cb * d;
      f[rs * j] = (T)d;
      if (j == n - 2) el = d;
    }
    R fn = (R)0;
    if (PER) {
      fn = (last - cc * d - a * el) / (R)F.den();
      f[rs * (n - 1)] = (T)fn;
    }
    if (PER || ADDU)
      for (int j = 0; j < n; ++j) {
        R x = (R)f[rs * j];
        if (PER && j < m) x += fn * (R)F.w(j);
        if (ADDU) A.us(comp)[base + rs * j] = (T)((R)A.u(comp)[base + rs * j] + x);
        else f[rs * j] = (T)x;
      }
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
constexpr int kSweepXMax = 768;      // points of a line held by a warp, 24 per lane
constexpr int kSweepMaxRows = 6144;  // 256 chunks of 24 rows

template <class T> static SweepArgs<T> sweep_args(const ch3d_ctx* c) {
  T** f = (T**)c->f;
  return {f[7], f[8], f[9], f[0], f[1], f[2], f[12], f[13], f[14]};
}

// rows of length n at stride rs, `no` sets of ni lines at stride os.  Up to 768 rows a
// block's 8 or 16 lines fill whole 32-byte sectors of both precisions; longer lines take
// the chunks of 4, 2 or 1 lines a block of 256 threads can hold.  ADI's x and z sweeps at
// 1024x32x32 60 us together and at 32x32x1024 93 (one thread per line 500 and 450), all
// solves of 32x1024x32 85 us (one thread per line 890).
template <class T, class R, bool PER, bool ADDU>
static cudaError_t sweep_rows(ch3d_ctx* c, int ni, int n, long long rs, long long os, int no, const double* pf, int addp) {
  const SweepArgs<T> A = sweep_args<T>(c);
  const R* tab = (const R*)c->mtab;
  const size_t pfs = ptri_doubles(c->nx, c->ny, c->nz);
  if (n > kSweepMaxRows) {
    k_sweep_long<T, R, PER, ADDU><<<dim3((ni + 127) / 128, no < 65535 ? no : 65535, 3), 128, 0, c->stream>>>(A, ni, 1, n, rs, os, no, pf, pfs, tab, addp, c->sc);
    return cudaGetLastError();
  }
  cudaError_t err = cudaSuccess;
  auto go = [&](auto kern, PerDevice& site, int C, int RPT, int maxt) {
    const int CW = 32 / C, P = ((n + RPT - 1) / RPT + CW - 1) / CW * CW, threads = C * P, nw = threads / 32;
    const size_t row = (size_t)2 * (ADDU ? 2 : 1) * RPT * sizeof(T);  // staging per thread
    const size_t smem = sweep_scan_bytes<R>(nw, C) + row * threads;
    err = smem_limit_once(site, c->device, kern, sweep_scan_bytes<R>(maxt / 32, C) + row * maxt);
    if (err != cudaSuccess) return;
    const int gx = (ni + C - 1) / C;
    // a few line sets per block, so that their coefficients are formed once, while the GPU stays full
    const long long want = (long long)sm_count(c->device) * (2048 / threads > 0 ? 2048 / threads : 1);
    long long gy = (want + 3LL * gx - 1) / (3LL * gx);
    if (gy > no) gy = no;
    if (gy < 1) gy = 1;
    if (gy > 65535) gy = 65535;
    kern<<<dim3(gx, (unsigned)gy, 3), threads, smem, c->stream>>>(A, ni, n, rs, os, no, pf, pfs, tab, addp, c->sc);
  };
  static PerDevice s8, s8w, s12, s24, s4, s2, s1, sx;  // per template instance
  if constexpr (PER && !ADDU)  // lines along x: one line a block, consecutive points
    if (ni == 1 && n <= 2048) {
      go(k_sweep<T, R, 1, 8, 256, 2, PER, ADDU>, sx, 1, 8, 256);
      return err != cudaSuccess ? err : cudaGetLastError();
    }
  if (n <= 128) go(k_sweep<T, R, 16, 8, 256, 2, PER, ADDU>, s8, 16, 8, 256);
  else if (n <= 256) go(k_sweep<T, R, 8, 8, 256, 2, PER, ADDU>, s8w, 8, 8, 256);
  else if (n <= 384) go(k_sweep<T, R, 8, 12, 256, 1, PER, ADDU>, s12, 8, 12, 256);
  else if (n <= 768) go(k_sweep<T, R, 8, 24, 256, 1, PER, ADDU>, s24, 8, 24, 256);
  else if (n <= 1536) go(k_sweep<T, R, 4, 24, 256, 1, PER, ADDU>, s4, 4, 24, 256);
  else if (n <= 3072) go(k_sweep<T, R, 2, 24, 256, 1, PER, ADDU>, s2, 2, 24, 256);
  else go(k_sweep<T, R, 1, 24, 256, 1, PER, ADDU>, s1, 1, 24, 256);
  return err != cudaSuccess ? err : cudaGetLastError();
}

template <class T> static cudaError_t sweep_x(ch3d_ctx* c, const double* pf) {
  T** f = (T**)c->f;
  const long long nlines = (long long)c->ny * c->nz;
  if (c->nx > kSweepXMax) return sweep_rows<T, T, true, false>(c, 1, c->nx, 1, c->nx, (int)nlines, pf, 0);
  const long long nb = (nlines + 3) / 4, cap = (long long)sm_count(c->device) * 6;
  const dim3 grid((unsigned)(nb < cap ? nb : cap), 3);
  auto go = [&](auto kern) { kern<<<grid, 128, 0, c->stream>>>(c->nx, nlines, pf, ptri_doubles(c->nx, c->ny, c->nz), f[7], f[8], f[9], c->sc); };
  if (c->nx <= 64) go(k_sweep_x<T, 2>);
  else if (c->nx <= 128) go(k_sweep_x<T, 4>);
  else if (c->nx <= 256) go(k_sweep_x<T, 8>);
  else if (c->nx <= 384) go(k_sweep_x<T, 12>);
  else go(k_sweep_x<T, 24>);
  return cudaGetLastError();
}

template <class T> static cudaError_t ptri_xz_t(ch3d_ctx* c) {
  const cudaError_t e = sweep_x<T>(c, ptri_block(c, 0));
  if (e != cudaSuccess) return e;
  return sweep_rows<T, T, true, false>(c, c->nx, c->nz, (long long)c->nx * c->ny, c->nx, c->ny, ptri_block(c, 1), 0);
}
cudaError_t launch_ptri_xz(ch3d_ctx* c) { return c->fp32 ? ptri_xz_t<float>(c) : ptri_xz_t<double>(c); }

// periodic y: u* = u + solution; the partially implicit RhsX gets the mean
// pressure gradient first (clcRhsX_PIMP adds it; the FIMP RhsX carries it already)
template <class T> static cudaError_t ptri_y_t(ch3d_ctx* c) {
  return sweep_rows<T, T, true, true>(c, c->nx, c->ny, c->nx, (long long)c->nx * c->ny, c->nz, ptri_block(c, 2),
                                   c->cfg.IsImplicit == 1);
}
cudaError_t launch_ptri_y(ch3d_ctx* c) { return c->fp32 ? ptri_y_t<float>(c) : ptri_y_t<double>(c); }

// y between walls: u* = u + solution; the 4th-order, FIMP and LES RhsX already carry the forcing
template <class T, class R> static cudaError_t uhat_t(ch3d_ctx* c) {
  return sweep_rows<T, R, false, true>(c, c->nx, c->ny, c->nx, (long long)c->nx * c->ny, c->nz, nullptr,
                                       c->cfg.order != 4 && c->cfg.IsImplicit != 2 && c->cfg.LES_type == 0);
}
cudaError_t launch_uhat(ch3d_ctx* c) {
  if (!c->fp32) return uhat_t<double, double>(c);
  return c->cfg.LES_type > 0 ? uhat_t<float, double>(c) : uhat_t<float, float>(c);  // LES: FP64 solves
}

}  // namespace ch3d
