// ch3d_substep.cu -- the scalar work between the field kernels: one launch at
// the start of each substep (the step's CFL number and dt, PMcoeUpdate, the
// bulk constraint from the partial sums, the line solves' coefficient tables)
// and one at its end (the bulk mean, the limit checks).
//
// Few partial sums are reduced by one block; many by CH3D_NRED blocks, the
// last of which to finish sums the blocks' results in block order and does the
// scalar work, so the result does not depend on the order the blocks run in.
// Letting the projection's last block do this work instead, without a launch, took
// 4 us more of the projection and 145 against 141 us per step at 64^3.
#include "ch3d_march.cuh"

namespace ch3d {

constexpr int kSetupThreads = 512;
constexpr int kSumPer = 8;         // partial sums per thread that one block loads at once
constexpr int kStagedRows = 1024;  // rows whose coefficient vectors fit in the shared memory of the setup block

// Sum of part[0..n) over the grid, valid in thread 0 of the block for which the
// function returns true (the only block, or the last one to finish).  All loads of
// a thread are in flight together and the block sums by shuffles: one thread per
// loop trip with a barrier per halving took 6 us of a launch that is otherwise
// two round trips to L2.
__device__ __forceinline__ bool grid_sum(const double* __restrict__ part, int n, double* __restrict__ red,
                                         unsigned* ticket, double* sh /* kSetupThreads / 32 */, double& sum) {
  const int nb = gridDim.x, chunk = (n + nb - 1) / nb;
  const int lo = blockIdx.x * chunk, hi = min(n, lo + chunk);
  auto block_sum = [&](double v) {
    for (int w = 16; w > 0; w >>= 1) v += __shfl_down_sync(0xffffffffu, v, w);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x < 32) {
      r = threadIdx.x < kSetupThreads / 32 ? sh[threadIdx.x] : 0.0;
      for (int w = kSetupThreads / 64; w > 0; w >>= 1) r += __shfl_down_sync(0xffffffffu, r, w);
    }
    return r;
  };
  double s = 0.0;
  for (int q0 = lo + (int)threadIdx.x; q0 < hi; q0 += kSumPer * kSetupThreads) {
    double v[kSumPer];
#pragma unroll
    for (int u = 0; u < kSumPer; ++u) v[u] = q0 + u * kSetupThreads < hi ? __ldg(part + q0 + u * kSetupThreads) : 0.0;
#pragma unroll
    for (int u = 0; u < kSumPer; ++u) s += v[u];
  }
  sum = block_sum(s);
  if (nb == 1) return true;
  __shared__ bool last;
  if (threadIdx.x == 0) {
    red[blockIdx.x] = sum;
    __threadfence();
    last = atomicInc(ticket, nb - 1) == (unsigned)nb - 1;  // back to 0 for the next launch
  }
  __syncthreads();  // also: the first sum's values in sh have been read
  if (!last) return false;
  __threadfence();
  s = 0.0;
  for (int q = threadIdx.x; q < nb; q += kSetupThreads) s += __ldcg(red + q);
  sum = block_sum(s);
  return true;
}

struct SubstepPar {
  int ns, begin, last;  // begin: the step starts here; last: the step's diagnostics follow
  double gam, the, alp;
  int iCFL, IsUxConst, order;
  double CFLc, dtMax, xnu, ubulk, norm_bulk, nxnz, yly, visc_wall;
};

// Elimination factors of the row table for pmBeta (see ch3d_march.cuh) of one
// Helmholtz set, upwards: a, 1/m, c/m
template <class T>
__device__ void update_row_factors(const HelmCoef& hc, int set, int ny, double pmBeta, T* __restrict__ tab) {
  T* col = tab + (set ? MT_A1 : MT_A0);
  double cpp = 0.0;
  for (int j = 0; j < ny; ++j) {
    double a, b, c;
    helm_abc(hc, set, pmBeta, j, a, b, c);
    const double rm = 1.0 / (j == 0 ? b : b - a * cpp);
    const double cp = c * rm;
    col[(size_t)j * MT_W + 0] = (T)a;
    col[(size_t)j * MT_W + 1] = (T)rm;
    col[(size_t)j * MT_W + 2] = j == ny - 1 ? (T)0 : (T)cp;
    cpp = cp;
  }
}
// and downwards (twisted march): c, 1/m', a/m'
template <class T>
__device__ void update_down_factors(const HelmCoef& hc, int set, int ny, double pmBeta, T* __restrict__ dtab) {
  T* col = dtab + (set ? MD_C1 : MD_C0);
  double aqn = 0.0;
  for (int j = ny - 1; j >= 0; --j) {
    double a, b, c;
    helm_abc(hc, set, pmBeta, j, a, b, c);
    const double rq = 1.0 / (j == ny - 1 ? b : b - c * aqn);
    const double aq = a * rq;
    col[(size_t)j * MD_W + 0] = (T)c;
    col[(size_t)j * MD_W + 1] = (T)rq;
    col[(size_t)j * MD_W + 2] = (T)aq;
    aqn = aq;
  }
}

// Factor block of one periodic direction (layout: ch3d_march.cuh) for spacing r2 = 1/h^2
__device__ void update_ptri_block(double* F, int n, double r2, double pmBeta) {
  double *ppj = F, *v1 = F + (n + 1), *v2 = F + 2 * (n + 1), *abc = F + 3 * (n + 1);
  const double a = -pmBeta * r2, c = -pmBeta * r2, b = pmBeta * r2 * 2.0 + 1.0;
  double p1 = -c / b, p2 = -a / b;
  v1[1] = p1;
  v2[1] = p2;
  v2[n] = 1.0;
  ppj[1] = 0.0;
  for (int j = 2; j <= n - 1; ++j) {
    const double pp = 1.0 / (b + a * p1);
    p1 = -c * pp;
    p2 = -a * p2 * pp;
    ppj[j] = pp;
    v1[j] = p1;
    v2[j] = p2;
  }
  double w = 1.0;
  for (int j = n - 1; j >= 1; --j) {
    w = v2[j] + v1[j] * w;
    v2[j] = w;
  }
  abc[0] = a; abc[1] = b; abc[2] = c;
  abc[3] = c * v2[1] + a * v2[n - 1] + b;
}

template <class T> struct TableArgs {
  HelmCoef hc;
  Metrics<T> m;
  int nx, ny, nz;
  T* tab;                     // row tables of the substeps (null: none)
  bool walls;                 // y solves between walls: their factors in the row tables
  T* dtab;                    // their downward tables (null: not used)
  double* pf;                 // periodic factor blocks of the substeps (null: none)
  double r2x, r2y, r2z;       // 1/h^2 of the x, y and z sweeps; 0: no such sweep
  unsigned long long* slots;  // pmBeta the tables of each substep hold (all ones: none)
};

// The tables of substep ns for pmBeta, by the whole block; left as they are when
// they hold those already (constant dt).  Every chain of factors, sequential in its
// direction, has a warp: 0 to 3 the Helmholtz sets upwards and downwards, 4 to 6 the
// periodic blocks.  The Helmholtz coefficients come through shared memory (smem, 5
// (ny + 1) values) up to kStagedRows rows: read from global memory row by row they
// cost 49 us at 64 rows.  A scheme forms the factors its solves read: none for the
// explicit one, whose table holds the metrics alone (key 0).  Steps with a changing
// time step, before with all factors and the walls' chain after the periodic ones: ADI
// at 128^3 829 -> 807 us, periodic at 64^3 191 -> 166, explicit there 164 -> 120.
template <class T>
__device__ void update_tables(const TableArgs<T>& ta, int ns, double pmBeta, unsigned char* smem) {
  const int q = ns - 1, ny = ta.ny;
  const bool factors = ta.walls || ta.r2x > 0.0 || ta.r2y > 0.0 || ta.r2z > 0.0;
  const unsigned long long bits = (unsigned long long)__double_as_longlong(factors ? pmBeta : 0.0);
  if (ta.slots[q] == bits) return;  // uniform: every thread reads it before thread 0 writes below
  HelmCoef hc = ta.hc;
  if (ta.walls && ny <= kStagedRows) {
    double* const co = reinterpret_cast<double*>(smem);
    const double* src[5] = {ta.hc.ap2cForCN, ta.hc.am2cForCN, ta.hc.ap2p, ta.hc.ac2p, ta.hc.am2p};
    const double** dst[5] = {&hc.ap2cForCN, &hc.am2cForCN, &hc.ap2p, &hc.ac2p, &hc.am2p};
    for (int v = 0; v < 5; ++v) {
      double* o = co + (size_t)v * (ny + 1);
      for (int j = threadIdx.x; j <= ny; j += blockDim.x) o[j] = src[v][j];
      *dst[v] = o;
    }
  }
  __syncthreads();
  T* const tab = ta.tab + (size_t)q * ny * MT_W;
  if ((threadIdx.x & 31) == 0) {
    const int who = threadIdx.x >> 5, set = who & 1;
    if (who < 2) {
      if (ta.walls) update_row_factors(hc, set, ny, pmBeta, tab);
    } else if (who < 4) {
      if (ta.dtab) update_down_factors(hc, set, ny, pmBeta, ta.dtab + (size_t)q * ny * MD_W);
    } else if (ta.pf) {
      const int d = who - 4;  // x, z, y
      const double r2 = d == 0 ? ta.r2x : d == 1 ? ta.r2z : d == 2 ? ta.r2y : 0.0;
      double* F = ta.pf + (size_t)q * ptri_doubles(ta.nx, ny, ta.nz);
      if (r2 > 0.0)
        update_ptri_block(d == 0 ? F : d == 1 ? F + ptri_stride(ta.nx) : F + ptri_stride(ta.nx) + ptri_stride(ta.nz),
                          d == 0 ? ta.nx : d == 1 ? ta.nz : ny, r2, pmBeta);
    }
  }
  const Metrics<T>& m = ta.m;
  for (int j = threadIdx.x; j < ny; j += blockDim.x) {
    const int jc = j + 1;
    T* row = tab + (size_t)j * MT_W;
    row[MT_IY1] = m.yinterp[jc]; row[MT_IY3] = m.yinterp[jc + 1];
    row[MT_RDYP] = m.rdyp[jc]; row[MT_RDYC] = m.rdyc[jc];
    row[MT_AP2C] = m.ap2c[jc]; row[MT_AC2C] = m.ac2c[jc]; row[MT_AM2C] = m.am2c[jc];
    row[MT_AP2P] = m.ap2p[jc]; row[MT_AC2P] = m.ac2p[jc]; row[MT_AM2P] = m.am2p[jc];
  }
  __syncthreads();
  if (threadIdx.x == 0) ta.slots[q] = bits;
}

// The tables that belong to the current scalars, for the stage entry points: a host
// may call a stage whose substep's coefficients were never set up (after an upload
// they are zero and ns is 1).
template <class T>
__global__ void __launch_bounds__(kSetupThreads) k_tables(const DevScalars* __restrict__ sc, TableArgs<T> ta) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  if (sc->status) return;
  update_tables(ta, sc->ns, sc->pmBeta, smem_raw);
}

template <class T>
__global__ void __launch_bounds__(kSetupThreads) k_substep(DevScalars* sc, const double* __restrict__ part, int npart,
                                                           double* __restrict__ red, SubstepPar p, TableArgs<T> ta) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double sh[kSetupThreads / 32];
  __shared__ double beta;
  // read before the sums, so that thread 0 makes no further round trip to memory
  const int itime0 = sc->itime;
  const double uddx = __longlong_as_double((long long)sc->uddx), dt0 = sc->dt, time0 = sc->SimTime,
               pgaver0 = p.ns == 1 ? 0.0 : sc->PrGradAver;
  if (sc->status) return;
  double s1;
  if (!grid_sum(part, npart, red, &sc->ticket, sh, s1)) return;
  if (threadIdx.x == 0) {
    double dt = dt0;
    if (p.begin) {  // src/CFD_2nd/m_ChannelSystem.f90:81-88 (CalcMaxCFL result -> cflmp, dt)
      sc->itime = itime0 + 1;
      sc->cflmp = uddx * dt0;
      dt = p.dtMax;
      if (p.iCFL == 1) {
        const double d = p.CFLc / uddx;
        dt = d < p.dtMax ? d : p.dtMax;
      }
      sc->dt = dt;
    }
    // src/CFD_2nd/m_Parameters.f90:329-342 (PMcoeUpdate)
    const double pmAlpha = p.alp * dt;
    sc->pmGamma = p.gam * dt;
    sc->pmTheta = p.the * dt;
    sc->pmAlpha = pmAlpha;
    beta = 0.5 * p.alp * p.xnu * dt;
    sc->pmBeta = beta;
    sc->SimTime = time0 + dt * p.alp;
    sc->pmAlphaC = p.alp;
    sc->pmBetaT = 0.5 * p.alp * dt;
    sc->ns = p.ns;
    sc->divmax1 = 0ull;
    double pg = 0.0;  // this substep's mean pressure gradient
    if (p.IsUxConst && p.order == 4) {
      // the partial sums are those of the mean viscous stress (src/CFD_4th/m_TScheme.f90:364-377)
      pg = p.xnu * (s1 / p.nxnz + p.visc_wall) / p.yly;
      sc->PrGradNow = pg;
      sc->dpmdxns = -(pmAlpha * pg);  // RhsX - pmAlpha*dpmdxns
    } else if (p.IsUxConst) {
      // the bulk constraint of src/CFD_2nd/m_TSchemePIMP_inc.f90:60-74 from the sums of the current ux
      const double s1tot1 = s1 * p.norm_bulk;
      pg = (p.ubulk - s1tot1) / dt;
      sc->s1tot1 = s1tot1;
      sc->dpmdxns = p.alp * (p.ubulk - s1tot1);
      sc->PrGradNow = pg;
    } else {
      sc->dpmdxns = 0.0;
    }
    sc->PrGradAver = pgaver0 + p.alp * pg;
    if (p.last) {  // the maxima the diagnostics of this step accumulate
      sc->divmax2 = 0ull;
      sc->vmax[0] = sc->vmax[1] = sc->vmax[2] = 0ull;
      sc->uddx = 0ull;
    }
  }
  if (!ta.tab) return;
  __syncthreads();
  update_tables(ta, p.ns, beta, smem_raw);
}

// src/CFD_2nd/m_ChannelSystem.f90:127-130 (limit checks after the step) and
// CalcUxAver (src/CFD_2nd/m_Tools.f90:250-270) from partial sums.
__global__ void __launch_bounds__(kSetupThreads) k_step_end(DevScalars* sc, const double* __restrict__ part, int npart,
                                                            double* __restrict__ red, double norm_uxm, double div_limit,
                                                            double vel_limit) {
  __shared__ double sh[kSetupThreads / 32];
  if (sc->status) return;
  double s;
  if (!grid_sum(part, npart, red, &sc->ticket, sh, s) || threadIdx.x != 0) return;
  sc->uxm = s * norm_uxm;
  const double d2 = __longlong_as_double((long long)sc->divmax2);
  const double v0 = __longlong_as_double((long long)sc->vmax[0]);
  const double v1 = __longlong_as_double((long long)sc->vmax[1]);
  const double v2 = __longlong_as_double((long long)sc->vmax[2]);
  const double vmin = fmin(v0, fmin(v1, v2));
  if (!(d2 <= div_limit)) sc->status = 1;        // NaN trips too
  else if (!(vmin <= vel_limit)) sc->status = 2;
}

// first level of the deterministic two-level sum of block partials
__global__ void __launch_bounds__(256) k_reduce_partials(const double* __restrict__ in, int n, double* __restrict__ out) {
  __shared__ double red[256];
  const int nb = gridDim.x;
  const int chunk = (n + nb - 1) / nb;
  const int lo = blockIdx.x * chunk, hi = min(n, lo + chunk);
  double s = 0.0;
  for (int q = lo + threadIdx.x; q < hi; q += blockDim.x) s += in[q];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = red[0];
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
size_t march_table_bytes(int ny) {
  return (size_t)kMarchTables * ny * (MT_W + MD_W) * sizeof(double) + kMarchTables * sizeof(unsigned long long);
}
cudaError_t march_table_reset(ch3d_ctx* c) {
  return cudaMemsetAsync(march_beta_slots(c->mtab, c->ny), 0xff, kMarchTables * sizeof(unsigned long long),
                         c->stream);
}

cudaError_t launch_reduce_partials(ch3d_ctx* c, const double* in, int n, double* out) {
  k_reduce_partials<<<CH3D_NRED, 256, 0, c->stream>>>(in, n, out);
  return cudaGetLastError();
}

// One block up to 4096 partial sums, all in flight at once, else CH3D_NRED.
static unsigned setup_blocks(int n) { return n <= kSumPer * kSetupThreads ? 1u : (unsigned)CH3D_NRED; }

template <class T> static TableArgs<T> table_args(ch3d_ctx* c) {
  TableArgs<T> ta;
  ta.hc = helm_coef(c);
  ta.m = c->cfg.LES_type == 0 ? metrics_of<T>(c) : Metrics<T>();
  if constexpr (sizeof(T) == 8)
    if (c->cfg.LES_type > 0) ta.m = c->m64full;
  ta.nx = c->nx; ta.ny = c->ny; ta.nz = c->nz;
  // the eddy-viscosity closures form their own coefficients
  ta.tab = c->cfg.LES_type == 0 || les_const(c) ? (T*)c->mtab : nullptr;
  ta.pf = c->pfac;
  const bool fimp = c->cfg.order == 2 && c->cfg.IsImplicit == 2;
  ta.r2x = fimp ? c->rdx2 : 0.0;
  ta.r2z = fimp ? c->rdz2 : 0.0;
  ta.r2y = y_periodic(c) && c->cfg.IsImplicit != 0 ? c->rdy2 : 0.0;
  ta.walls = ta.tab && !y_periodic(c) && c->cfg.IsImplicit != 0;
  ta.dtab = ta.tab && ((c->march && !march_rows_path(c)) || c->cfg.order == 4) && march_twisted(c) ? march_down_tables<T>(c->mtab, c->ny) : nullptr;
  ta.slots = march_beta_slots(c->mtab, c->ny);
  return ta;
}
template <class T> static size_t table_smem(const ch3d_ctx* c, const TableArgs<T>& ta) {
  return ta.walls && c->ny <= kStagedRows ? (size_t)5 * (c->ny + 1) * sizeof(double) : 0;
}

template <class T> static cudaError_t substep_t(ch3d_ctx* c, int ns, bool whole_step) {
  SubstepPar p;
  p.ns = ns;
  p.begin = whole_step && ns == 1;
  p.last = whole_step && ns == c->iadvance;
  p.gam = c->gam[ns - 1]; p.the = c->the[ns - 1]; p.alp = c->alp[ns - 1];
  p.iCFL = c->cfg.iCFL; p.IsUxConst = c->cfg.IsUxConst; p.order = c->cfg.order;
  p.CFLc = c->cfg.CFLc; p.dtMax = c->cfg.dtMax; p.xnu = c->cfg.xnu; p.ubulk = c->cfg.ubulk;
  p.norm_bulk = 1.0 / ((double)c->nx * (double)c->nz) / (c->cfg.ybulk2 - c->cfg.ybulk1);
  p.nxnz = (double)(c->nx * c->nz);
  p.yly = c->cfg.yly;
  p.visc_wall = c->visc_wall;
  const TableArgs<T> ta = table_args<T>(c);
  // the partials of the bulk sums or of the mean viscous stress (the projection or k_bulk_march)
  const int np = c->npart_m;
  k_substep<T><<<setup_blocks(np), kSetupThreads, table_smem(c, ta), c->stream>>>(c->sc, c->part, np, c->red1, p, ta);
  return cudaGetLastError();
}
cudaError_t launch_substep_setup(ch3d_ctx* c, int ns, bool whole_step) {
  // LES: FP64 coefficients on either field type
  return c->fp32 && c->cfg.LES_type == 0 ? substep_t<float>(c, ns, whole_step) : substep_t<double>(c, ns, whole_step);
}

template <class T> static cudaError_t tables_t(ch3d_ctx* c) {
  const TableArgs<T> ta = table_args<T>(c);
  if (!ta.tab) return cudaSuccess;
  k_tables<T><<<1, kSetupThreads, table_smem(c, ta), c->stream>>>(c->sc, ta);
  return cudaGetLastError();
}
cudaError_t launch_tables(ch3d_ctx* c) {
  return c->fp32 && c->cfg.LES_type == 0 ? tables_t<float>(c) : tables_t<double>(c);
}

cudaError_t launch_step_end(ch3d_ctx* c) {
  const double norm = 1.0 / ((double)c->nx * (double)c->nz) / c->cfg.yly;
  // part2: written by the fused projection (march layout) or by k_diag
  const int np = march_diag_fusable(c) ? c->npart_m : diag_npart(c);
  k_step_end<<<setup_blocks(np), kSetupThreads, 0, c->stream>>>(c->sc, c->part2, np, c->red2, norm, c->cfg.div_limit, c->cfg.vel_limit);
  return cudaGetLastError();
}

}  // namespace ch3d
