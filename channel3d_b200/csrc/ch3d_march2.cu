// ch3d_march2.cu -- the FP32 column march that stops at g (see ch3d_march.cu), two
// columns per thread.
//
// With one column per thread the march executes 10 warp instructions per cell,
// as many as the FP64 one on half the bytes, and was bound by instruction issue
// (56-71% of the issue slots at 50% of the DRAM bandwidth).  Here a thread owns
// the columns i and i+1 and works on pairs of FP32 values: the sm_100
// instructions add, mul and fma .f32x2 take two operands in a 64-bit register,
// and aligned pairs of the staged rows are single 8-byte reads.  The arithmetic
// is that of rhs2_cell, with the constants folded; the two face fluxes of a term are
// subtracted before they are scaled and added, so that the sum never holds a single
// flux (adding them one by one raised the pressure error of 768x384x576 runs by a fifth and more).  The old Hist of a thread's columns
// comes through shared memory as well, D + 1 rows ahead: two rows ahead in registers
// 256x192x256 took 193 us per launch, now 150; 768x384x576 1.81 ms, now 1.75.
#include "ch3d_march.cuh"

namespace ch3d {

// a pair of FP32 values (columns i and i+1)
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float x, float y) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ F2 f2(float x) { return f2(x, x); }
__device__ __forceinline__ float lo(F2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
  return x;
}
__device__ __forceinline__ float hi(F2 a) {
  float x, y;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a.v));
  return y;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// Tile of 64 x 4 columns, 128 threads; rows staged in 16-byte vectors with the x
// halo rounded up to 4 points, D rows ahead.
constexpr int M2_BZ = 4, M2_SX = 64 + 8, M2_PL = M2_SX * (M2_BZ + 2);
constexpr int M2_NS = (M2_PL / 4 + 127) / 128;  // staging vectors per thread and field
// rows, table entries, old Hist
constexpr size_t m2_smem(int D) {
  return (size_t)4 * (D + 4) * M2_PL * sizeof(float) + (size_t)(D + 4) * MT_W * sizeof(F2) + (size_t)3 * (D + 1) * 128 * sizeof(F2);
}

template <int D>
__global__ void __launch_bounds__(128, 4)
    k_rhs_march2(Geo<float> g, const float* __restrict__ tab, const float* __restrict__ ux,
                 const float* __restrict__ uy, const float* __restrict__ uz, const float* __restrict__ pr,
                 float* __restrict__ hx, float* __restrict__ hy, float* __restrict__ hz, float* __restrict__ gx,
                 float* __restrict__ gy, float* __restrict__ gz, const DevScalars* __restrict__ sc) {
  constexpr int SX = M2_SX, PL = M2_PL, RS = D + 4, NT = 128;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float (*ring)[RS][PL] = reinterpret_cast<float (*)[RS][PL]>(smem_raw);
  F2 (*trs)[MT_W] = reinterpret_cast<F2 (*)[MT_W]>(smem_raw + (size_t)4 * RS * PL * sizeof(float));  // entries twice
  unsigned long long (*hring)[3][NT] = reinterpret_cast<unsigned long long (*)[3][NT]>(&trs[RS][0]);  // the thread's own old Hist
  if (sc->status) return;
  const int nx = g.nx, ny = g.ny, nz = g.nz;
  const long long plane = (long long)nx * ny;
  tab += (size_t)(sc->ns - 1) * ny * MT_W;  // this substep's table
  const int tid = threadIdx.x, tx = tid & 31, tz = tid >> 5;
  auto slot = [](int r) { return (r + 1) % RS; };  // r >= -1
  long long so[M2_NS];
  auto issue_row = [&](int r) {
    const long long ro = (long long)r * nx;
    const int sl = slot(r);
#pragma unroll
    for (int q = 0; q < M2_NS; ++q) {
      const int s = (tid + q * NT) * 4;
      if (s < PL) {
        cp_async_el(reinterpret_cast<float4*>(&ring[0][sl][s]), reinterpret_cast<const float4*>(ux + so[q] + ro));
        cp_async_el(reinterpret_cast<float4*>(&ring[1][sl][s]), reinterpret_cast<const float4*>(uy + so[q] + ro));
        cp_async_el(reinterpret_cast<float4*>(&ring[2][sl][s]), reinterpret_cast<const float4*>(uz + so[q] + ro));
        cp_async_el(reinterpret_cast<float4*>(&ring[3][sl][s]), reinterpret_cast<const float4*>(pr + so[q] + ro));
      }
    }
    if (tid < 2 * MT_W)  // the row's table, each entry twice
      cp_async_el(reinterpret_cast<float*>(&trs[sl][0]) + tid, tab + (size_t)r * MT_W + (tid >> 1));
  };
  // wall ghost rows from the thread's own staged vectors (m_BC_and_Halo.f90:241-282)
  auto ghost_row = [&](int r) {
    const int sl = slot(r);
#pragma unroll
    for (int qv = 0; qv < M2_NS * 4; ++qv) {
      const int s = (tid + (qv / 4) * NT) * 4 + qv % 4;
      if (s >= PL) continue;
      if (r < 0) {
        const float u = ring[0][slot(0)][s], w = ring[2][slot(0)][s], v1 = ring[1][slot(1)][s];
        ring[0][sl][s] = g.bc.lo == -1 ? (float)(g.bc.ux_lo * 2.0) - u : u - (float)(g.bc.ux_lo * g.bc.dyp1);
        ring[1][sl][s] = (float)(g.bc.uy_lo * 2.0) - v1;
        ring[2][sl][s] = g.bc.lo == -1 ? (float)(g.bc.uz_lo * 2.0) - w : w - (float)(g.bc.uz_lo * g.bc.dyp1);
        ring[3][sl][s] = ring[3][slot(0)][s];
      } else {
        const int sn = slot(ny - 1);
        const float u = ring[0][sn][s], w = ring[2][sn][s];
        ring[0][sl][s] = g.bc.hi == -1 ? (float)(g.bc.ux_hi * 2.0) - u : (float)(g.bc.ux_hi * g.bc.dypN) + u;
        ring[1][sl][s] = (float)g.bc.uy_hi;
        ring[2][sl][s] = g.bc.hi == -1 ? (float)(g.bc.uz_hi * 2.0) - w : (float)(g.bc.uz_hi * g.bc.dypN) + w;
        ring[3][sl][s] = ring[3][sn][s];
      }
    }
  };
  const float pmA = (float)sc->pmAlpha;
  const F2 gam = f2((float)sc->pmGamma), the = f2((float)sc->pmTheta), beta2 = f2(2.f * (float)sc->pmBeta);
  const F2 dpm = f2((float)sc->dpmdxns);
  const F2 nax = f2(-pmA * g.rdx), naz = f2(-pmA * g.rdz), na = f2(-pmA);
  const F2 q1 = f2(0.25f * g.rdx), q3 = f2(0.25f * g.rdz), nq1 = f2(-0.25f * g.rdx), nq3 = f2(-0.25f * g.rdz);
  const F2 d1 = f2(0.5f * g.rdx), d3 = f2(0.5f * g.rdz);
  const F2 nux = f2(g.xnu * g.rdx2), nuz = f2(g.xnu * g.rdz2), m1 = f2(-1.f), m2 = f2(-2.f), p2 = f2(2.f);
  const int c0 = (tz + 1) * SX + 4 + 2 * tx;
  const int ntx = (nx + 63) / 64, ntiles = ntx * ((nz + M2_BZ - 1) / M2_BZ);
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int i0 = (tile % ntx) * 64, k0 = (tile / ntx) * M2_BZ;
    const int i = i0 + 2 * tx, k = k0 + tz;
    const bool act = i < nx && k < nz;  // nx even: both columns or none
#pragma unroll
    for (int q = 0; q < M2_NS; ++q) {
      const int s = (tid + q * NT) * 4;  // a vector never wraps: nx and i0 - 4 are multiples of 4
      int ig = (i0 - 4 + s % SX) % nx, kg = (k0 - 1 + s / SX) % nz;
      if (ig < 0) ig += nx;
      if (kg < 0) kg += nz;
      so[q] = s < PL ? ig + plane * kg : 0;
    }
    long long idx = act ? i + plane * k : 0;
    const bool hread = act && (float)sc->pmTheta != 0.f;  // pmTheta = 0: the old Hist does not enter
    auto issue_hist = [&](int r, int hsl, long long o) {
      if (hread && r < ny) {
        cp_async_el(&hring[hsl][0][tid], reinterpret_cast<const unsigned long long*>(hx + o));
        cp_async_el(&hring[hsl][1][tid], reinterpret_cast<const unsigned long long*>(hy + o));
        cp_async_el(&hring[hsl][2][tid], reinterpret_cast<const unsigned long long*>(hz + o));
      }
    };
#pragma unroll
    for (int r = 0; r <= D + 1; ++r) {
      if (r < ny) issue_row(r);
      if (r > 0) issue_hist(r - 1, r - 1, idx + (long long)(r - 1) * nx);
      cp_async_commit();
    }
    F2 e0 = f2(0.f), e1 = f2(0.f), e2 = f2(0.f);  // eliminated right-hand sides of the previous row
    auto stp = [](float* a, long long o, F2 v) { *reinterpret_cast<unsigned long long*>(a + o) = v.v; };
    int hsl = 0;  // Hist slot of row j
    for (int j = 0; j < ny; ++j, idx += nx) {
      cp_async_wait<D>();  // this thread's copies of rows <= j+1 are done
      if (j + 1 == ny) ghost_row(ny);
      if (j == 0) ghost_row(-1);
      __syncthreads();
      if (j + D + 2 < ny) issue_row(j + D + 2);
      F2 ho0 = f2(0.f), ho1 = f2(0.f), ho2 = f2(0.f);
      if (hread) { ho0.v = hring[hsl][0][tid]; ho1.v = hring[hsl][1][tid]; ho2.v = hring[hsl][2][tid]; }
      if (act) {
        const int s0 = slot(j - 1), s1 = slot(j), s2 = slot(j + 1);
        const F2* tr = trs[s1];
        auto at = [&](int a, int sl, int o) { return F2{*reinterpret_cast<const unsigned long long*>(&ring[a][sl][c0 + o])}; };
        auto right = [&](int a, int sl, int o, F2 c) { return f2(hi(c), ring[a][sl][c0 + o + 2]); };  // i+1 of both columns
        auto left = [&](int a, int sl, int o, F2 c) { return f2(ring[a][sl][c0 + o - 1], lo(c)); };   // i-1
        const F2 u = at(0, s1, 0), ujp = at(0, s2, 0), ujm = at(0, s0, 0), ukp = at(0, s1, SX), ukm = at(0, s1, -SX);
        const F2 v = at(1, s1, 0), vjp = at(1, s2, 0), vjm = at(1, s0, 0), vkp = at(1, s1, SX), vkm = at(1, s1, -SX);
        const F2 vjpkm = at(1, s2, -SX);
        const F2 w = at(2, s1, 0), wjp = at(2, s2, 0), wjm = at(2, s0, 0), wkp = at(2, s1, SX), wkm = at(2, s1, -SX);
        const F2 wjmkp = at(2, s0, SX);
        const F2 uip = right(0, s1, 0, u), uim = left(0, s1, 0, u), uipjm = right(0, s0, 0, ujm), uipkm = right(0, s1, -SX, ukm);
        const F2 vip = right(1, s1, 0, v), vim = left(1, s1, 0, v), vimjp = left(1, s2, 0, vjp);
        const F2 wip = right(2, s1, 0, w), wim = left(2, s1, 0, w), wimkp = left(2, s1, SX, wkp);
        const F2 p = at(3, s1, 0), pim = left(3, s1, 0, p), pjm = at(3, s0, 0), pkm = at(3, s1, -SX);
        const F2 IY1 = tr[MT_IY1], IY3 = tr[MT_IY3], one = f2(1.f);
        const F2 IY2 = one - IY1, IY4 = one - IY3;
        const F2 suc = f2(0.5f) * tr[MT_RDYP];
        // velocities interpolated in y at the lower and upper faces
        const F2 ul = fma(IY1, ujm, IY2 * u), uu = fma(IY3, u, IY4 * ujp);
        const F2 wl = fma(IY1, wjm, IY2 * w), wu = fma(IY3, w, IY4 * wjp);
        F2 r0, r1, r2;
        {  // RhsX
          const F2 sx = uip + uim;
          F2 c = fma(nux, fma(m2, u, sx), f2(g.g1));
          c = fma(nuz, fma(m2, u, ukp + ukm), c);
          c = fma((uip - uim) * fma(p2, u, sx), nq1, c);  // (u_ip + u)^2 - (u + u_im)^2
          c = fma(fma(v + vim, ul, m1 * ((vjp + vimjp) * uu)), suc, c);
          c = fma(fma(w + wim, u + ukm, m1 * ((wkp + wimkp) * (ukp + u))), q3, c);
          const F2 d22 = fma(tr[MT_AP2C], ujp, fma(tr[MT_AC2C], u, tr[MT_AM2C] * ujm));
          r0 = fma(gam, c, fma(the, ho0, fma(beta2, d22, fma(nax, p - pim, dpm))));
          stp(hx, idx, c);
        }
        {  // RhsY
          const F2 sx = vip + vim;
          const F2 rc = tr[MT_RDYC], qrc = f2(-0.25f) * rc;
          F2 c = fma(nux, fma(m2, v, sx), f2(g.g2));
          c = fma(nuz, fma(m2, v, vkp + vkm), c);
          c = fma(fma(ul, v + vim, m1 * (fma(IY1, uipjm, IY2 * uip) * (vip + v))), d1, c);
          c = fma((vjp - vjm) * fma(p2, v, vjp + vjm), qrc, c);
          c = fma(fma(wl, v + vkm, m1 * (fma(IY1, wjmkp, IY2 * wkp) * (vkp + v))), d3, c);
          const F2 d22 = fma(tr[MT_AP2P], vjp, fma(tr[MT_AC2P], v, tr[MT_AM2P] * vjm));
          r1 = fma(gam, c, fma(the, ho1, fma(beta2, d22, (na * rc) * (p - pjm))));
          stp(hy, idx, c);
        }
        {  // RhsZ
          const F2 sz = wkp + wkm;
          F2 c = fma(nux, fma(m2, w, wip + wim), f2(g.g3));
          c = fma(nuz, fma(m2, w, sz), c);
          c = fma(fma(u + ukm, w + wim, m1 * ((uip + uipkm) * (wip + w))), q1, c);
          c = fma(fma(v + vkm, wl, m1 * ((vjp + vjpkm) * wu)), suc, c);
          c = fma((wkp - wkm) * fma(p2, w, sz), nq3, c);  // (w_kp + w)^2 - (w + w_km)^2
          const F2 d22 = fma(tr[MT_AP2C], wjp, fma(tr[MT_AC2C], w, tr[MT_AM2C] * wjm));
          r2 = fma(gam, c, fma(the, ho2, fma(beta2, d22, naz * (p - pkm))));
          stp(hz, idx, c);
        }
        if (j == 0) r1 = f2(0.f);  // duy_ym: uy_ym is constant (Update_uy_ym_CH)
        e0 = (r0 - tr[MT_A0] * e0) * tr[MT_RM0];
        e1 = (r1 - tr[MT_A1] * e1) * tr[MT_RM1];
        e2 = (r2 - tr[MT_A0] * e2) * tr[MT_RM0];
        stp(gx, idx, fma(tr[MT_CP0], ujp, u + e0));
        stp(gy, idx, fma(tr[MT_CP1], vjp, v + e1));
        stp(gz, idx, fma(tr[MT_CP0], wjp, w + e2));
      }
      issue_hist(j + D + 1, hsl, idx + (long long)(D + 1) * nx);  // the slot just used
      cp_async_commit();
      hsl = hsl == D ? 0 : hsl + 1;
    }
    cp_async_wait<0>();
    __syncthreads();  // the ring is refilled by the next tile's prologue
  }
}

template <int D> static cudaError_t march2_t(ch3d_ctx* c, long long ntiles, int bps) {
  static PerDevice site;  // per instance
  const cudaError_t e = smem_limit_once(site, c->device, k_rhs_march2<D>, m2_smem(D));
  if (e != cudaSuccess) return e;
  float** f = (float**)c->f;
  const long long cap = (long long)bps * sm_count(c->device);  // persistent blocks
  k_rhs_march2<D><<<(unsigned)(ntiles < cap ? ntiles : cap), 128, m2_smem(D), c->stream>>>(
      make_geo<float>(c), (const float*)c->mtab, f[0], f[1], f[2], f[3], f[4], f[5], f[6], f[12], f[13], f[14], c->sc);
  return cudaGetLastError();
}
// nx is a multiple of 128 here (x lengths with a register plan), so rows are whole 16-byte
// vectors.  Three rows ahead and three blocks per SM, or two and four where that takes
// fewer rounds of tiles: 256 tiles 150 / 162 us (256x192x256), 512 tiles 108 / 98
// (512x64x256), 864 tiles 147 / 163 (768x64x288), 1728 tiles 1767 / 1748 (768x384x576).
cudaError_t launch_rhs_march2(ch3d_ctx* c) {
  const long long ntiles = (long long)((c->nx + 63) / 64) * ((c->nz + M2_BZ - 1) / M2_BZ), nsm = sm_count(c->device);
  const long long rounds3 = (ntiles + 3 * nsm - 1) / (3 * nsm), rounds4 = (ntiles + 4 * nsm - 1) / (4 * nsm);
  return rounds3 <= rounds4 ? march2_t<3>(c, ntiles, 3) : march2_t<2>(c, ntiles, 4);
}

}  // namespace ch3d
