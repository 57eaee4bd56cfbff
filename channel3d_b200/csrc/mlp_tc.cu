// mlp_tc.cu -- the learned subgrid-stress closure: a 10 -> 64 -> 64 -> 64 -> 6
// MLP (GELU in its tanh form, BF16 operands, FP32 accumulation) on the
// 5th-generation tensor cores.  The inference and training kernels issue tcgen05.mma from one thread of the CTA with operands
// in shared memory and the accumulator in tensor memory, read back with
// tcgen05.ld.  One CTA processes a tile of 128 points (M = 128, one TMEM
// lane per point).  The operand layout, the wrappers and the forward pass of
// a tile are in mlp_tc.cuh.
#include "mlp_tc.cuh"
#include "ch3d_common.cuh"

namespace ch3d_mlp {

// ---------------------------------------------------------------------------
// inference: X [B x 10] FP32 -> Y [B x 6] FP32
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(TILE, 6) k_mlp_fwd(const float* __restrict__ X, int B,
                                                     const float* __restrict__ P, float* __restrict__ Y,
                                                     int* __restrict__ status) {
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x;
  const long long pt = (long long)blockIdx.x * TILE + tid;
  const bool valid = pt < B;
  float x[NIN];
#pragma unroll
  for (int k = 0; k < NIN; ++k) x[k] = valid ? X[pt * NIN + k] : 0.f;
  fwd_prologue(smem, P, x);
  float y[NOUT];
  if (!fwd_layers(smem, y)) {
    if (tid == 0) atomicExch(status, 1);
    return;
  }
  if (valid)
    for (int c = 0; c < NOUT; ++c) Y[pt * NOUT + c] = y[c];
}

// ---------------------------------------------------------------------------
// Training: forward and backward of the mean-squared loss L = sum (Y - T)^2 /
// (B*6) in one persistent kernel, a CTA walking tiles of 128 points; per-CTA
// partial gradients part[blockIdx.x][NPARAM] and partial loss.
//
// Everything between the inputs and the gradients stays on the SM: the
// pre-activations Z1..Z3 in their MMA accumulators in tensor memory, the
// activations as BF16 tiles in shared memory, and the weight gradients
// accumulate in tensor memory over the CTA's tiles.  The weight gradients
// dW = dZ^T H_prev read the same dZ and H tiles (points x features) as the
// other GEMMs, as MN-major operands: the 8 x 16-byte core matrices of the
// K-major layout are those of the MN-major one with the roles of the two
// indices exchanged; likewise dH = dZ W reads the forward's weight operand.
// Warps w and w + 4 share the points of tensor-memory lanes 32 (w % 4).. and
// take 32 of the 64 columns each.
// ---------------------------------------------------------------------------
constexpr int kTrainThreads = 256;
constexpr int kTrainCtas = 148;  // at most one CTA per SM (it holds all 512 tensor-memory columns)
struct TrainSmem {
  static constexpr size_t X = 128;
  static constexpr size_t H1 = X + TILE * NINP * 2;
  static constexpr size_t DZ = H1 + 3 * TILE * NH * 2;   // 128 x 64, then as much again: as an M = 128 MN-major
  static constexpr size_t W1 = DZ + 2 * TILE * NH * 2;   // operand its features 64..127 are read and ignored
  static constexpr size_t RED = W1 + kPackedBytes;       // 4 warps x (3 x 64 + 16) column sums
  static constexpr size_t BYTES = 120 * 1024;            // more than half an SM: one CTA per SM
  static_assert(RED + 4 * (3 * NH + 16) * 4 <= BYTES, "shared memory");
};
// tensor-memory columns
constexpr uint32_t TZ = 0, TY = 192, TDH = 208, TG1 = 272, TG2 = 288, TG3 = 352, TG4 = 416;

// sum over the warp's 32 lanes of v[c] for c = 0..31; lane c returns column c
__device__ __forceinline__ float column_sums32(float (&v)[32], int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int c = 0; c < o; ++c) {
      const float keep = up ? v[c + o] : v[c], give = up ? v[c] : v[c + o];
      v[c] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  return v[0];
}

__global__ void __launch_bounds__(kTrainThreads, 1) k_mlp_train(const float* __restrict__ X, const float* __restrict__ T,
                                                                int B, const float* __restrict__ P,
                                                                float* __restrict__ part, float* __restrict__ lpart,
                                                                int* __restrict__ status) {
  extern __shared__ __align__(1024) unsigned char smem[];
  Smem* S = (Smem*)smem;
  unsigned char* XT = smem + TrainSmem::X;
  unsigned char* DZ = smem + TrainSmem::DZ;
  unsigned char* WB = smem + TrainSmem::W1;  // the parameter image, laid out from FwdSmem::W1 on
  unsigned char* const Wop[4] = {WB, WB + (FwdSmem::W2 - FwdSmem::W1), WB + (FwdSmem::W3 - FwdSmem::W1),
                                 WB + (FwdSmem::W4 - FwdSmem::W1)};
  const float* bs = (const float*)(WB + (FwdSmem::BIAS - FwdSmem::W1));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row = (warp & 3) * 32 + lane, half = warp >> 2, c0 = half * 32;
  if (tid == 0) { mbar_init(&S->bar, 1); S->err = 0; }
  if (warp == 0) { tmem_alloc(&S->tmem, 512); tmem_relinquish(); }
  pack_params(WB, P);
  fence_async_smem();
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tm = S->tmem;
  const uint32_t lane_addr = tm + ((uint32_t)((warp & 3) * 32) << 16);
  uint32_t phase = 0;
  // operands written -> MMAs issued by one thread -> their completion; false on an expired wait (uniform)
  auto run_mmas = [&](auto issue) {
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    if (tid == 0) {
      issue();
      mma_commit(&S->bar);
    }
    const bool ok = __syncthreads_or(mbar_wait(&S->bar, phase) ? 0 : 1) == 0;
    phase ^= 1;
    if (ok) fence_after();
    return ok;
  };
  const float invn = 1.0f / ((float)B * (float)NOUT);
  float db[3][32];  // bias gradients of this thread's columns over its points
#pragma unroll
  for (int l = 0; l < 3; ++l)
#pragma unroll
    for (int c = 0; c < 32; ++c) db[l][c] = 0.f;
  float db4[NOUT] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, lsum = 0.f;
  const int ntiles = (int)(((long long)B + TILE - 1) / TILE);
  bool ok = true;
  uint32_t acc = 0;  // the first tile's weight-gradient MMAs overwrite the accumulators
  for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, acc = 1) {
    const long long pt = (long long)tile * TILE + row;
    const bool valid = pt < B;
    {
      float xp[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) xp[k] = valid && half * 8 + k < NIN ? __ldg(X + pt * NIN + half * 8 + k) : 0.f;
      st_bf16x8(XT, row, half * 8, TILE, xp);
    }
    float tq[NOUT];
#pragma unroll
    for (int c = 0; c < NOUT; ++c) tq[c] = valid && half == 0 ? __ldg(T + pt * NOUT + c) : 0.f;
    ok = run_mmas([&] { gemm_issue(tm + TZ, XT, Wop[0], NH, NINP); });
#pragma unroll 1
    for (int l = 0; l < 3 && ok; ++l) {
      unsigned char* H = smem + TrainSmem::H1 + l * TILE * NH * 2;
#pragma unroll 1
      for (int q0 = 0; q0 < 32; q0 += 16) {
        float a[16], h[16];
        tmem_ld<16>(lane_addr + TZ + l * NH + c0 + q0, a);
#pragma unroll
        for (int q = 0; q < 16; ++q) h[q] = gelu(a[q] + bs[l * NH + c0 + q0 + q]);
        st_bf16x8(H, row, c0 + q0, TILE, h);
        st_bf16x8(H, row, c0 + q0 + 8, TILE, h + 8);
      }
      ok = run_mmas([&] {
        if (l < 2) gemm_issue(tm + TZ + (l + 1) * NH, H, Wop[l + 1], NH, NH);
        else gemm_issue(tm + TY, H, Wop[3], NOUTP, NH);
      });
    }
    if (!ok) break;
    if (half == 0) {  // dY and the loss
      float a[16], d[16];
      tmem_ld<16>(lane_addr + TY, a);
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        d[c] = 0.f;
        if (valid && c < NOUT) {
          const float e = a[c] + bs[3 * NH + c] - tq[c];
          lsum += e * e;
          d[c] = 2.0f * e * invn;
          db4[c] += d[c];
        }
      }
      st_bf16x8(DZ, row, 0, TILE, d);
      st_bf16x8(DZ, row, 8, TILE, d + 8);
    }
    ok = run_mmas([&] {
      gemm_issue_t(tm + TG4, DZ, smem + TrainSmem::H1 + 2 * TILE * NH * 2, NH, acc);
      gemm_issue_bt(tm + TDH, DZ, Wop[3], NH, NOUTP, NOUTP);
    });
#pragma unroll
    for (int l = 2; l >= 0; --l) {
      if (!ok) break;
#pragma unroll
      for (int q0 = 0; q0 < 32; q0 += 16) {
        float a[16], d[16];
        tmem_ld<16>(lane_addr + TZ + l * NH + c0 + q0, a);
        tmem_ld<16>(lane_addr + TDH + c0 + q0, d);
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          d[q] = valid ? d[q] * gelu_d(a[q] + bs[l * NH + c0 + q0 + q]) : 0.f;
          db[l][q0 + q] += d[q];
        }
        st_bf16x8(DZ, row, c0 + q0, TILE, d);
        st_bf16x8(DZ, row, c0 + q0 + 8, TILE, d + 8);
      }
      ok = run_mmas([&] {
        if (l > 0) {
          gemm_issue_t(tm + (l == 2 ? TG3 : TG2), DZ, smem + TrainSmem::H1 + (l - 1) * TILE * NH * 2, NH, acc);
          gemm_issue_bt(tm + TDH, DZ, Wop[l], NH, NH, NH);
        } else {
          gemm_issue_t(tm + TG1, DZ, XT, NINP, acc);
        }
      });
    }
  }
  if (!ok) {
    if (tid == 0) atomicExch(status, 1);
  } else {
    float* G = part + (long long)blockIdx.x * NPARAM;
    float* red = (float*)(smem + TrainSmem::RED);
    constexpr int RW = 3 * NH + 16;  // per warp of points: the three layers' columns, then dY's and the loss
#pragma unroll
    for (int l = 0; l < 3; ++l) red[(warp & 3) * RW + l * NH + c0 + lane] = column_sums32(db[l], lane);
    if (half == 0) {
#pragma unroll
      for (int c = 0; c <= NOUT; ++c) {
        float v = c < NOUT ? db4[c] : lsum;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp * RW + 3 * NH + c] = v;
      }
    }
    __syncthreads();
    if (tid < 3 * NH + NOUT + 1) {
      const float v = red[tid] + red[RW + tid] + red[2 * RW + tid] + red[3 * RW + tid];
      if (tid < 3 * NH) G[(tid < NH ? OB1 : tid < 2 * NH ? OB2 : OB3) + tid % NH] = v;
      else if (tid < 3 * NH + NOUT) G[OB4 + tid - 3 * NH] = v;
      else lpart[blockIdx.x] = v;
    }
    // weight gradients: tensor-memory lane = output feature, column = input
    float w[16];
#pragma unroll 1
    for (int q0 = 0; q0 < 32; q0 += 16)
#pragma unroll 1
      for (int l = 1; l < 4; ++l) {
        tmem_ld<16>(lane_addr + (l == 1 ? TG2 : l == 2 ? TG3 : TG4) + c0 + q0, w);
        if (row < (l == 3 ? NOUT : NH)) {
          float* o = G + (l == 1 ? OW2 : l == 2 ? OW3 : OW4) + row * NH + c0 + q0;
#pragma unroll
          for (int c = 0; c < 16; ++c) o[c] = w[c];
        }
      }
    tmem_ld<16>(lane_addr + TG1, w);
    if (half == 0 && row < NH)
#pragma unroll
      for (int c = 0; c < NIN; ++c) G[OW1 + row * NIN + c] = w[c];
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) tmem_dealloc(tm, 512);
}

// fixed-order sum of the per-CTA partials, grad[q] = sum_b part[b][q]: a block
// of 32 parameters x 8 slices of the CTAs
__global__ void __launch_bounds__(256) k_mlp_reduce(const float* __restrict__ part, const float* __restrict__ lpart,
                                                    int nb, float* __restrict__ grad, float* __restrict__ loss) {
  __shared__ float red[8][32];
  const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
  const int q = blockIdx.x * 32 + lane;
  float s = 0.f;
  if (q <= NPARAM)
#pragma unroll 8
    for (int b = sl; b < nb; b += 8) s += q < NPARAM ? part[(long long)b * NPARAM + q] : lpart[b];
  red[sl][lane] = s;
  __syncthreads();
  if (sl == 0 && q <= NPARAM) {
    for (int r = 1; r < 8; ++r) s += red[r][lane];
    if (q < NPARAM) grad[q] = s;
    else *loss = s;
  }
}

// Adam (Kingma & Ba 2015) on the FP32 master parameters
__global__ void k_adam(float* __restrict__ P, const float* __restrict__ g, float* __restrict__ m,
                       float* __restrict__ v, float lr, float b1, float b2, float eps, float bc1, float bc2) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= NPARAM) return;
  const float gq = g[q];
  const float mq = b1 * m[q] + (1.f - b1) * gq;
  const float vq = b2 * v[q] + (1.f - b2) * gq * gq;
  m[q] = mq;
  v[q] = vq;
  P[q] -= lr * (mq / bc1) / (sqrtf(vq / bc2) + eps);
}

constexpr size_t SMEM_FWD = FwdSmem::BYTES;

// The expiry path of the bounded waits: one thread waits on an mbarrier that
// nothing arrives at (no MMA issued, no tensor memory held) and, when the
// wait gives up after `limit` polls, records the expiry in *status as the
// MLP kernels do.
__global__ void k_mlp_wait_check(unsigned limit, int* __restrict__ status) {
  __shared__ uint64_t bar;
  if (threadIdx.x != 0) return;
  mbar_init(&bar, 1);
  if (!mbar_wait(&bar, 0, limit)) atomicExch(status, 1);
}

}  // namespace ch3d_mlp

using namespace ch3d_mlp;

// One-time attribute set-up per device a process drives (cudaFuncSetAttribute
// applies to the current device only), under the library's set-up lock.
template <class F> static bool setup_on_current_device(ch3d::PerDevice& site, F&& setup) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  return ch3d::once_per_device(site, dev, setup) == cudaSuccess;
}

extern "C" {

static int train_ctas(int batch) {
  const long long nt = ((long long)batch + TILE - 1) / TILE;
  return (int)(nt < kTrainCtas ? nt : kTrainCtas);
}

// the partial gradients and losses of the training kernel's CTAs
CH3D_MLP_API size_t ch3d_mlp_workspace_bytes(int batch) {
  return (size_t)train_ctas(batch) * (NPARAM + 1) * sizeof(float) + 256;
}

CH3D_MLP_API int ch3d_mlp_wait_check(unsigned limit, int* status, void* stream) {
  if (!status || limit == 0) return 1;
  k_mlp_wait_check<<<1, 32, 0, (cudaStream_t)stream>>>(limit, status);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

CH3D_MLP_API int ch3d_mlp_forward(const float* X, int batch, const float* params, float* Y, int* status,
                                  void* stream) {
  if (!X || !params || !Y || !status || batch <= 0) return 1;
  static ch3d::PerDevice attr;
  if (!setup_on_current_device(attr, [] {
        cudaError_t r = cudaFuncSetAttribute(k_mlp_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_FWD);
        if (r == cudaSuccess) r = cudaFuncSetAttribute(k_mlp_fwd, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
        return r;
      }))
    return 2;
  k_mlp_fwd<<<(batch + TILE - 1) / TILE, TILE, SMEM_FWD, (cudaStream_t)stream>>>(X, batch, params, Y, status);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

CH3D_MLP_API int ch3d_mlp_grad(const float* X, const float* T, int batch, const float* params, void* work,
                               float* grad, float* loss, int* status, void* stream) {
  if (!X || !T || !params || !work || !grad || !loss || !status || batch <= 0) return 1;
  static ch3d::PerDevice attr;
  if (!setup_on_current_device(attr, [] {
        return cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TrainSmem::BYTES);
      }))
    return 2;
  cudaStream_t st = (cudaStream_t)stream;
  const int nb = train_ctas(batch);
  float* part = (float*)work;
  float* lpart = part + (size_t)nb * NPARAM;
  k_mlp_train<<<nb, kTrainThreads, TrainSmem::BYTES, st>>>(X, T, batch, params, part, lpart, status);
  k_mlp_reduce<<<(NPARAM + 1 + 31) / 32, 256, 0, st>>>(part, lpart, nb, grad, loss);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

CH3D_MLP_API int ch3d_mlp_adam(float* params, const float* grad, float* m, float* v, float lr, float beta1,
                               float beta2, float eps, int step, void* stream) {
  if (!params || !grad || !m || !v || step < 1) return 1;
  const float bc1 = 1.0f - powf(beta1, (float)step), bc2 = 1.0f - powf(beta2, (float)step);
  k_adam<<<(NPARAM + 255) / 256, 256, 0, (cudaStream_t)stream>>>(params, grad, m, v, lr, beta1, beta2, eps, bc1, bc2);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // extern "C"
