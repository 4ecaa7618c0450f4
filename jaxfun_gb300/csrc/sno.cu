// CUDA-core kernels of the spectral neural operator that are too small or too
// irregular for the tensor cores: per-mode channel mixing (forward/backward),
// bias gradients, the loss and its gradient, and the Adam update.
#include <algorithm>
#include <cuda_bf16.h>
#include <math.h>

#include "jfg_internal.cuh"

namespace jfg {
namespace {

constexpr int MAXC = 64;  // channel width limit of the mode-mixing kernels

// Per-mode channel mixing.  Forward: out[b][co][q] = sum_ci R[q][co][ci] x[b][q][ci].
// Backward: dx[b][ci][q] = sum_co R[q][co][ci] dy[b][q][co] and
// dR[q][co][ci] = sum_b dy[b][q][co] x[b][q][ci].  Sums run in ascending order.
//
// A block owns MB neighbouring modes and works through (32 samples, mode)
// steps: the mode's R and the samples' rows are copied to shared memory one
// step ahead (cp.async), 256 threads hold 2 x 4 (sample, channel) and 4 x 4
// (dR) register tiles, and bf16 results of the MB modes are gathered in shared
// memory so that each (sample, channel) gets MB modes in one store.  Bound by
// shared-memory reads, about 10 wavefronts per 32 FMA instructions.  32 samples,
// 1024 modes, 64 channels: forward 78 -> 21 us, backward 108 -> 32 us against
// one mode (forward: eight) at a time with a barrier or two per sample.
constexpr int MM_B = 32;             // samples per step
constexpr int MM_T = 256;
constexpr int MM_LD = MAXC + 4;      // 16-byte rows, neighbouring rows 4 banks apart
constexpr int MM_Q = 8;              // the forward call takes multiples of this

struct MixStage {
  float R[MAXC][MM_LD];
  float x[MM_B][MM_LD];
  float d[MM_B][MM_LD];
};
template <int MB>
struct MixSmem {
  MixStage st[2];
  __nv_bfloat16 o[MM_B * MAXC][MB];
};

__device__ __forceinline__ void cp16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

// rows of C floats at src + r * ld into dst[r][0..C)
__device__ __forceinline__ void mix_copy(float (*dst)[MM_LD], const float* src, long long ld,
                                         int rows, int C, bool vec) {
  if (vec) {
    const int c4 = C / 4;
    for (int i = threadIdx.x; i < rows * c4; i += MM_T) {
      const int r = i / c4, c = (i - r * c4) * 4;
      cp16(&dst[r][c], src + r * ld + c);
    }
  } else {
    for (int i = threadIdx.x; i < rows * C; i += MM_T) {
      const int r = i / C, c = i - r * C;
      dst[r][c] = src[r * ld + c];
    }
  }
}

template <int MB, bool BWD>
__global__ void __launch_bounds__(MM_T, 2)
    k_modemix(int batch, int nq, int C, int per_block, int vec, int wide,
              const float* __restrict__ R,
              const float* __restrict__ x, const float* __restrict__ dy,
              __nv_bfloat16* __restrict__ out, float* __restrict__ dR) {
  extern __shared__ __align__(16) uint8_t mix_smem[];
  MixSmem<MB>& sm = *reinterpret_cast<MixSmem<MB>*>(mix_smem);
  const int t = threadIdx.x;
  const int q0 = blockIdx.x * MB;
  const int b0 = blockIdx.y * per_block, b1 = min(batch, b0 + per_block);
  const int nm = min(MB, nq - q0);
  const int steps = (b1 - b0 + MM_B - 1) / MM_B * nm;  // (samples, mode), modes inside
  // channels past C are zero
  for (int i = t; i < (int)(sizeof(sm.st) / 16); i += MM_T)
    reinterpret_cast<float4*>(&sm.st[0])[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  auto fetch = [&](int step) {
    MixStage& s = sm.st[step & 1];
    const int b = b0 + step / nm * MM_B, q = q0 + step % nm;
    const int n = min(MM_B, b1 - b);
    mix_copy(s.R, R + (long long)q * C * C, C, C, C, vec);
    mix_copy(s.x, x + ((long long)b * nq + q) * C, (long long)nq * C, n, C, vec);
    if (BWD) mix_copy(s.d, dy + ((long long)b * nq + q) * C, (long long)nq * C, n, C, vec);
  };
  float acc[BWD ? MB : 1][4][4];
#pragma unroll
  for (int m = 0; m < (BWD ? MB : 1); ++m)
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[m][i / 4][i % 4] = 0.f;
  const int lo = t & 15, hi = t >> 4;
  if (steps > 0) fetch(0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int bb = b0, step = 0; bb < b1; bb += MM_B) {
    const int n = min(MM_B, b1 - bb);
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      if (m >= nm) break;
      if (step + 1 < steps) fetch(step + 1);
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      const MixStage& s = sm.st[step & 1];
      ++step;
      // samples 2 hi, 2 hi + 1; channels 4 lo + j (backward), lo + 16 j (forward:
      // rows of R that lie in different banks)
      float v[2][4] = {};
      const float(*in)[MM_LD] = BWD ? s.d : s.x;
#pragma unroll 4
      for (int c = 0; c < MAXC; c += 4) {
        if (c >= C) break;
        float y[2][4], r[4][4];
#pragma unroll
        for (int u = 0; u < 2; ++u)
          *reinterpret_cast<float4*>(y[u]) = *reinterpret_cast<const float4*>(&in[2 * hi + u][c]);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<float4*>(r[j]) = *reinterpret_cast<const float4*>(
              BWD ? &s.R[c + j][4 * lo] : &s.R[lo + 16 * j][c]);
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int j = 0; j < 4; ++j) v[u][j] = fmaf(BWD ? r[k][j] : r[j][k], y[u][k], v[u][j]);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          sm.o[(2 * hi + u) * MAXC + (BWD ? 4 * lo + j : lo + 16 * j)][m] = __float2bfloat16(v[u][j]);
      if (BWD) {
#pragma unroll 4
        for (int b = 0; b < n; ++b) {
          float xv[4], dv[4];
          *reinterpret_cast<float4*>(xv) = *reinterpret_cast<const float4*>(&s.x[b][4 * lo]);
          *reinterpret_cast<float4*>(dv) = *reinterpret_cast<const float4*>(&s.d[b][4 * hi]);
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[m][i][j] = fmaf(dv[i], xv[j], acc[m][i][j]);
        }
      }
      __syncthreads();  // the stage may be filled again
    }
    // MB modes of every (sample, channel); the next results come after a barrier
    for (int i = t; i < n * C; i += MM_T) {
      const int b = i / C, c = i - b * C;
      const __nv_bfloat16* o = sm.o[b * MAXC + c];
      __nv_bfloat16* g = out + ((long long)(bb + b) * C + c) * nq + q0;
      if (MB == 4 && wide)
        *reinterpret_cast<uint2*>(g) = *reinterpret_cast<const uint2*>(o);
      else
        for (int m = 0; m < nm; ++m) g[m] = o[m];
    }
  }
  if (BWD) {
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      if (m >= nm) break;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int co = 4 * hi + i;
        if (co >= C) continue;
        float* g = dR + ((long long)(q0 + m) * C + co) * C + 4 * lo;
        if (vec) {
          if (4 * lo < C)
            *reinterpret_cast<float4*>(g) =
                make_float4(acc[m][i][0], acc[m][i][1], acc[m][i][2], acc[m][i][3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (4 * lo + j < C) g[j] = acc[m][i][j];
        }
      }
    }
  }
}

template <int MB, bool BWD>
int mix_launch(int groups, int per_block, int batch, int nq, int C, const float* R, const float* x,
               const float* dy, void* out, float* dR, cudaStream_t st) {
  static bool set[64] = {};  // per device; call before a capture
  int dev = 0;
  JFG_CUDA_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return JFG_ERR_UNSUPPORTED;
  if (!set[dev]) {
    JFG_CUDA_TRY(cudaFuncSetAttribute(k_modemix<MB, BWD>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)sizeof(MixSmem<MB>)));
    set[dev] = true;
  }
  // copies of 16 bytes; stores of MB modes at once
  const int vec = C % 4 == 0 && (((uintptr_t)R | (uintptr_t)x | (uintptr_t)dy | (uintptr_t)dR) & 15) == 0;
  const int wide = nq % MB == 0 && ((uintptr_t)out & 7) == 0;
  k_modemix<MB, BWD><<<dim3((nq + MB - 1) / MB, groups), MM_T, sizeof(MixSmem<MB>), st>>>(
      batch, nq, C, per_block, vec, wide, R, x, dy, (__nv_bfloat16*)out, dR);
  JFG_LAUNCHED();
  return JFG_OK;
}

// Four modes a block (8-byte stores), one where that would leave SMs idle.
constexpr int MM_FEW = 512;

__global__ void k_colsum_bf16(long long rows, int n, const __nv_bfloat16* __restrict__ src,
                              float* __restrict__ out, long long rows_per_block) {
  const int c = threadIdx.x;
  if (c >= n) return;
  const long long r0 = blockIdx.x * rows_per_block;
  const long long r1 = min(rows, r0 + rows_per_block);
  float s = 0.f;
  for (long long r = r0; r < r1; ++r) s += __bfloat162float(src[r * n + c]);
  atomicAdd(out + c, s);
}

__global__ void k_adam(long long n, float* __restrict__ p, const float* __restrict__ g,
                       float* __restrict__ m, float* __restrict__ v, float lr, float b1, float b2,
                       float eps, float c1, float c2, __nv_bfloat16* __restrict__ pb,
                       __nv_bfloat16* __restrict__ ptb, int rows, int cols) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pi;
    const __nv_bfloat16 h = __float2bfloat16(pi);
    if (pb) pb[i] = h;
    if (ptb && rows > 0 && cols > 0) {
      const long long r = i / cols, c = i % cols;
      ptb[c * rows + r] = h;
    }
  }
}

__global__ void k_mse(long long rows, const float* __restrict__ pred, long long ld,
                      const float* __restrict__ target, __nv_bfloat16* __restrict__ dq,
                      __nv_bfloat16* __restrict__ dqt, float* __restrict__ loss) {
  __shared__ float red[32];
  float s = 0.f;
  const float inv = 1.0f / (float)rows;
  for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < rows;
       r += (long long)gridDim.x * blockDim.x) {
    const float e = pred[r * ld] - target[r];
    s += e * e;
    const __nv_bfloat16 h = __float2bfloat16(e * inv);
    const __nv_bfloat16 z = __float2bfloat16(0.f);
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      if (dq) dq[r * 16 + c] = c == 0 ? h : z;
      if (dqt) dqt[c * rows + r] = c == 0 ? h : z;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
    atomicAdd(loss, t);
  }
}

inline int nblocks(long long n, int cap) {
  long long b = (n + 255) / 256;
  if (b > cap) b = cap;
  return (int)(b < 1 ? 1 : b);
}

}  // namespace
}  // namespace jfg

using namespace jfg;

extern "C" int jfg_sno_modemix_fwd(int batch, int nmodes, int C, const float* R, const float* x,
                                   void* out, void* stream) {
  if (batch < 0 || nmodes < 0 || C < 1 || C > MAXC || !R || !x || !out) return JFG_ERR_ARG;
  if (batch == 0 || nmodes == 0) return JFG_OK;
  if (nmodes % MM_Q != 0) return JFG_ERR_ARG;
  // samples spread over the blocks' second index where modes are few
  const int mblocks = nmodes >= MM_FEW ? nmodes / 4 : nmodes;
  int sms = 0;
  JFG_TRY(sm_count(&sms));
  const int groups = std::max(1, std::min((2 * sms + mblocks - 1) / mblocks, (batch + MM_B - 1) / MM_B));
  const int per_block = (batch + groups - 1) / groups;
  auto* f = nmodes >= MM_FEW ? mix_launch<4, false> : mix_launch<1, false>;
  return f((batch + per_block - 1) / per_block, per_block, batch, nmodes, C, R, x, nullptr, out,
           nullptr, (cudaStream_t)stream);
}

extern "C" int jfg_sno_modemix_bwd(int batch, int nmodes, int C, const float* R, const float* x,
                                   const float* dy, void* dx, float* dR, void* stream) {
  if (batch < 0 || nmodes < 0 || C < 1 || C > MAXC || !R || !x || !dy || !dx || !dR)
    return JFG_ERR_ARG;
  if (nmodes == 0) return JFG_OK;
  auto* f = nmodes >= MM_FEW ? mix_launch<4, true> : mix_launch<1, true>;
  return f(1, batch, batch, nmodes, C, R, x, dy, dx, dR, (cudaStream_t)stream);
}

extern "C" int jfg_colsum_bf16(long long rows, int n, const void* src, float* out,
                               int accumulate, void* stream) {
  if (rows < 0 || n < 1 || n > 1024 || !src || !out) return JFG_ERR_ARG;
  if (!accumulate) JFG_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(float) * n, (cudaStream_t)stream));
  if (rows == 0) return JFG_OK;
  const long long rpb = 256;
  const long long nb = (rows + rpb - 1) / rpb;
  if (nb > 2147483647LL) return JFG_ERR_ARG;
  k_colsum_bf16<<<(int)nb, ((n + 31) / 32) * 32, 0, (cudaStream_t)stream>>>(
      rows, n, (const __nv_bfloat16*)src, out, rpb);
  JFG_LAUNCHED();
  return JFG_OK;
}

extern "C" int jfg_adam_step(long long n, float* p, const float* g, float* m, float* v, float lr,
                             float beta1, float beta2, float eps, int step, void* p_bf16,
                             void* pt_bf16, int rows, int cols, void* stream) {
  if (n < 0 || !p || !g || !m || !v || step < 1) return JFG_ERR_ARG;
  if (pt_bf16 && ((long long)rows * cols != n)) return JFG_ERR_ARG;
  if (n == 0) return JFG_OK;
  const float c1 = 1.f - powf(beta1, (float)step);
  const float c2 = 1.f - powf(beta2, (float)step);
  k_adam<<<nblocks(n, 8192), 256, 0, (cudaStream_t)stream>>>(
      n, p, g, m, v, lr, beta1, beta2, eps, c1, c2, (__nv_bfloat16*)p_bf16,
      (__nv_bfloat16*)pt_bf16, rows, cols);
  JFG_LAUNCHED();
  return JFG_OK;
}

extern "C" int jfg_sno_mse(long long rows, const float* pred, long long ld_pred,
                           const float* target, void* dq, void* dqt, float* loss_out,
                           void* stream) {
  if (rows < 1 || !pred || !target || !loss_out || ld_pred < 1) return JFG_ERR_ARG;
  k_mse<<<nblocks(rows, 2048), 256, 0, (cudaStream_t)stream>>>(
      rows, pred, ld_pred, target, (__nv_bfloat16*)dq, (__nv_bfloat16*)dqt, loss_out);
  JFG_LAUNCHED();
  return JFG_OK;
}
