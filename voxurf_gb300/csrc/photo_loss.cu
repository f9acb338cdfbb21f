// The photometric training loss (run.py:604-627) and its gradients:
//   loss = w_main mse(rgb, target) + w_entropy H(p) + w_rgb0 mse(rgb0, target),
//   H(p) = -(p log p + (1 - p) log(1 - p)),  p = clamp(alphainv_last, 1e-6, 1 - 1e-6).
// As separate elementwise and reduction launches the loss of an 8192-ray batch
// was about 50 launches of 1-5 us, over a millisecond of host time in which the
// GPU waited; here it is one launch forward and one backward: the FP32 training
// step 3,145 -> 2,368 us.  Bound: latency (three tensors of 98 KB).  A thread
// sums its squares (at most 64) in FP32 and the threads' sums are added in 64
// bits, in a fixed order: with every addition in 64 bits the one block took 33
// us, 10 us now.  The gradients are formed as the elementwise chain forms them
// (the norm 2/n times the difference, times the upstream scalar).
#include <algorithm>

#include "common.cuh"

namespace vx {

constexpr int PL_THREADS = 1024;
constexpr int64_t PL_PER_BLOCK = 1 << 16;   // elements per block; one block finishes alone

// Sum over the block, in thread 0 (fixed order).
__device__ __forceinline__ double block_sum(double v, double (&warps)[PL_THREADS / 32]) {
  v = warp_sum(v);
  if (lane_id() == 0) warps[threadIdx.x >> 5] = v;
  __syncthreads();
  double s = 0.0;
  if (threadIdx.x < 32) s = warp_sum(warps[threadIdx.x]);
  __syncthreads();
  return s;
}

struct PhotoLoss {
  const float* rgb;
  const float* rgb0;           // null: no such term
  const float* target;
  int64_t n;
  const float* alphainv_last;  // null: no entropy term
  float w_main, w_rgb0, w_entropy;
};

// torch's clamp keeps a NaN.
__device__ __forceinline__ float clamp_p(float x) {
  return x < 1e-6f ? 1e-6f : (x > 1.f - 1e-6f ? 1.f - 1e-6f : x);
}

__device__ __forceinline__ float photo_value(const PhotoLoss& P, double s, double s0) {
  float loss = fmul(P.w_main, (float)(s / (double)P.n));
  if (P.alphainv_last) {
    const float p = clamp_p(*P.alphainv_last), q = 1.f - p;
    loss = fadd(loss, fmul(P.w_entropy, -fadd(fmul(p, logf(p)), fmul(q, logf(q)))));
  }
  if (P.rgb0) loss = fadd(loss, fmul((float)(s0 / (double)P.n), P.w_rgb0));
  return loss;
}

__global__ void __launch_bounds__(PL_THREADS) photo_loss_kernel(PhotoLoss P, double2* __restrict__ part,
                                                               float* __restrict__ loss) {
  __shared__ double warps[PL_THREADS / 32];
  float sf = 0.f, s0f = 0.f;
  const int64_t end = min(P.n, (int64_t)(blockIdx.x + 1) * PL_PER_BLOCK);
#pragma unroll 8
  for (int64_t i = (int64_t)blockIdx.x * PL_PER_BLOCK + threadIdx.x; i < end; i += PL_THREADS) {
    const float t = P.target[i], d = fsub(P.rgb[i], t);
    sf = fadd(sf, fmul(d, d));
    if (P.rgb0) {
      const float d0 = fsub(P.rgb0[i], t);
      s0f = fadd(s0f, fmul(d0, d0));
    }
  }
  const double s = block_sum((double)sf, warps), s0 = block_sum((double)s0f, warps);
  if (threadIdx.x == 0) {
    if (gridDim.x == 1) *loss = photo_value(P, s, s0);
    else part[blockIdx.x] = make_double2(s, s0);
  }
}

__global__ void __launch_bounds__(PL_THREADS) photo_loss_finish_kernel(PhotoLoss P, const double2* __restrict__ part,
                                                                      int n_part, float* __restrict__ loss) {
  __shared__ double warps[PL_THREADS / 32];
  double s = 0.0, s0 = 0.0;
  for (int i = threadIdx.x; i < n_part; i += PL_THREADS) {
    s += part[i].x;
    s0 += part[i].y;
  }
  s = block_sum(s, warps);
  s0 = block_sum(s0, warps);
  if (threadIdx.x == 0) *loss = photo_value(P, s, s0);
}

__global__ void __launch_bounds__(256) photo_loss_bwd_kernel(PhotoLoss P, const float* __restrict__ g,
                                                             float* __restrict__ d_rgb, float* __restrict__ d_rgb0,
                                                             float* __restrict__ d_alphainv, int64_t n_alphainv) {
  const float up = *g, norm = (float)(2.0 / (double)P.n);
  const float gm = fmul(up, P.w_main), g0 = fmul(up, P.w_rgb0);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x, at = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t i = at; i < P.n; i += stride) {
    const float t = P.target[i];
    d_rgb[i] = fmul(fmul(norm, fsub(P.rgb[i], t)), gm);
    if (P.rgb0) d_rgb0[i] = fmul(fmul(norm, fsub(P.rgb0[i], t)), g0);
  }
  if (!P.alphainv_last) return;
  for (int64_t i = at; i < n_alphainv; i += stride) {
    float d = 0.f;
    if (i == n_alphainv - 1) {
      const float x = *P.alphainv_last, p = clamp_p(x);
      if (x >= 1e-6f && x <= 1.f - 1e-6f) d = fmul(fmul(up, P.w_entropy), logf(1.f - p) - logf(p));
    }
    d_alphainv[i] = d;
  }
}

}  // namespace vx

using namespace vx;

extern "C" {

size_t vx_photo_loss_scratch_bytes(int64_t n) {
  const int64_t blocks = (std::max<int64_t>(n, 1) + PL_PER_BLOCK - 1) / PL_PER_BLOCK;
  return blocks == 1 ? 0 : (size_t)blocks * sizeof(double2);
}

int vx_photo_loss(const float* rgb, const float* rgb0, const float* target, int64_t n, const float* alphainv_last,
                  float w_main, float w_rgb0, float w_entropy, float* loss, void* scratch, size_t scratch_bytes,
                  void* stream) {
  if (n < 1 || !rgb || !target || !loss) return VX_ERR_ARG;
  const size_t need = vx_photo_loss_scratch_bytes(n);
  if (scratch_bytes < need || (need && (!scratch || (reinterpret_cast<uintptr_t>(scratch) & 15)))) return VX_ERR_ARG;
  const PhotoLoss P{rgb, rgb0, target, n, alphainv_last, w_main, w_rgb0, w_entropy};
  const int64_t blocks = (n + PL_PER_BLOCK - 1) / PL_PER_BLOCK;
  if (blocks > INT32_MAX) return VX_ERR_ARG;
  cudaStream_t st = as_stream(stream);
  photo_loss_kernel<<<(unsigned)blocks, PL_THREADS, 0, st>>>(P, reinterpret_cast<double2*>(scratch), loss);
  int s = launch_status();
  if (s || blocks == 1) return s;
  photo_loss_finish_kernel<<<1, PL_THREADS, 0, st>>>(P, reinterpret_cast<const double2*>(scratch), (int)blocks, loss);
  return launch_status();
}

int vx_photo_loss_backward(const float* rgb, const float* rgb0, const float* target, int64_t n,
                           const float* alphainv_last, float w_main, float w_rgb0, float w_entropy, const float* g,
                           float* d_rgb, float* d_rgb0, float* d_alphainv, int64_t n_alphainv, void* stream) {
  if (n < 1 || !rgb || !target || !g || !d_rgb || (rgb0 && !d_rgb0)) return VX_ERR_ARG;
  if (alphainv_last && (!d_alphainv || n_alphainv < 1)) return VX_ERR_ARG;
  const PhotoLoss P{rgb, rgb0, target, n, alphainv_last, w_main, w_rgb0, w_entropy};
  const unsigned blocks = (unsigned)std::min<int64_t>((std::max(n, n_alphainv) + 255) / 256, (int64_t)sm_count() * 8);
  photo_loss_bwd_kernel<<<blocks, 256, 0, as_stream(stream)>>>(P, g, d_rgb, d_rgb0, d_alphainv, n_alphainv);
  return launch_status();
}

}  // extern "C"
