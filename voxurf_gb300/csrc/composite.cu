// Per-ray transmittance / weight scan (alpha2weight) and its backward.
//
// Drop-in for render_utils_cuda.alpha2weight / alpha2weight_backward
// (render_utils.cpp:182-183; kernels render_utils_kernel.cu:577-707).  The
// reference walks each ray with one thread (8192 rays -> 32 CTAs on 152 SMs)
// and a serial loop.  Here one warp owns one ray and walks it 128 samples at
// a time: four 32-sample prefix products that do not depend on one another,
// then the running transmittance through the four.  It is carried as a
// FloatPair on segments of more than 512 samples (so the prefix stays
// accurate on rays of thousands of samples) and in FP32 on shorter ones, as
// the reference's float loop.  Semantics kept exactly:
//   T[i] = prod_{j<i} (1 - alpha[j]),  w[i] = T[i] * alpha[i],
//   stop after the first sample whose inclusive product drops below 1e-3,
//   samples after the stop keep w = 0, T = 1, grad = 0,
//   empty rays report i_start = i_end = 0 and alphainv_last = 1.
// Segment bounds come from a search in the sorted ray_id instead of the
// reference's scatter kernel + device-indexed host write (:607-635).
//
// Bound: the latency of a ray's chain (search, loads, scans).  At 8192 rays x
// 400 samples every input read and every output written once (alpha, ray_id,
// grad_weights in; weight, T, grad out: 28 bytes a sample) would take 14 us;
// the two kernels move 36 (12 forward, where ray_id is only probed, and 24
// backward, which reads weight and T again and clears grad first): 17 us.
// Forward and backward there, with the host's two calls: 178 us with 32
// samples a step, a bisection per bound and FP64 beyond 512 samples (62 + 105
// us of kernels), 74 us now, where the calls themselves take as long as the
// kernels.
#include <type_traits>

#include "common.cuh"

namespace vx {

// Segment [beg, end) of ray r in a sorted ray_id array.  Each half of the
// warp searches one bound, sixteen probes a step: six dependent loads for
// millions of samples, where a bisection takes 22.  The probes are 1/16 of the
// range and one sample apart: a shift, where sixteen even parts of it took
// 64-bit divisions that cost a million short rays more than they saved.
__device__ __forceinline__ void ray_segment(const int64_t* __restrict__ ray_id, int64_t n_pts, int64_t r,
                                            int64_t* beg, int64_t* end) {
  const int lane = lane_id(), half = lane >> 4, sub = lane & 15;
  const int64_t key = r + half;
  int64_t lo = 0, hi = n_pts;
  while (__any_sync(0xffffffffu, lo < hi)) {
    const int64_t step = ((hi - lo) >> 4) + 1;             // 16 steps reach past hi
    const int64_t at = lo + step * (sub + 1) - 1;
    const bool less = at < hi && ray_id[at] < key;
    const int c = __popc((__ballot_sync(0xffffffffu, less) >> (16 * half)) & 0xffffu);
    lo = min(lo + step * c, hi);                           // (beyond hi only where ray_id is not sorted)
    hi = min(hi, lo + step - 1);
  }
  *beg = __shfl_sync(0xffffffffu, lo, 0);
  *end = __shfl_sync(0xffffffffu, lo, 16);
}

// 32-sample scans in flight per warp: as many as the segment fills, up to
// four (one or two are a single step).  With four for every segment and the
// even search above, 1M rays of 1 to 5 samples took 803 us forward and 327 us
// backward, where one scan and a bisection took 656 and 287.
template <typename F>
__device__ __forceinline__ void by_length(int64_t len, F scan) {
  if (len <= 32) scan(0.f, std::integral_constant<int, 1>());
  else if (len <= 64) scan(0.f, std::integral_constant<int, 2>());
  else if (len <= VX_FP32_SCAN_MAX_STEPS) scan(0.f, std::integral_constant<int, 4>());
  else scan(FloatPair(), std::integral_constant<int, 4>());
}

// Warp-level forward scan of one segment.  Writes weight/T for every sample
// of [beg, end); returns i_end and alphainv_last in every lane.
template <typename Acc, int CHUNKS>
__device__ __forceinline__ void scan_segment_fwd(const float* __restrict__ alpha, int64_t beg, int64_t end,
                                                 float* __restrict__ weight, float* __restrict__ T,
                                                 int64_t* i_end_out, float* last_out) {
  using Op = AccOps<Acc>;
  const int lane = lane_id();
  Acc carry = Op::of(1.f);
  float nxt[CHUNKS];
#pragma unroll
  for (int c = 0; c < CHUNKS; ++c) nxt[c] = beg + 32 * c + lane < end ? alpha[beg + 32 * c + lane] : 0.f;
  for (int64_t base = beg; base < end; base += 32 * CHUNKS) {
    float a[CHUNKS];
    Acc incl[CHUNKS];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      a[c] = nxt[c];
      incl[c] = Op::one_minus(a[c]);
      if (CHUNKS == 4) {                                   // the next step's samples, while this one scans
        const int64_t i = base + 32 * (CHUNKS + c) + lane;
        nxt[c] = i < end ? alpha[i] : 0.f;
      }
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
      for (int c = 0; c < CHUNKS; ++c) {
        const Acc u = warp_shfl_up(incl[c], o);
        if (lane >= o) incl[c] = incl[c] * u;
      }
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int64_t first = base + 32 * c, i = first + lane;
      if (first >= end) break;
      const bool valid = i < end;
      const Acc v = incl[c] * carry;
      Acc excl = warp_shfl_up(v, 1);
      if (lane == 0) excl = carry;
      const unsigned stop_mask = __ballot_sync(0xffffffffu, valid && Op::below_stop(v));
      // the first sample that drops below 1e-3 is the last one with a weight
      const int k = stop_mask ? __ffs(stop_mask) - 1 : 31;
      if (valid) {
        const float t = lane <= k ? Op::value(excl) : 1.f;
        T[i] = t;
        weight[i] = lane <= k ? t * a[c] : 0.f;
      }
      carry = warp_shfl(v, k);
      if (stop_mask) {
        for (int64_t j = i + 32; j < end; j += 32) {
          weight[j] = 0.f;
          T[j] = 1.f;
        }
        *i_end_out = first + k + 1;
        *last_out = Op::value(carry);
        return;
      }
    }
    if (CHUNKS < 4) break;   // the one step of a short segment
  }
  *i_end_out = end;
  *last_out = Op::value(carry);
}

__global__ void alpha2weight_kernel(const float* __restrict__ alpha, const int64_t* __restrict__ ray_id,
                                    int64_t n_pts, int64_t n_rays, float* __restrict__ weight,
                                    float* __restrict__ T, float* __restrict__ alphainv_last,
                                    int64_t* __restrict__ i_start, int64_t* __restrict__ i_end) {
  const int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (r >= n_rays) return;
  int64_t beg, end;
  ray_segment(ray_id, n_pts, r, &beg, &end);
  if (beg >= end) {
    if (lane_id() == 0) {
      i_start[r] = 0;
      i_end[r] = 0;
      alphainv_last[r] = 1.f;
    }
    return;
  }
  int64_t ie;
  float last;
  by_length(end - beg, [&](auto acc, auto chunks) {
    scan_segment_fwd<decltype(acc), chunks>(alpha, beg, end, weight, T, &ie, &last);
  });
  if (lane_id() == 0) {
    i_start[r] = beg;
    i_end[r] = ie;
    alphainv_last[r] = last;
  }
}

// Reverse scan, render_utils_kernel.cu:671-675:
//   back = grad_last*alphainv_last;  for i = i_end-1 .. i_start:
//     grad[i] = gw[i]*T[i] - back/(1-alpha[i]+1e-10);  back += gw[i]*w[i]
// The running sum `back` is carried in Acc (a FloatPair on segments of more
// than 512 samples).
template <typename Acc, int CHUNKS>
__device__ __forceinline__ void scan_segment_bwd(const float* __restrict__ alpha, const float* __restrict__ weight,
                                                 const float* __restrict__ T, const float* __restrict__ grad_w,
                                                 int64_t beg, int64_t end, float back0,
                                                 float* __restrict__ grad) {
  using Op = AccOps<Acc>;
  const int lane = lane_id();
  Acc carry = Op::of(back0);
  for (int64_t top = end; top > beg; top -= 32 * CHUNKS) {
    float gw_t[CHUNKS], a[CHUNKS];
    Acc suffix[CHUNKS];
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int64_t i = top - 32 * (c + 1) + lane;
      float gw = 0.f, w = 0.f, t = 0.f;
      a[c] = 0.f;
      if (i >= beg) {
        gw = grad_w[i];
        w = weight[i];
        t = T[i];
        a[c] = alpha[i];
      }
      gw_t[c] = gw * t;
      suffix[c] = Op::of(i >= beg ? gw * w : 0.f);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
#pragma unroll
      for (int c = 0; c < CHUNKS; ++c) {
        const Acc u = warp_shfl_down(suffix[c], o);
        if (lane + o < 32) suffix[c] = suffix[c] + u;
      }
#pragma unroll
    for (int c = 0; c < CHUNKS; ++c) {
      const int64_t i = top - 32 * (c + 1) + lane;
      Acc after = warp_shfl_down(suffix[c], 1);   // the lanes above this one
      if (lane == 31) after = Op::of(0.f);
      const Acc back = carry + after;
      if (i >= beg) grad[i] = Op::grad(gw_t[c], back, a[c]);
      if (CHUNKS == 4 || c + 1 < CHUNKS) carry = carry + warp_shfl(suffix[c], 0);
    }
    if (CHUNKS < 4) break;
  }
}

__global__ void alpha2weight_backward_kernel(const float* __restrict__ alpha, const float* __restrict__ weight,
                                             const float* __restrict__ T,
                                             const float* __restrict__ alphainv_last,
                                             const int64_t* __restrict__ i_start,
                                             const int64_t* __restrict__ i_end, int64_t n_pts, int64_t n_rays,
                                             const float* __restrict__ grad_weights,
                                             const float* __restrict__ grad_last, float* __restrict__ grad,
                                             int* err) {
  const int64_t r = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (r >= n_rays) return;
  const int64_t beg = i_start[r], end = i_end[r];
  if (beg >= end) return;
  if (beg < 0 || end > n_pts) {
    if (lane_id() == 0) set_device_error(err, VX_ERR_BOUNDS);
    return;
  }
  const float back = grad_last[r] * alphainv_last[r];
  by_length(end - beg, [&](auto acc, auto chunks) {
    scan_segment_bwd<decltype(acc), chunks>(alpha, weight, T, grad_weights, beg, end, back, grad);
  });
}

}  // namespace vx

using namespace vx;

extern "C" {

int vx_alpha2weight(const float* alpha, const int64_t* ray_id, int64_t n_pts, int64_t n_rays, float* weight,
                    float* T, float* alphainv_last, int64_t* i_start, int64_t* i_end, void* stream) {
  if (n_pts < 0 || n_rays < 0) return VX_ERR_ARG;
  cudaStream_t st = as_stream(stream);
  if (n_rays == 0) return VX_OK;
  if (!alphainv_last || !i_start || !i_end) return VX_ERR_ARG;
  if (n_pts > 0 && (!alpha || !ray_id || !weight || !T)) return VX_ERR_ARG;
  const int wpb = VX_THREADS / 32;
  alpha2weight_kernel<<<(unsigned)((n_rays + wpb - 1) / wpb), VX_THREADS, 0, st>>>(
      alpha, ray_id, n_pts, n_rays, weight, T, alphainv_last, i_start, i_end);
  return launch_status();
}

int vx_alpha2weight_backward(const float* alpha, const float* weight, const float* T, const float* alphainv_last,
                             const int64_t* i_start, const int64_t* i_end, int64_t n_pts, int64_t n_rays,
                             const float* grad_weights, const float* grad_last, float* grad, void* stream) {
  if (n_pts < 0 || n_rays < 0) return VX_ERR_ARG;
  cudaStream_t st = as_stream(stream);
  if (n_pts > 0) {
    if (!grad) return VX_ERR_ARG;
    int s = cuda_status(cudaMemsetAsync(grad, 0, (size_t)n_pts * sizeof(float), st));
    if (s) return s;
  }
  if (n_rays == 0 || n_pts == 0) return VX_OK;
  if (!alpha || !weight || !T || !alphainv_last || !i_start || !i_end || !grad_weights || !grad_last)
    return VX_ERR_ARG;
  const int wpb = VX_THREADS / 32;
  alpha2weight_backward_kernel<<<(unsigned)((n_rays + wpb - 1) / wpb), VX_THREADS, 0, st>>>(
      alpha, weight, T, alphainv_last, i_start, i_end, n_pts, n_rays, grad_weights, grad_last, grad,
      device_error_ptr());
  return launch_status();
}

}  // extern "C"
