// Shared helpers for the voxurf_gb300 CUDA library (sm_103a only).
//
// Every exported entry point is `extern "C"`, takes plain device pointers,
// sizes and a cudaStream_t, never allocates device memory, and returns an
// int status (VX_OK on success).  Launch errors are caught with
// cudaGetLastError() right after each launch, unlike the pybind11 ops they
// replace, which never check (render_utils.cpp:46-48 only checks inputs).
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "voxurf_gb300.h"

#define VX_THREADS 256

namespace vx {

// Last CUDA error seen by any entry point of this library (host-side copy).
extern int g_last_cuda_error;
// Number of kernel launches issued by this library (every launch is
// followed by exactly one launch_status() call).
extern unsigned long long g_launch_count;

inline int launch_status() {
  __atomic_add_fetch(&g_launch_count, 1ull, __ATOMIC_RELAXED);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    g_last_cuda_error = (int)e;
    return VX_ERR_LAUNCH;
  }
  return VX_OK;
}

inline int cuda_status(cudaError_t e) {
  if (e != cudaSuccess) {
    g_last_cuda_error = (int)e;
    return VX_ERR_CUDA;
  }
  return VX_OK;
}

// Device-resident error word (one per device, in runtime.cu).  Kernels that
// detect an out-of-range index or an overflowing capacity record the first
// error code there (and skip the access) instead of faulting;
// vx_device_error() reads and clears it.  Host code passes its address to
// the kernels that may report (device_error_ptr()).
int* device_error_ptr();

__device__ __forceinline__ void set_device_error(int* err, int code) {
  if (err) atomicCAS(err, 0, code);
}

inline unsigned int grid_for(int64_t n, int threads = VX_THREADS) {
  int64_t b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  return (unsigned int)b;
}

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// Number of SMs of the current device (cached per process).
int sm_count();

// Device-wide exclusive scan (scan.cu).  out has n+1 entries, out[n] = total.
int64_t scan_n_tiles(int64_t n);
template <typename Tin, typename Tout>
int exclusive_scan(const Tin* in, int64_t n, Tout* out, void* scratch, size_t scratch_bytes, cudaStream_t st);

// ---------------------------------------------------------------------------
// Uncontracted IEEE float arithmetic.  The index-producing stages (ray/bbox
// clip, sample counts, sample positions, mask rounding) round every
// operation once, except the multiply-adds that the reference's compiled
// kernels fuse (written as __fmaf_rn where they occur), so that the results
// equal the reference's kernels and a CPU restatement bit for bit.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }

// Two floats in a 64-bit register pair: one instruction does both halves, each
// rounded as the scalar operation, at half the issue slots (the FP32 pipes'
// rate is the same: 76.6 against 73.4 TFLOP/s measured).
typedef unsigned long long f32x2;

__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// |v| as torch's norm reduction forms it: squares accumulated with fused
// multiply-adds in x, y, z order, then a correctly rounded square root.
__device__ __forceinline__ float norm3(float x, float y, float z) {
  return __fsqrt_rn(__fmaf_rn(z, z, __fmaf_rn(y, y, fmul(x, x))));
}

// |d| of a ray as the reference's compiled sampling kernels compute
// sqrt(dx*dx + dy*dy + dz*dz) (render_utils_kernel.cu:48-51, 67-70; nvcc's
// --fmad=true fuses dx*dx and then dz*dz into the sum).
__device__ __forceinline__ float ray_norm3(float x, float y, float z) {
  return __fsqrt_rn(__fmaf_rn(z, z, __fmaf_rn(x, x, fmul(y, y))));
}

// Transmittance precision: a ray of more samples than this carries its
// transmittance products (forward) and its suffix sums (backward) in FP64;
// shorter rays in FP32.  GB300 runs FP64 at a small fraction of its FP32
// rate, and at 512 factors an FP32 product is still within a few 1e-6 of
// the exact one.  The decision is per ray (warp-uniform).
constexpr int64_t VX_FP32_SCAN_MAX_STEPS = 512;

// Warp-wide helpers -----------------------------------------------------------
__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ---- accumulators of the transmittance scans --------------------------------
// FloatPair: the unevaluated sum hi + lo of two floats, |lo| <= ulp(hi) / 2:
// about 48 significant bits.  It carries the products and sums of long rays
// (VX_FP32_SCAN_MAX_STEPS), whose results are rounded to one float in the
// end: GB300 issues an FP64 operation at 1/64 of the FP32 rate, a pair
// product is seven FP32 operations.  Sums after Knuth (TwoSum) and Dekker
// (FastTwoSum), products through the exact error of a fused multiply-add.
// The arithmetic is __f*_rn throughout, so nvcc contracts nothing.  An
// infinite or NaN result keeps lo = 0 and propagates as the plain float would.
struct FloatPair {
  float hi, lo;
};

__device__ __forceinline__ bool is_finite(float v) { return fabsf(v) <= 3.402823466e38f; }

__device__ __forceinline__ FloatPair pair_fast(float a, float b) {  // |a| >= |b| or a == 0
  const float s = fadd(a, b);
  return {s, fsub(b, fsub(s, a))};
}
__device__ __forceinline__ FloatPair pair_sum(float a, float b) {
  const float s = fadd(a, b), t = fsub(s, a);
  if (!is_finite(s)) return {s, 0.f};
  return {s, fadd(fsub(a, fsub(s, t)), fsub(b, t))};
}
__device__ __forceinline__ FloatPair operator*(FloatPair a, FloatPair b) {
  const float p = fmul(a.hi, b.hi);
  if (!is_finite(p)) return {p, 0.f};
  const float e = __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.hi, b.hi, -p)));
  return pair_fast(p, e);
}
__device__ __forceinline__ FloatPair operator+(FloatPair a, FloatPair b) {
  const FloatPair s = pair_sum(a.hi, b.hi);
  if (!is_finite(s.hi)) return s;
  return pair_fast(s.hi, fadd(s.lo, fadd(a.lo, b.lo)));
}

template <typename Acc>
struct AccOps;
template <>
struct AccOps<float> {
  static __device__ __forceinline__ float of(float v) { return v; }
  static __device__ __forceinline__ float value(float v) { return v; }
  static __device__ __forceinline__ float one_minus(float a) { return 1.f - a; }
  static __device__ __forceinline__ bool below_stop(float v) { return v < 1e-3f; }
  // gw * T - back / (1 - alpha + 1e-10) of the transmittance backward
  static __device__ __forceinline__ float grad(float gw_t, float back, float alpha) {
    return gw_t - back / ((1.f - alpha) + 1e-10f);
  }
};
template <>
struct AccOps<FloatPair> {
  static __device__ __forceinline__ FloatPair of(float v) { return {v, 0.f}; }
  static __device__ __forceinline__ float value(FloatPair v) { return v.hi; }
  static __device__ __forceinline__ FloatPair one_minus(float a) { return pair_sum(1.f, -a); }
  static __device__ __forceinline__ bool below_stop(FloatPair v) {
    const float c = 1e-3f, cl = (float)(1e-3 - (double)1e-3f);
    return v.hi < c || (v.hi == c && v.lo < cl);
  }
  // the quotient from one float division and one correction step, the
  // difference summed exactly up to its last rounding
  static __device__ __forceinline__ float grad(float gw_t, FloatPair back, float alpha) {
    const float c = 1e-10f, cl = (float)(1e-10 - (double)1e-10f);
    FloatPair d = pair_sum(1.f - alpha, c);
    d.lo = fadd(d.lo, cl);
    const float q = fdiv(back.hi, d.hi);
    if (!is_finite(q)) return gw_t - q;
    const float r = __fmaf_rn(-q, d.lo, fadd(__fmaf_rn(-q, d.hi, back.hi), back.lo));
    const FloatPair s = pair_sum(gw_t, -q);
    return fadd(s.hi, fsub(s.lo, __fdividef(r, d.hi)));
  }
};

__device__ __forceinline__ float warp_shfl(float v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }
__device__ __forceinline__ float warp_shfl_up(float v, int o) { return __shfl_up_sync(0xffffffffu, v, o); }
__device__ __forceinline__ float warp_shfl_down(float v, int o) { return __shfl_down_sync(0xffffffffu, v, o); }
__device__ __forceinline__ FloatPair warp_shfl(FloatPair v, int lane) {
  return {warp_shfl(v.hi, lane), warp_shfl(v.lo, lane)};
}
__device__ __forceinline__ FloatPair warp_shfl_up(FloatPair v, int o) {
  return {warp_shfl_up(v.hi, o), warp_shfl_up(v.lo, o)};
}
__device__ __forceinline__ FloatPair warp_shfl_down(FloatPair v, int o) {
  return {warp_shfl_down(v.hi, o), warp_shfl_down(v.lo, o)};
}

// Inclusive warp prefix product (Hillis-Steele; 5 shuffle rounds).
template <typename T>
__device__ __forceinline__ T warp_inclusive_prod(T v) {
  const int lane = lane_id();
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v *= u;
  }
  return v;
}

// Inclusive warp suffix sum: lane i gets sum of lanes i..31.
template <typename T>
__device__ __forceinline__ T warp_inclusive_suffix_sum(T v) {
  const int lane = lane_id();
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T u = __shfl_down_sync(0xffffffffu, v, o);
    if (lane + o < 32) v += u;
  }
  return v;
}

template <typename T>
__device__ __forceinline__ T warp_inclusive_sum(T v) {
  const int lane = lane_id();
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

// One 32-sample step of a ray's transmittance scan with the T < 1e-3 stop
// (render_utils_kernel.cu:577-605): the lanes with `keep` multiply in
// (1 - alpha) in Acc.  T = this lane's exclusive product (FP32); returns the
// lanes up to and including the first whose inclusive product drops below
// 1e-3 (all kept lanes when none does).  carry advances to the next step
// unless the ray stops here, in which case last = the stopping product.
template <typename Acc>
__device__ __forceinline__ unsigned transmittance_step(bool keep, float alpha, Acc& carry, Acc& last, bool& stopped,
                                                       float& T) {
  const int lane = lane_id();
  const unsigned keep_mask = __ballot_sync(0xffffffffu, keep);
  const Acc fct = keep ? Acc(1) - (Acc)alpha : Acc(1);
  const Acc incl = warp_inclusive_prod(fct) * carry;
  Acc excl = __shfl_up_sync(0xffffffffu, incl, 1);
  if (lane == 0) excl = carry;
  const unsigned stop_mask = __ballot_sync(0xffffffffu, keep && incl < Acc(1e-3));
  unsigned live = keep_mask;
  if (stop_mask) {
    const int ks = __ffs(stop_mask) - 1;
    live &= (ks == 31) ? 0xffffffffu : ((2u << ks) - 1u);
    last = __shfl_sync(0xffffffffu, incl, ks);
    stopped = true;
  }
  T = (float)excl;
  if (!stopped) carry = __shfl_sync(0xffffffffu, incl, 31);
  return live;
}

}  // namespace vx
