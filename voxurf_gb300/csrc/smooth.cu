// Gaussian smoothing of the SDF grid and its adjoint.
//
// Replaces nn.Conv3d(1,1,k,padding=k//2,padding_mode='replicate') with the
// normalised Gaussian of Voxurf._gaussian_3dconv (lib/voxurf_fine.py:246-258,
// applied every step at voxurf_fine.py:638; voxurf_coarse.py:180-198, 531).
// exp(-(x^2+y^2+z^2)/(2 s^2)) / sum factorises exactly into three normalised
// 1-D kernels, so the k^3-tap convolution becomes three k-tap passes with
// clamped (replicate) indices.  The backward is the exact adjoint of each
// clamped pass.
//
// One kernel does all three passes in one sweep of the grid
// (smooth_rows_kernel below for large grids of whole float4 rows,
// smooth_march_kernel for the others).  In the latter a CTA owns a
// 32 (y) x 32 (z) column tile and a chunk of x; it streams the chunk's
// x-planes (plus an H-plane halo on each side) through a 4-deep ring of
// shared-memory stages filled by 4-byte cp.async copies (clamped source
// coordinates for the forward, zero fill outside the grid for the adjoint;
// each thread's copy offsets are computed once).  The z pass runs on
// four-output register windows of the staged rows, the y pass on a
// four-output window of the z-passed column of each lane (a warp owns four
// y rows), and the last 2H+1 y-passed values of each of a thread's four
// output columns stay in registers for the x pass; output planes leave as
// 128-byte coalesced rows.  Shared rows have odd padded strides (no bank
// conflicts).  Each input voxel is read from DRAM about once; the x halos
// are mostly L2 hits because the chunks of one tile are neighbouring CTAs.
#include <algorithm>

#include "common.cuh"

namespace vx {

struct Taps {
  float w[9];
  int h;  // half width, ksize = 2h+1 (<= 9)
};

constexpr int SM_T = 32;        // column tile: 32 (y) x 32 (z)
constexpr int SM_THREADS = 256, SM_STAGES = 4;
constexpr int SM_ROWS = SM_T / (SM_THREADS / 32);  // y rows per warp
static_assert(SM_ROWS == 4, "four y rows per warp: one window of pass4");

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// 4-byte asynchronous global->shared copy to a shared-window address;
// src_bytes 0 writes a zero.
__device__ __forceinline__ void cp_async4_s(uint32_t dst, const void* src, uint32_t src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit_group() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Adjoint of one clamped 1-D convolution at output position j (0 or n-1) of
// an axis of length n, reading the gradient at position j+d through rel(d)
// for d in [-H, H] (zero outside [0, n)).  Only the two boundary positions
// take this path: they also collect the taps that the forward clamped onto
// them.  The offsets are compile-time after unrolling, so rel may index a
// register array.
template <int H, typename Rel>
__device__ __forceinline__ float adjoint_boundary(const float (&w)[2 * H + 1], int j, int n, Rel rel) {
  float acc = 0.f;
  if (n == 1) {
    float s = 0.f;
#pragma unroll
    for (int tt = -H; tt <= H; ++tt) s += w[tt + H];
    return s * rel(0);
  }
  if (j == 0) {
#pragma unroll
    for (int i = 0; i <= H; ++i) {  // gradient positions i = 0 .. H
      if (i < n) {
        float s = 0.f;
#pragma unroll
        for (int tt = -H; tt <= -i; ++tt) s += w[tt + H];
        acc += s * rel(i);
      }
    }
  } else {  // j == n - 1
#pragma unroll
    for (int d = -H; d <= 0; ++d) {  // gradient positions n-1+d, ascending
      if (n - 1 + d >= 0) {
        float s = 0.f;
#pragma unroll
        for (int tt = -d; tt <= H; ++tt) s += w[tt + H];
        acc += s * rel(d);
      }
    }
  }
  return acc;
}

// Four consecutive outputs j0 .. j0+3 of one 1-D pass along an axis of
// length n, from a register window win[k] = value at position j0 - H + k
// (clamped copies for the forward, zero outside [0, n) for the adjoint).
// The adjoint is the transposed convolution (flipped taps) except at the
// two boundary positions.  Window offsets are compile-time after unrolling.
template <bool ADJOINT, int H>
__device__ __forceinline__ void pass4(const float (&w)[2 * H + 1], const float (&win)[4 + 2 * H], int j0, int n,
                                      float (&out)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int j = j0 + i;
    float acc = 0.f;
    if (ADJOINT) {
      if (j == 0 || j == n - 1) {
        acc = adjoint_boundary<H>(w, j, n, [&](int d) { return win[i + H + d]; });
      } else {
#pragma unroll
        for (int tt = H; tt >= -H; --tt) acc += w[H - tt] * win[i + H + tt];
      }
    } else {
#pragma unroll
      for (int tt = -H; tt <= H; ++tt) acc += w[tt + H] * win[i + H + tt];
    }
    out[i] = acc;
  }
}

template <int H>
struct SmGeom {
  static constexpr int PY = SM_T + 2 * H;          // staged rows (y) incl. halo
  static constexpr int PZ = SM_T + 2 * H;          // staged columns (z) incl. halo
  static constexpr int SPZ = PZ + 1;               // padded row stride: odd, bank-conflict free
  static constexpr int SZQ = SM_T + 1;             // padded row stride of the z-passed rows
  static constexpr int NE = (PY * PZ + SM_THREADS - 1) / SM_THREADS;  // copies per thread and plane
};

template <bool ADJOINT, bool ACCUM, int H>
__global__ void __launch_bounds__(SM_THREADS, 3) smooth_march_kernel(const float* __restrict__ in,
                                                                     float* __restrict__ out, int X, int Y, int Z,
                                                                     int CX, int n_xc, int n_zt, Taps t) {
  using G = SmGeom<H>;
  constexpr int R = 2 * H + 1, PY = G::PY, PZ = G::PZ, SPZ = G::SPZ, SZQ = G::SZQ, NE = G::NE;
  constexpr int W = 4 + 2 * H;  // window of four outputs
  __shared__ __align__(16) float s_in[SM_STAGES][PY][SPZ];
  __shared__ float s_zq[PY][SZQ];
  float w[R];
#pragma unroll
  for (int i = 0; i < R; ++i) w[i] = t.w[i];
  const int xc = blockIdx.x % n_xc, tile = blockIdx.x / n_xc;
  const int y0 = (tile / n_zt) * SM_T, z0 = (tile % n_zt) * SM_T;
  const int x0 = xc * CX, x1 = min(X, x0 + CX);
  const int NP = x1 - x0 + 2 * H;  // input planes x0-H .. x1-1+H
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gz = z0 + lane;
  const int64_t plane = (int64_t)Y * Z;

  // Copy plan of this thread (the same for every plane): halo-tile element
  // e = tid + 256 i -> shared offset soff (-1: none) and in-plane source
  // offset goff (clamped for the forward; -1 outside the grid for the adjoint).
  int soff[NE], goff[NE];
#pragma unroll
  for (int i = 0; i < NE; ++i) {
    const int e = tid + SM_THREADS * i;
    const int b = e / PZ, c = e - b * PZ;
    int gy = y0 + b - H, gzz = z0 + c - H;
    soff[i] = e < PY * PZ ? (b * SPZ + c) * 4 : -1;
    if (!ADJOINT) {
      gy = min(max(gy, 0), Y - 1);
      gzz = min(max(gzz, 0), Z - 1);
      goff[i] = gy * Z + gzz;
    } else {
      goff[i] = (gy >= 0 && gy < Y && gzz >= 0 && gzz < Z) ? gy * Z + gzz : -1;
    }
  }
  const uint32_t sbase = smem_addr(&s_in[0][0][0]);
  auto issue = [&](int q) {  // input plane x0 - H + q -> stage q % SM_STAGES
    const int gx = x0 - H + q;
    const uint32_t st = sbase + (uint32_t)((q % SM_STAGES) * PY * SPZ * 4);
    if (!ADJOINT) {
      const float* base = in + (int64_t)min(max(gx, 0), X - 1) * plane;
#pragma unroll
      for (int i = 0; i < NE; ++i)
        if (soff[i] >= 0) cp_async4_s(st + (uint32_t)soff[i], base + goff[i], 4u);
    } else {
      const bool xin = gx >= 0 && gx < X;
      const float* base = in + (int64_t)(xin ? gx : 0) * plane;
#pragma unroll
      for (int i = 0; i < NE; ++i) {
        if (soff[i] < 0) continue;
        const bool ok = xin && goff[i] >= 0;
        cp_async4_s(st + (uint32_t)soff[i], ok ? base + goff[i] : in, ok ? 4u : 0u);
      }
    }
  };

#pragma unroll
  for (int s = 0; s < SM_STAGES - 1; ++s) {
    if (s < NP) issue(s);
    cp_async_commit_group();
  }
  float ring[SM_ROWS][R];
#pragma unroll
  for (int r = 0; r < SM_ROWS; ++r)
#pragma unroll
    for (int k = 0; k < R; ++k) ring[r][k] = 0.f;

  for (int p = 0; p < NP; ++p) {
    cp_async_wait_group<SM_STAGES - 2>();  // plane p has landed
    __syncthreads();
    {
      const int q = p + SM_STAGES - 1;  // refill the stage plane p-1 used
      if (q < NP) issue(q);
      cp_async_commit_group();
    }
    const float(*sp)[SPZ] = s_in[p % SM_STAGES];
    // z pass: task = four consecutive z outputs of one staged row
    for (int task = tid; task < PY * (SM_T / 4); task += SM_THREADS) {
      const int oct = task / PY, b = task - oct * PY;
      float win[W], o4[4];
#pragma unroll
      for (int k = 0; k < W; ++k) win[k] = sp[b][4 * oct + k];
      pass4<ADJOINT, H>(w, win, z0 + 4 * oct, Z, o4);
#pragma unroll
      for (int i = 0; i < 4; ++i) s_zq[b][4 * oct + i] = o4[i];
    }
    __syncthreads();
    // y pass: this warp's four rows of this lane's column, into the x ring
    {
      float win[W], o4[4];
#pragma unroll
      for (int k = 0; k < W; ++k) win[k] = s_zq[SM_ROWS * warp + k][lane];
      pass4<ADJOINT, H>(w, win, y0 + SM_ROWS * warp, Y, o4);
#pragma unroll
      for (int r = 0; r < SM_ROWS; ++r) {
#pragma unroll
        for (int k = 0; k < R - 1; ++k) ring[r][k] = ring[r][k + 1];
        ring[r][R - 1] = o4[r];
      }
    }
    // x pass: ring[r][k] holds input plane gxo - H + k of output plane gxo
    const int gxo = x0 + p - 2 * H;
    if (gxo < x0 || gz >= Z) continue;
#pragma unroll
    for (int r = 0; r < SM_ROWS; ++r) {
      const int gy = y0 + SM_ROWS * warp + r;
      if (gy >= Y) continue;
      float acc = 0.f;
      if (ADJOINT) {
        if (gxo == 0 || gxo == X - 1) {
          acc = adjoint_boundary<H>(w, gxo, X, [&](int d) { return ring[r][d + H]; });
        } else {
#pragma unroll
          for (int tt = H; tt >= -H; --tt) acc += w[H - tt] * ring[r][tt + H];
        }
      } else {
#pragma unroll
        for (int tt = -H; tt <= H; ++tt) acc += w[tt + H] * ring[r][tt + H];
      }
      const int64_t o = (int64_t)gxo * plane + (int64_t)gy * Z + gz;
      if (ACCUM)
        out[o] += acc;
      else
        out[o] = acc;
    }
  }
  cp_async_wait_group<0>();
}

// The same sweep without passes through shared memory, for rows of whole
// float4s (Z % 4 == 0, 16-byte aligned buffers) and up to five taps: a warp owns
// 4 (y) x 128 (z) outputs of a chunk of x and a lane four consecutive z.  It
// reads the 4 + 2H rows of a plane as float4s (cp.async into the lane's own
// 16 bytes of shared memory, no barrier: 49 KB a block for five taps), takes the z neighbours of a lane's four values by
// shuffle (the two lanes at the tile's ends by a load of their own), runs the y
// pass over the rows in registers and keeps the last 2H + 1 y-passed planes for
// the x pass; the plane loop is unrolled 2H + 1 times, so the ring needs no
// moves, and the y and x passes work on pairs of z (fma2).  Every output sums
// the same products in the same order as the kernel above: the bits are equal.
// Bound: L2 reads (each row is read by two warps) and their latency; 74 thread
// instructions an output became about 20.  The planes arrive by cp.async, three
// deep.  Five taps, inputs from HBM: 256^3 forward 55 -> 35 us, adjoint 77 -> 50 us
// (20 us of HBM); 384^3 149 -> 100 and 221 -> 137 us.
constexpr int SR_WARPS = 4;      // consecutive y tiles share rows through L1
constexpr int SR_Z = 128;
constexpr int SR_STAGES = 3;     // planes on their way or in use

// Bytes of one plane of a warp: each lane's float4 of every row, and the pairs
// of values beside the tile.
template <int H>
struct SrGeom {
  static constexpr int ROWS = 4 + 2 * H, EDGE = ROWS * 512, STAGE = EDGE + ROWS * 16;
  static constexpr int SMEM = SR_WARPS * SR_STAGES * STAGE;
};

// 16- or 8-byte asynchronous copy through L1, zero where src_bytes is 0.
template <int N>
__device__ __forceinline__ void cp_async_s(uint32_t dst, const void* src, uint32_t src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(N), "r"(src_bytes) : "memory");
}

// The adjoint's weights at the two ends of an axis of more than 2H positions
// (adjoint_boundary with its sums of taps formed once).
template <int H>
struct EndTaps {
  float lo[H + 1], hi[H + 1];   // position i from the first, H - i from the last
  __device__ __forceinline__ explicit EndTaps(const float (&w)[2 * H + 1]) {
#pragma unroll
    for (int i = 0; i <= H; ++i) {
      lo[i] = 0.f;
#pragma unroll
      for (int k = 0; k <= H - i; ++k) lo[i] += w[k];
      hi[i] = 0.f;
#pragma unroll
      for (int k = 2 * H - i; k <= 2 * H; ++k) hi[i] += w[k];
    }
  }
  // the first position from the values at it and above, the last from those
  // up to it: v(i), i = 0 .. H, ascending
  template <typename V>
  __device__ __forceinline__ float first(V v) const {
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i <= H; ++i) acc += lo[i] * v(i);
    return acc;
  }
  template <typename V>
  __device__ __forceinline__ float last(V v) const {
    float acc = 0.f;
#pragma unroll
    for (int i = 0; i <= H; ++i) acc += hi[i] * v(i);
    return acc;
  }
};

// Four consecutive z outputs of a row from the lane's values and its
// neighbours: win[k] = value at z - H + k (clamped copies for the forward, zero
// outside the grid for the adjoint).
template <bool ADJOINT, int H>
__device__ __forceinline__ void rows_z_pass(const float (&w)[2 * H + 1], const EndTaps<H>& ends,
                                            const float (&win)[4 + 2 * H], int z, int Z, f32x2 (&o)[2]) {
  o[0] = o[1] = 0;
#pragma unroll
  for (int s = 0; s < 2 * H + 1; ++s) {
    const int k = ADJOINT ? 2 * H - s : s;            // tap position in the window
    const f32x2 ww = pack2(w[s], w[s]);
    o[0] = fma2(ww, pack2(win[k], win[k + 1]), o[0]);
    o[1] = fma2(ww, pack2(win[k + 2], win[k + 3]), o[1]);
  }
  if (ADJOINT) {
    float2 v = unpack2(o[0]);
    const float a = ends.first([&](int i) { return win[H + i]; });
    o[0] = pack2(z == 0 ? a : v.x, v.y);
    v = unpack2(o[1]);
    const float b = ends.last([&](int i) { return win[3 + i]; });
    o[1] = pack2(v.x, z + 4 == Z ? b : v.y);
  }
}

template <bool ADJOINT, bool ACCUM, int H>
__global__ void __launch_bounds__(32 * SR_WARPS, 3) smooth_rows_kernel(const float* __restrict__ in,
                                                                      float* __restrict__ out, int X, int Y, int Z,
                                                                      int CX, Taps t) {
  constexpr int R = 2 * H + 1, ROWS = 4 + 2 * H;
  float w[R];
#pragma unroll
  for (int i = 0; i < R; ++i) w[i] = t.w[i];
  const EndTaps<H> ends(w);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int y0 = 4 * (blockIdx.x * SR_WARPS + warp), z0 = blockIdx.y * SR_Z, z = z0 + 4 * lane;
  const int x0 = blockIdx.z * CX, x1 = min(X, x0 + CX);
  if (y0 >= Y) return;
  const bool live = z < Z;
  const int64_t plane = (int64_t)Y * Z;
  // the values beside the tile, for its first and last lane
  const bool left = H > 0 && lane == 0 && z0 > 0, right = H > 0 && lane == 31 && z0 + SR_Z < Z;
  const int ze = left ? z0 - 2 : z0 + SR_Z;

  f32x2 ring[R][4][2];   // y-passed planes of this lane's 4 rows x 4 z
#pragma unroll
  for (int k = 0; k < R; ++k)
#pragma unroll
    for (int r = 0; r < 4; ++r) ring[k][r][0] = ring[k][r][1] = 0;

  // A lane copies and reads its own values only: the ring needs no barrier.
  extern __shared__ __align__(16) uint8_t sr_smem[];
  using G = SrGeom<H>;
  uint8_t* mine = sr_smem + warp * (SR_STAGES * G::STAGE);
  const uint32_t mine_s = smem_addr(mine);
  const int edge_at = G::EDGE + (lane == 0 ? 0 : 8);
  auto issue = [&](int p) {   // input plane x0 - H + p
    const int gx = x0 - H + p;
    const bool xin = gx >= 0 && gx < X;
    const float* src = in + (int64_t)min(max(gx, 0), X - 1) * plane;
    const uint32_t dst = mine_s + (uint32_t)(p % SR_STAGES * G::STAGE);
#pragma unroll
    for (int b = 0; b < ROWS; ++b) {
      const int gy = y0 + b - H;
      const bool in_row = !ADJOINT || (xin && gy >= 0 && gy < Y);
      const float* row = src + (int64_t)min(max(gy, 0), Y - 1) * Z;
      const bool ok = live && in_row;
      cp_async_s<16>(dst + (uint32_t)(b * 512 + lane * 16), ok ? row + z : in, ok ? 16u : 0u);
      if (left || right) cp_async_s<8>(dst + (uint32_t)(edge_at + b * 16), row + ze, in_row ? 8u : 0u);
    }
  };
  auto load_plane = [&](int p, f32x2 (&q)[ROWS][2]) {   // z-passed rows y0 - H .. of plane p
    const uint8_t* src = mine + p % SR_STAGES * G::STAGE;
    float4 v[ROWS];
    float2 e[ROWS];
#pragma unroll
    for (int b = 0; b < ROWS; ++b) {
      v[b] = *reinterpret_cast<const float4*>(src + b * 512 + lane * 16);
      e[b] = left || right ? *reinterpret_cast<const float2*>(src + edge_at + b * 16) : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int b = 0; b < ROWS; ++b) {
      float win[ROWS];
      win[H] = v[b].x;
      win[H + 1] = v[b].y;
      win[H + 2] = v[b].z;
      win[H + 3] = v[b].w;
      if constexpr (H > 0) {
        float l1 = __shfl_up_sync(0xffffffffu, v[b].w, 1), r0 = __shfl_down_sync(0xffffffffu, v[b].x, 1);
        if (lane == 0) l1 = e[b].y;
        if (lane == 31) r0 = e[b].x;
        if (z == 0) l1 = ADJOINT ? 0.f : v[b].x;
        if (z + 4 == Z) r0 = ADJOINT ? 0.f : v[b].w;
        win[H - 1] = l1;
        win[H + 4] = r0;
      }
      if constexpr (H > 1) {
        float l0 = __shfl_up_sync(0xffffffffu, v[b].z, 1), r1 = __shfl_down_sync(0xffffffffu, v[b].y, 1);
        if (lane == 0) l0 = e[b].x;
        if (lane == 31) r1 = e[b].y;
        if (z == 0) l0 = ADJOINT ? 0.f : v[b].x;
        if (z + 4 == Z) r1 = ADJOINT ? 0.f : v[b].w;
        win[H - 2] = l0;
        win[H + 5] = r1;
      }
      rows_z_pass<ADJOINT, H>(w, ends, win, z, Z, q[b]);
    }
  };

  const int NP = x1 - x0 + 2 * H;   // input planes x0 - H .. x1 - 1 + H
#pragma unroll
  for (int p = 0; p < SR_STAGES; ++p) {
    if (p < NP) issue(p);
    cp_async_commit_group();
  }
  for (int p0 = 0; p0 < NP; p0 += R) {
#pragma unroll
    for (int u = 0; u < R; ++u) {
      const int p = p0 + u;
      if (p >= NP) break;
      cp_async_wait_group<SR_STAGES - 1>();
      f32x2 q[ROWS][2];
      load_plane(p, q);
      if (p + SR_STAGES < NP) issue(p + SR_STAGES);   // the values above are in registers
      cp_async_commit_group();
      // y pass into the ring's slot of this plane
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int gy = y0 + r;
        if (ADJOINT && (gy == 0 || gy == Y - 1)) {
          float2 c[ROWS][2];
#pragma unroll
          for (int b = 0; b < ROWS; ++b)
#pragma unroll
            for (int h = 0; h < 2; ++h) c[b][h] = unpack2(q[b][h]);
#pragma unroll
          for (int h = 0; h < 2; ++h)
            ring[u][r][h] = gy == 0 ? pack2(ends.first([&](int i) { return c[r + H + i][h].x; }),
                                            ends.first([&](int i) { return c[r + H + i][h].y; }))
                                    : pack2(ends.last([&](int i) { return c[r + i][h].x; }),
                                            ends.last([&](int i) { return c[r + i][h].y; }));
        } else {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            f32x2 acc = 0;
#pragma unroll
            for (int s = 0; s < R; ++s) acc = fma2(pack2(w[s], w[s]), q[r + (ADJOINT ? 2 * H - s : s)][h], acc);
            ring[u][r][h] = acc;
          }
        }
      }
      // x pass: output plane gxo from the planes gxo - H + k, slot (u + 1 + k) % R
      const int gxo = x0 + p - 2 * H;
      if (gxo < x0 || !live) continue;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int gy = y0 + r;
        if (gy >= Y) break;
        float2 o[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (ADJOINT && (gxo == 0 || gxo == X - 1)) {
            float2 c[R];
#pragma unroll
            for (int k = 0; k < R; ++k) c[k] = unpack2(ring[(u + 1 + k) % R][r][h]);
            o[h].x = gxo == 0 ? ends.first([&](int i) { return c[H + i].x; }) : ends.last([&](int i) { return c[i].x; });
            o[h].y = gxo == 0 ? ends.first([&](int i) { return c[H + i].y; }) : ends.last([&](int i) { return c[i].y; });
          } else {
            f32x2 acc = 0;
#pragma unroll
            for (int s = 0; s < R; ++s)
              acc = fma2(pack2(w[s], w[s]), ring[(u + 1 + (ADJOINT ? 2 * H - s : s)) % R][r][h], acc);
            o[h] = unpack2(acc);
          }
        }
        float4* dst = reinterpret_cast<float4*>(out + (int64_t)gxo * plane + (int64_t)gy * Z + z);
        float4 v = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
        if (ACCUM) {
          const float4 old = *dst;
          v = make_float4(old.x + v.x, old.y + v.y, old.z + v.z, old.w + v.w);
        }
        *dst = v;
      }
    }
  }
}

// x chunking: the number of chunks (of >= 8 planes; each reads 2H more than it
// writes) whose waves of three CTAs a multiprocessor pass the fewest planes.
// (Twelve warps a multiprocessor rounded up to whole chunks left a second wave
// with a few CTAs: 512 x 512 x 132 adjoint 192 us, 146 now.)
template <bool ADJOINT, bool ACCUM, int H>
static int launch_rows(const float* in, float* out, int X, int Y, int Z, const Taps& t, cudaStream_t st) {
  const int n_yt = (Y + 4 * SR_WARPS - 1) / (4 * SR_WARPS), n_zt = (Z + SR_Z - 1) / SR_Z;
  const int64_t slots = (int64_t)sm_count() * 3, tiles = (int64_t)n_yt * n_zt;
  int CX = X;
  int64_t best = INT64_MAX;
  for (int n = 1; n <= (X + 7) / 8; ++n) {
    const int cx = (X + n - 1) / n, n_xc = (X + cx - 1) / cx;
    const int64_t cost = (tiles * n_xc + slots - 1) / slots * (cx + 2 * H);
    if (cost < best) best = cost, CX = cx;
  }
  const dim3 grid((unsigned)n_yt, (unsigned)n_zt, (unsigned)((X + CX - 1) / CX));
  auto kernel = smooth_rows_kernel<ADJOINT, ACCUM, H>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SrGeom<H>::SMEM);
  if (e != cudaSuccess) return cuda_status(e);
  kernel<<<grid, 32 * SR_WARPS, SrGeom<H>::SMEM, st>>>(in, out, X, Y, Z, CX, t);
  return launch_status();
}

// x chunking: about two waves of 3 resident CTAs per SM, chunks of >= 8 planes.
template <bool ADJOINT, bool ACCUM, int H>
static int launch_march(const float* in, float* out, int X, int Y, int Z, const Taps& t, cudaStream_t st) {
  const int n_zt = (Z + SM_T - 1) / SM_T, n_yt = (Y + SM_T - 1) / SM_T;
  const int64_t tiles = (int64_t)n_zt * n_yt;
  const int64_t want = (int64_t)sm_count() * 3 * 2;
  int64_t nx = (want + tiles - 1) / tiles;
  const int64_t nx_max = (X + 7) / 8;
  nx = nx < 1 ? 1 : (nx > nx_max ? nx_max : nx);
  int n_xc = (int)nx;
  const int CX = (X + n_xc - 1) / n_xc;
  n_xc = (X + CX - 1) / CX;
  const unsigned blocks = (unsigned)(tiles * n_xc);
  smooth_march_kernel<ADJOINT, ACCUM, H><<<blocks, SM_THREADS, 0, st>>>(in, out, X, Y, Z, CX, n_xc, n_zt, t);
  return launch_status();
}

// Where the row kernel is the faster one.  Below 128^3 it has too few warps to
// hide its loads (96^3 forward 15 against 13 us).  Its tile is 128 z wide and the
// other's 32: a single tile pays from 33 z on forward (512 x 512 x 32: 50 against
// 32 us, x 36: 50 against 92) and from 65 on in the adjoint (x 64: 82 against 78,
// x 80: 82 against 97), and an adjoint whose last tile holds no more than 32
// pays from about three million voxels on (100 x 200 x 140: 22.5 against 21 us,
// 148^3: 23 against 31, 512 x 512 x 132: 146 against 176).
template <bool ADJOINT>
static bool takes_rows(int X, int Y, int Z) {
  const int64_t voxels = (int64_t)X * Y * Z;
  const int tail = Z % SR_Z;
  if (Z % 4 || std::min(X, std::min(Y, Z)) <= 4 || (Z + SR_Z - 1) / SR_Z > 65535 || (X + 7) / 8 > 65535) return false;
  if (ADJOINT) return Z > 64 && voxels >= (tail > 0 && tail <= 32 ? 3 << 20 : 1 << 21);
  return Z > 32 && voxels >= 1 << 21;
}

template <bool ADJOINT, bool ACCUM>
static int launch_h(const float* in, float* out, int X, int Y, int Z, const Taps& t, cudaStream_t st) {
  const bool rows = takes_rows<ADJOINT>(X, Y, Z) &&
                    ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  if (rows && t.h <= 2) {
    if (t.h == 0) return launch_rows<ADJOINT, ACCUM, 0>(in, out, X, Y, Z, t, st);
    if (t.h == 1) return launch_rows<ADJOINT, ACCUM, 1>(in, out, X, Y, Z, t, st);
    return launch_rows<ADJOINT, ACCUM, 2>(in, out, X, Y, Z, t, st);
  }
  switch (t.h) {
    case 0: return launch_march<ADJOINT, ACCUM, 0>(in, out, X, Y, Z, t, st);
    case 1: return launch_march<ADJOINT, ACCUM, 1>(in, out, X, Y, Z, t, st);
    case 2: return launch_march<ADJOINT, ACCUM, 2>(in, out, X, Y, Z, t, st);
    case 3: return launch_march<ADJOINT, ACCUM, 3>(in, out, X, Y, Z, t, st);
    default: return launch_march<ADJOINT, ACCUM, 4>(in, out, X, Y, Z, t, st);
  }
}

static int make_taps(const float* taps_host, int ksize, Taps& t) {
  if (ksize < 1 || ksize > 9 || (ksize % 2) == 0) return VX_ERR_ARG;
  t.h = ksize / 2;
  for (int i = 0; i < 9; ++i) t.w[i] = i < ksize ? taps_host[i] : 0.f;
  return VX_OK;
}

}  // namespace vx

using namespace vx;

extern "C" {

int vx_smooth3d(const float* in, float* out, float* tmp1, float* tmp2, int64_t X, int64_t Y, int64_t Z,
                const float* taps_host, int ksize, void* stream) {
  (void)tmp1;
  (void)tmp2;
  if (X <= 0 || Y <= 0 || Z <= 0 || !in || !out || !taps_host) return VX_ERR_ARG;
  if (X * Y * Z > INT32_MAX) return VX_ERR_ARG;
  Taps t;
  const int s = make_taps(taps_host, ksize, t);
  if (s) return s;
  return launch_h<false, false>(in, out, (int)X, (int)Y, (int)Z, t, as_stream(stream));
}

int vx_smooth3d_adjoint(const float* grad_out, float* grad_in, float* tmp1, float* tmp2, int64_t X, int64_t Y,
                        int64_t Z, const float* taps_host, int ksize, int accumulate, void* stream) {
  (void)tmp1;
  (void)tmp2;
  if (X <= 0 || Y <= 0 || Z <= 0 || !grad_out || !grad_in || !taps_host) return VX_ERR_ARG;
  if (X * Y * Z > INT32_MAX) return VX_ERR_ARG;
  Taps t;
  const int s = make_taps(taps_host, ksize, t);
  if (s) return s;
  cudaStream_t st = as_stream(stream);
  return accumulate ? launch_h<true, true>(grad_out, grad_in, (int)X, (int)Y, (int)Z, t, st)
                    : launch_h<true, false>(grad_out, grad_in, (int)X, (int)Y, (int)Z, t, st);
}

}  // extern "C"
