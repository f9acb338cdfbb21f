// The FP32 MLP backward on the tensor cores: FP32 operands as three BF16
// parts each, FP32 accumulation whose truncation is kept small.
//
// x = hi + mid + lo with hi = bf16(x), mid = bf16(x - hi), lo = bf16(x - hi -
// mid): 3 x 8 significant bits, all 24 of an FP32 value.  The operands are
// scaled by 2^24 first (and the sums by 2^-48), so that the parts of the smallest
// value, subnormals included, are normal BF16 numbers: unscaled, lo and then mid
// of a value below about 2^-110 fall under BF16's smallest.  a b is summed as the
// six products hi hi, hi mid, mid hi, mid mid, hi lo, lo hi; the three dropped
// ones are below 2^-24 of it.  A product of BF16 values is exact, but each MMA
// (16 k) truncates its running FP32 sum once.  So
//   * the five small products go into a sum of their own, which is 2^-8 of the
//     result, and only the hi hi sums see truncation that matters;
//   * in the row GEMM a hi hi sum is 8 MMAs long at most, and the last 64 k's
//     products end the small sum; then the two are added in registers with
//     rounding to nearest;
//   * in the weight gradient a hi hi sum is 4 MMAs long, and every second one
//     is truncated the other way (negated(), below).
// Measured against 64 bits (test_f32_split_gpu.py, test_f32_split_range_gpu.py),
// relative: rows x 192 x 192 9.3e-8 where the CUDA-core sums are at 2.5e-7, a
// weight gradient over 131,003 rows 1.4e-7 against 3.7e-7.  On operands of one
// sign, where truncation does not average out: rows 1.3e-7 against 2.1e-7, but
// their column sums 1.2e-7 (one unit in the last place) against 2e-9; weight
// gradients after their ordered sum 5.0e-8 both over 60,001 rows, 5.5e-8 against
// 5.9e-8 over 131,003 (1.4e-7 with sums of 8 MMAs in one direction; 2 us less).
// The forward keeps its CUDA-core sums: a ReLU whose input lies within a
// rounding of zero would switch with them.
//
// A value that has no such parts (infinite or NaN), or one so large that a
// product with another could overflow (hi hi to +inf beside hi mid to -inf), is
// noticed while it is split; the tile or the CTA's partial that holds one is
// computed again by plain FP32 sums, as the CUDA-core kernels form them.
//
//   split_rowgemm_kernel  C = A Bt (dz_l = (dz_{l+1} W_l) * [h_l > 0] with the
//                         column sums of the bias gradient; dX = dz_1 W_0):
//                         persistent, the weight's parts in shared memory, 128
//                         rows a tile, A's parts written to tensor memory 64 k
//                         at a time while the previous 64 are multiplied;
//   split_wgrad_kernel    D = A^T B over a CTA's rows (dz^T h): both operands
//                         split into MN-major shared-memory tiles of 32 rows.
//                         A warp of its own issues the MMAs (24 of them take a
//                         thread ~2,000 cycles: a warp that also splits kept
//                         the others waiting, 105 -> 91 us), and the partials
//                         leave in whole sectors (4 us).
// 131,003 rows, 192 x 192: the row GEMM with mask and column sums 176 -> 84 us
// (its three FP32 matrices take 44 us of HBM), the weight gradient 208 -> 92
// us (30 us of HBM).  Bound now: the row GEMM's loads and stores beside its
// MMAs; in the weight gradient the MMAs and the splitting of 32 rows, each
// about 1 us, two stages deep, and about 10 us of filling and storing per CTA.
#include <algorithm>

#include "mlp_f32.cuh"
#include "tcgen05.cuh"

namespace vx {
namespace mf {

using namespace tc;
using bf16 = __nv_bfloat16;

constexpr int SP_THREADS = 512;     // 16 warps: TMEM lane quarter = warp % 4, column part = warp / 4
constexpr int TILE_M = 128;
constexpr float SCALE = 0x1p24f;      // of the operands before they are split
constexpr float UNSCALE = 0x1p-48f;   // of the sums of their products
constexpr float SPLIT_MAX = 0x1p34f;  // below it no scaled product overflows, nor the sum of 1,024 of them

// The parts of two neighbouring values times SCALE, packed (the first in the
// lower half).
struct Split2 {
  uint32_t hi, mid, lo;
};

__device__ __forceinline__ float bf16_lo(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }

__device__ __forceinline__ Split2 split2(float a, float b, bool& bad) {
  Split2 s;
  bad |= !(fabsf(a) < SPLIT_MAX) || !(fabsf(b) < SPLIT_MAX);
  a *= SCALE;
  b *= SCALE;
  s.hi = pack_bf16(a, b);
  a -= bf16_lo(s.hi);
  b -= bf16_hi(s.hi);
  s.mid = pack_bf16(a, b);
  a -= bf16_lo(s.mid);
  b -= bf16_hi(s.mid);
  s.lo = pack_bf16(a, b);
  return s;
}

// 16 lanes x 8 columns of tensor memory: lane l holds columns 2 (l % 4), + 1 of
// rows l / 4 (r0, r1) and l / 4 + 8 (r2, r3).
__device__ __forceinline__ void st_16x8(uint32_t taddr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
  asm volatile("tcgen05.st.sync.aligned.16x256b.x1.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(r0), "r"(r1),
               "r"(r2), "r"(r3)
               : "memory");
}
__device__ __forceinline__ void ld_16x8(uint32_t taddr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}

// ============================================================================
// C = A Bt
// ============================================================================
constexpr int KCH = 64;                       // k per chunk of A in tensor memory
constexpr int A_PART = KCH / 2;               // columns of one part of a chunk

template <int K, int N>
struct RowGemmGeo {
  static constexpr int CHUNKS = K / KCH;
  static constexpr int D_SMALL = 0, D_HI = N, A_COL = 2 * N;    // tensor-memory columns
  static constexpr int PART = K * N;                            // BF16 values of one part of Bt
  static constexpr int BLOCKS = (N / 8 + 3) / 4;                // 8-column blocks of D per warp, every fourth
  static constexpr int H_BLOCKS = (BLOCKS + CHUNKS - 1) / CHUNKS;   // of them per chunk for the ReLU decisions
  static constexpr size_t SMEM = (size_t)3 * PART * 2 + 5 * N * sizeof(float) + 64;
  static_assert(K % KCH == 0 && N % 16 == 0 && A_COL + 3 * A_PART <= 512 && CHUNKS >= 2, "tensor memory");
};

// Chunk c of A for the warp's 32 rows: rows l / 4 + 8 i and, of the 16 k of
// the warp's part, 4 (l % 4) ..+3: four lanes read 64 bytes of a row.
__device__ __forceinline__ void load_chunk(const RowGemmParams& P, int64_t row0, int64_t M, int c, int part, int lane,
                                           float4 (&x)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int64_t row = row0 + (lane >> 2) + 8 * i;
    const float4* src = reinterpret_cast<const float4*>(P.A + row * P.lda + KCH * c + 16 * part) + (lane & 3);
    x[i] = row < M ? __ldg(src) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// A tile by plain FP32 sums, as the CUDA-core kernel forms them.  The column
// sums are added in an order of their own too: a thread's rows, then the groups
// of threads (red: [4][N], free until the last tile).
template <int K, int N>
__device__ __noinline__ void plain_tile(const RowGemmParams& P, int64_t m0, int64_t M, float* extra, float* red) {
  constexpr int GROUPS = SP_THREADS / N < 4 ? SP_THREADS / N : 4;
  const int col = threadIdx.x % N, group = threadIdx.x / N;
  if (group < GROUPS) {
    const int64_t end = min(M, m0 + TILE_M);
    float sum = 0.f;
    for (int64_t row = m0 + group; row < end; row += GROUPS) {
      float v = 0.f;
      for (int k = 0; k < K; ++k) v = fmaf(P.A[row * P.lda + k], P.Bt[(int64_t)k * N + col], v);
      if (P.mode == 1) {
        v = P.H[row * P.ldh + col] > 0.f ? v : 0.f;
        sum += v;
      }
      if (col < P.n_store) P.C[row * P.ldc + col] = v;
    }
    red[group * N + col] = sum;
  }
  __syncthreads();
  for (int n = threadIdx.x; n < N; n += SP_THREADS)
    for (int g = 0; g < GROUPS; ++g) extra[n] += red[g * N + n];
  __syncthreads();
}

template <int K, int N>
__global__ void __launch_bounds__(SP_THREADS, 1) split_rowgemm_kernel(RowGemmParams P, int* err) {
  using G = RowGemmGeo<K, N>;
  extern __shared__ __align__(1024) uint8_t smem[];
  bf16* Bs = reinterpret_cast<bf16*>(smem);                         // [3 parts][K/8][N][8]
  float* red = reinterpret_cast<float*>(smem + (size_t)3 * G::PART * 2);   // [4][N]
  float* extra = red + 4 * N;                                       // column sums of the tiles summed plainly
  uint64_t* bar = reinterpret_cast<uint64_t*>(extra + N);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);
  int* bad_b = reinterpret_cast<int*>(tmem_slot + 1);               // Bt holds a value without parts
  int* bad_tile = bad_b + 1;                                        // [2] ... the tile of that parity does

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, part = warp >> 2;
  const int64_t M = rows_of(P.M, P.m_dev);
  const int64_t n_tiles = (M + TILE_M - 1) / TILE_M;
  if (warp == 0) alloc(tmem_slot, 512);
  if (tid == 0) {
    mbar_init(bar, 1);
    *bad_b = bad_tile[0] = bad_tile[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int n = tid; n < N; n += SP_THREADS) extra[n] = 0.f;
  __syncthreads();
  if ((int64_t)blockIdx.x < n_tiles) {
    bool bad = false;
#pragma unroll 3
    for (int i = tid; i < K / 8 * N; i += SP_THREADS) {
      const int kg = i / N, n = i - kg * N;
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __ldg(P.Bt + (int64_t)(8 * kg + j) * N + n);
      uint32_t p[3][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const Split2 s = split2(v[2 * j], v[2 * j + 1], bad);
        p[0][j] = s.hi;
        p[1][j] = s.mid;
        p[2][j] = s.lo;
      }
#pragma unroll
      for (int q = 0; q < 3; ++q)
        *reinterpret_cast<uint4*>(Bs + q * G::PART + (size_t)i * 8) = make_uint4(p[q][0], p[q][1], p[q][2], p[q][3]);
    }
    if (bad) *bad_b = 1;
  }
  fence_async_smem();
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tm_lanes = tmem + ((uint32_t)(32 * quarter) << 16);
  const uint32_t b_s = smem_u32(Bs);
  const bool all_bad = *bad_b != 0;

  bool ok = true;
  uint32_t phase = 0;
  float cs[2 * G::BLOCKS];                     // column sums of this thread's rows
#pragma unroll
  for (int j = 0; j < 2 * G::BLOCKS; ++j) cs[j] = 0.f;
  float4 x[4];
  int par = 0;
  if ((int64_t)blockIdx.x < n_tiles)
    load_chunk(P, (int64_t)blockIdx.x * TILE_M + 32 * quarter, M, 0, part, lane, x);
  for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, par ^= 1) {
    const int64_t row0 = tile * TILE_M + 32 * quarter;
    // [h > 0] of this thread's outputs; the loads of a share of the blocks
    // are in flight while a chunk is multiplied
    uint32_t live[(8 * G::BLOCKS + 31) / 32];
    float2 h[G::H_BLOCKS][4];
#pragma unroll
    for (int w = 0; w < (8 * G::BLOCKS + 31) / 32; ++w) live[w] = 0u;
    auto take_h = [&](int c) {
#pragma unroll
      for (int cc = 0; cc < G::CHUNKS; ++cc) {
        if (cc != c) continue;
#pragma unroll
        for (int b = 0; b < G::H_BLOCKS; ++b)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int bit = 8 * (G::H_BLOCKS * cc + b) + 2 * i;
            if (bit < 8 * G::BLOCKS)
              live[bit >> 5] |= ((h[b][i].x > 0.f ? 1u : 0u) | (h[b][i].y > 0.f ? 2u : 0u)) << (bit & 31);
          }
      }
    };
#pragma unroll 1
    for (int c = 0; c < G::CHUNKS; ++c) {
      // parts of chunk c, then the loads of the next chunk
      Split2 s[4][2];
      bool bad = false;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        s[i][0] = split2(x[i].x, x[i].y, bad);
        s[i][1] = split2(x[i].z, x[i].w, bad);
      }
      if (bad) bad_tile[par] = 1;
      const bool last = c == G::CHUNKS - 1;
      const int64_t nt = last ? tile + gridDim.x : tile;
      if (nt < n_tiles) load_chunk(P, nt * TILE_M + 32 * quarter, M, last ? 0 : c + 1, part, lane, x);
      if (c > 0) {                             // the MMAs of chunk c - 1 have read A
        ok = mbar_wait(bar, phase) && ok;
        phase ^= 1u;
        fence_after();
      }
      __syncwarp();
#pragma unroll
      for (int g = 0; g < 2; ++g) {            // rows 16 g .. 16 g + 15
        const uint32_t at = tm_lanes + ((uint32_t)(16 * g) << 16) + G::A_COL + (uint32_t)(8 * part);
        const Split2 *u = s[2 * g], *v = s[2 * g + 1];
        st_16x8(at, u[0].hi, u[1].hi, v[0].hi, v[1].hi);
        st_16x8(at + A_PART, u[0].mid, u[1].mid, v[0].mid, v[1].mid);
        st_16x8(at + 2 * A_PART, u[0].lo, u[1].lo, v[0].lo, v[1].lo);
      }
      wait_st();
      fence_before();
      if (c > 0 && P.mode == 1) take_h(c - 1);
      if (__syncthreads_or(!ok)) {
        ok = false;
        break;
      }
      if (tid == 0) {
        fence_after();
        const uint32_t id = idesc(TILE_M, N);
        const uint32_t a = tmem + G::A_COL;
        // part pairs (A, Bt): the small ones first
        const int pa[6] = {0, 2, 1, 0, 1, 0}, pb[6] = {2, 0, 1, 1, 0, 0};
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          const bool hh = q == 5;
          const uint32_t d = tmem + (uint32_t)(hh && !last ? G::D_HI : G::D_SMALL);
          for (int ks = 0; ks < KCH / 16; ++ks) {
            const uint32_t bt = b_s + (uint32_t)(pb[q] * G::PART * 2 + (KCH / 8 * c + 2 * ks) * (N * 16));
            const bool acc = hh ? (last || c > 0 || ks > 0) : (c > 0 || q > 0 || ks > 0);
            mma_ts(d, a + (uint32_t)(pa[q] * A_PART + 8 * ks), desc(bt, N * 16, 128), id, acc);
          }
        }
        commit(bar);
        if (c == 0) bad_tile[par ^ 1] = 0;
      }
      if (P.mode == 1) {
#pragma unroll
        for (int b = 0; b < G::H_BLOCKS; ++b)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int64_t row = row0 + (lane >> 2) + 8 * i;
            const int col = 8 * (4 * (G::H_BLOCKS * c + b) + part) + 2 * (lane & 3);
            h[b][i] = row < M && col < N ? __ldg(reinterpret_cast<const float2*>(P.H + row * P.ldh + col))
                                         : make_float2(0.f, 0.f);
          }
      }
    }
    if (!ok) break;
    const bool plain = all_bad || bad_tile[par] != 0;
    ok = mbar_wait(bar, phase);                // a timeout ends the loop at the next barrier
    phase ^= 1u;
    fence_after();
    if (P.mode == 1) take_h(G::CHUNKS - 1);
    if (plain) {
      plain_tile<K, N>(P, tile * TILE_M, M, extra, red);
      continue;
    }
    // ---- the tile's outputs: both sums, mask, store ----
#pragma unroll
    for (int j = 0; j < G::BLOCKS; ++j) {
      const int col = 8 * (4 * j + part) + 2 * (lane & 3);
      if (4 * j + part >= N / 8) break;        // warp-uniform
      uint32_t ds[2][4], dh[2][4];
      __syncwarp();
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        const uint32_t at = tm_lanes + ((uint32_t)(16 * g) << 16) + (uint32_t)(8 * (4 * j + part));
        ld_16x8(at + G::D_SMALL, ds[g]);
        ld_16x8(at + G::D_HI, dh[g]);
      }
      wait_ld();
#pragma unroll
      for (int g = 0; g < 2; ++g)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          asm volatile("" : "+r"(ds[g][q]));
          asm volatile("" : "+r"(dh[g][q]));
        }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int64_t row = row0 + (lane >> 2) + 8 * i;
        float v[2];
#pragma unroll
        for (int e = 0; e < 2; ++e)
          v[e] = UNSCALE * (__uint_as_float(ds[i >> 1][2 * (i & 1) + e]) + __uint_as_float(dh[i >> 1][2 * (i & 1) + e]));
        if (row >= M) continue;
        if (P.mode == 1) {
          const int bit = 8 * j + 2 * i;
          const uint32_t m = live[bit >> 5] >> (bit & 31);
          v[0] = (m & 1u) ? v[0] : 0.f;
          v[1] = (m & 2u) ? v[1] : 0.f;
          cs[2 * j] += v[0];
          cs[2 * j + 1] += v[1];
        }
        float* dst = P.C + row * P.ldc + col;
        if (col + 2 <= P.n_store)
          *reinterpret_cast<float2*>(dst) = make_float2(v[0], v[1]);
        else if (col < P.n_store)
          dst[0] = v[0];
      }
    }
    fence_before();
  }
  if (!ok) set_device_error(err, VX_ERR_TIMEOUT);
  if (P.mode == 1) {
    // rows of a warp (8 lanes share a column pair), then the four row quarters
#pragma unroll
    for (int j = 0; j < 2 * G::BLOCKS; ++j) {
      float s = cs[j];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const int col = 8 * (4 * (j >> 1) + part) + 2 * lane + (j & 1);
      if (lane < 4 && col < N) red[quarter * N + col] = s;
    }
    __syncthreads();
    for (int n = tid; n < N; n += SP_THREADS)
      P.colsum[(int64_t)blockIdx.x * N + n] = (((red[n] + red[N + n]) + red[2 * N + n]) + red[3 * N + n]) + extra[n];
    // the rows of the CUDA-core kernel's larger grid
    const int64_t total = P.n_colsum * N;
    for (int64_t i = (int64_t)(gridDim.x + blockIdx.x) * N; i < total; i += (int64_t)gridDim.x * N)
      for (int n = tid; n < N; n += SP_THREADS) P.colsum[i + n] = 0.f;
  }
  fence_before();
  __syncthreads();
  if (warp == 0) {
    fence_after();
    dealloc(tmem, 512);
  }
}

// Whether C's rows share memory with A's.  A CTA here reads the first columns of
// its next tile while it writes this one, through the read-only path, and forms
// plain tiles element by element from A; the CUDA-core kernel has read all of a
// tile's A when it writes it, and takes such calls.
static bool in_place(const RowGemmParams& P) {
  if (P.M <= 0) return false;
  const float *a1 = P.A + (P.M - 1) * P.lda + P.K, *c1 = P.C + (P.M - 1) * P.ldc + P.n_store;
  return P.A < c1 && P.C < a1;
}

bool split_rowgemm_takes(const RowGemmParams& P) {
  const uintptr_t a16 = reinterpret_cast<uintptr_t>(P.A), c8 = reinterpret_cast<uintptr_t>(P.C) |
                                                               reinterpret_cast<uintptr_t>(P.mode == 1 ? P.H : nullptr);
  return P.mode != 0 && (P.K == 128 || P.K == 192) && (P.Np == P.K || P.Np == 80 || P.Np == 64) && P.lda % 4 == 0 &&
         a16 % 16 == 0 && c8 % 8 == 0 && P.ldc % 2 == 0 && (P.mode != 1 || (P.ldh % 2 == 0 && P.n_store == P.Np)) &&
         !in_place(P);
}

unsigned split_rowgemm_grid(int64_t M) {
  return (unsigned)std::min<int64_t>(std::max<int64_t>(1, (M + TILE_M - 1) / TILE_M), sm_count());
}

template <int K, int N>
static int rowgemm_go(const RowGemmParams& P, cudaStream_t st) {
  using G = RowGemmGeo<K, N>;
  const cudaError_t e =
      cudaFuncSetAttribute(split_rowgemm_kernel<K, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::SMEM);
  if (e != cudaSuccess) return cuda_status(e);
  split_rowgemm_kernel<K, N><<<split_rowgemm_grid(P.M), SP_THREADS, G::SMEM, st>>>(P, device_error_ptr());
  return launch_status();
}

int split_rowgemm_launch(const RowGemmParams& P, cudaStream_t st) {
  if (P.K == 192) {
    if (P.Np == 192) return rowgemm_go<192, 192>(P, st);
    return P.Np == 80 ? rowgemm_go<192, 80>(P, st) : rowgemm_go<192, 64>(P, st);
  }
  if (P.Np == 128) return rowgemm_go<128, 128>(P, st);
  return P.Np == 80 ? rowgemm_go<128, 80>(P, st) : rowgemm_go<128, 64>(P, st);
}

// A whole 32-byte sector in one store: two of 16 bytes would each write half.
__device__ __forceinline__ void st_sector(float* p, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

// ============================================================================
// D = A^T B over a CTA's rows
// ============================================================================
constexpr int WS_ROWS = 32;         // rows per stage
constexpr int WS_SLOTS = 2;         // stages of split operands
constexpr int WS_RAW = 3;           // stages of FP32 rows on their way
constexpr int WS_GROUP = 2;         // stages between two reads of the hi hi sums: 4 MMAs
constexpr int WS_SMALL = 8;         // and of the small ones

// An MMA truncates its running sum, which for products of one sign always falls
// short.  So every other group of hi hi products is subtracted from the sum of
// the one before it (the MMA negates A): that sum D1 shrinks to D2 = D1 - S2 and
// is truncated the other way, and the two groups together are 2 D1 - D2.
__device__ __forceinline__ bool negated(int st) { return (st / WS_GROUP) & 1; }

// M columns of A, NC of B: MN-major tiles of 8 x 8 values, 8 rows of K a block
// (element (r, c) of a part at ((r / 8) (C / 8) + c / 8) 64 + (r % 8) 8 + c % 8).
template <int M, int NC>
struct WgradGeo {
  static constexpr int MT = (M + TILE_M - 1) / TILE_M;            // M-tiles; the last may reach past M
  static constexpr int D_HI = MT * NC, COLS = 2 * MT * NC;         // tensor-memory columns
  static constexpr int TM_COLS = COLS <= 128 ? 128 : (COLS <= 256 ? 256 : 512);
  static constexpr int A_PART = WS_ROWS * M * 2, B_PART = WS_ROWS * NC * 2;   // bytes of one part
  static constexpr int SLOT = 3 * (A_PART + B_PART);
  // 12 or 8 warps split: TMEM lane quarter = warp % 4, column part = warp / 4.
  // 16 threads (8 rows x 2 float4s) take a core matrix, the M / 8 groups of
  // threads a row block of A per item; the items of B follow.  One more warp
  // issues the MMAs.
  static constexpr int THREADS = 2 * M, TG = THREADS / 16, PARTS = THREADS / 128, WARPS = THREADS / 32;
  static constexpr int A_ITEMS = WS_ROWS / 8, B_ITEMS = (WS_ROWS / 8 * (NC / 8) + TG - 1) / TG;
  static constexpr int ITEMS = A_ITEMS + B_ITEMS;
  static constexpr int BLOCKS = (NC / 16 + PARTS - 1) / PARTS;     // 16-column blocks of D per warp, every PARTS-th
  static constexpr int RAW = ITEMS * THREADS * 16;                 // bytes of one raw stage
  static constexpr size_t SMEM = (size_t)WS_SLOTS * SLOT + (size_t)WS_RAW * RAW + 128;
  static_assert(COLS <= 512 && NC % 16 == 0 && M % 64 == 0, "tensor memory");
};

template <int M, int NC>
__global__ void __launch_bounds__(WgradGeo<M, NC>::THREADS + 32, 1) split_wgrad_kernel(WgradParams P, int NP, int n_ranges, int* err) {
  using G = WgradGeo<M, NC>;
  extern __shared__ __align__(1024) uint8_t smem[];
  float4* raw = reinterpret_cast<float4*>(smem + (size_t)WS_SLOTS * G::SLOT);   // [WS_RAW][ITEMS][G::THREADS]
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + (size_t)WS_SLOTS * G::SLOT + (size_t)WS_RAW * G::RAW);
  uint64_t* full = bar + WS_SLOTS;       // a slot's parts are written; bar: its MMAs have run
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(full + WS_SLOTS);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, part = warp >> 2;
  // the column halves of a row range are neighbours: the second reads A from L2
  const int halves = NP / NC, range = blockIdx.x / halves, n0 = (int)(blockIdx.x % halves) * NC;
  const int64_t rows = rows_of(P.rows, P.rows_dev);
  const int64_t per = (rows + n_ranges - 1) / n_ranges;
  const int64_t r0 = std::min<int64_t>(rows, (int64_t)range * per);
  const int64_t r1 = std::min<int64_t>(rows, r0 + per);
  const int nst = (int)((r1 - r0 + WS_ROWS - 1) / WS_ROWS);

  if (warp == 0) alloc(tmem_slot, G::TM_COLS);
  if (tid == 0) {
    for (int s = 0; s < WS_SLOTS; ++s) {
      mbar_init(bar + s, 1);
      mbar_init(full + s, G::WARPS);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t tm_lanes = tmem + ((uint32_t)(32 * quarter) << 16);

  // A thread's float4s: row in_r of a block of 8 rows, columns 4 h.. of an
  // 8-column group: 16 lanes read two whole sectors of 8 rows and write one
  // core matrix.  Item q of A is row block q of group tg; the items of B walk
  // its groups and row blocks in turn.  A thread splits what it copied itself,
  // so the raw stages need no barrier.
  const int h = tid & 1, in_r = (tid >> 1) & 7, tg = tid >> 4;
  const float* a_src = P.A + (r0 + in_r) * P.lda + 8 * tg + 4 * h;
  const float* b_src[G::B_ITEMS];
  int b_row[G::B_ITEMS], b_dst[G::B_ITEMS], b_n[G::B_ITEMS];   // row of the stage, byte of the part, columns
#pragma unroll
  for (int q = 0; q < G::B_ITEMS; ++q) {
    const int g = tg + G::TG * q, rb = g / (NC / 8), cg = g % (NC / 8);
    const int c = n0 + 8 * cg + 4 * h;
    b_row[q] = rb < WS_ROWS / 8 ? 8 * rb + in_r : -1;
    b_dst[q] = ((rb * (NC / 8) + cg) * 64 + in_r * 8) * 2 + 8 * h;
    b_n[q] = max(0, min(4, P.N - c));        // columns of B past N count as zero
    b_src[q] = P.B + (r0 + 8 * rb + in_r) * P.ldb + c;
  }
  const int a_dst = (tg * 64 + in_r * 8) * 2 + 8 * h;
  auto load = [&](int st) {
    float4* dst = raw + (size_t)(st % WS_RAW) * (G::ITEMS * G::THREADS) + tid;
    const int64_t row = (int64_t)st * WS_ROWS;
    const int left = (int)std::min<int64_t>(r1 - r0 - row, WS_ROWS);   // rows of the stage; others count as zero
    const float* a = a_src + row * P.lda;
#pragma unroll
    for (int q = 0; q < G::A_ITEMS; ++q) {
      const bool in = 8 * q + in_r < left;
      cp_async16(dst + q * G::THREADS, in ? a + 8 * q * P.lda : P.A, in ? 16u : 0u);
    }
#pragma unroll
    for (int q = 0; q < G::B_ITEMS; ++q) {
      if (b_row[q] < 0) continue;
      const int n = b_row[q] < left ? b_n[q] : 0;
      cp_async16(dst + (G::A_ITEMS + q) * G::THREADS, n ? b_src[q] + row * P.ldb : P.A, (uint32_t)(4 * n));
    }
  };
  auto put = [&](uint8_t* dst, int step, const float4& x, bool& bad) {
    const Split2 s0 = split2(x.x, x.y, bad), s1 = split2(x.z, x.w, bad);
    *reinterpret_cast<uint2*>(dst) = make_uint2(s0.hi, s1.hi);
    *reinterpret_cast<uint2*>(dst + step) = make_uint2(s0.mid, s1.mid);
    *reinterpret_cast<uint2*>(dst + 2 * step) = make_uint2(s0.lo, s1.lo);
  };

  float acc[G::MT][G::BLOCKS][16];
#pragma unroll
  for (int mt = 0; mt < G::MT; ++mt)
#pragma unroll
    for (int b = 0; b < G::BLOCKS; ++b)
#pragma unroll
      for (int e = 0; e < 16; ++e) acc[mt][b][e] = 0.f;
  bool ok = true, bad = false;
  auto add = [&](uint32_t col, float unit) {
#pragma unroll
    for (int mt = 0; mt < G::MT; ++mt) {
      if (mt * TILE_M + 32 * quarter >= M) break;   // warp-uniform: lanes past the last column of A
#pragma unroll
      for (int b = 0; b < G::BLOCKS; ++b) {
        const int c = 16 * (G::PARTS * b + part);
        if (c >= NC) break;
        uint32_t s[16];
        ld_cols<16>(tm_lanes + col + (uint32_t)(mt * NC + c), s);
#pragma unroll
        for (int e = 0; e < 16; ++e) acc[mt][b][e] = fmaf(unit, __uint_as_float(s[e]), acc[mt][b][e]);
      }
    }
  };
  // adds the groups that end with stage st to the registers
  auto drain = [&](int st) {
    const bool paired = (st / WS_GROUP + 1) * WS_GROUP < nst;       // another group follows
    ok = mbar_wait(bar + st % WS_SLOTS, (uint32_t)((st / WS_SLOTS) & 1)) && ok;
    fence_after();
    __syncwarp();
    if ((st + 1) % WS_SMALL == 0 || st == nst - 1) add(0, UNSCALE);
    add(G::D_HI, negated(st) ? -UNSCALE : (paired ? 2.f * UNSCALE : UNSCALE));
  };

  if (warp < G::WARPS) {
#pragma unroll
    for (int st = 0; st < WS_RAW; ++st) {
      if (st < nst) load(st);
      cp_async_commit();
    }
    for (int st = 0; st < nst && ok; ++st) {
      const int slot = st % WS_SLOTS;
      if (st >= WS_SLOTS) ok = mbar_wait(bar + slot, (uint32_t)((st / WS_SLOTS - 1) & 1)) && ok;
      asm volatile("cp.async.wait_group %0;" ::"n"(WS_RAW - 1) : "memory");
      uint8_t* base = smem + (size_t)slot * G::SLOT;
      const float4* mine = raw + (size_t)(st % WS_RAW) * (G::ITEMS * G::THREADS) + tid;
#pragma unroll
      for (int q = 0; q < G::A_ITEMS; ++q) put(base + a_dst + q * (M * 16), G::A_PART, mine[q * G::THREADS], bad);
#pragma unroll
      for (int q = 0; q < G::B_ITEMS; ++q)
        if (b_row[q] >= 0)
          put(base + 3 * G::A_PART + b_dst[q], G::B_PART, mine[(G::A_ITEMS + q) * G::THREADS], bad);
      if (st + WS_RAW < nst) load(st + WS_RAW);
      cp_async_commit();
      if (st > 0 && st % WS_GROUP == 0) drain(st - 1);
      fence_async_smem();
      fence_before();
      ok = __all_sync(0xffffffffu, ok);
      if (lane == 0) mbar_arrive(full + slot);
    }
    cp_async_wait_all();
    if (nst > 0 && ok) drain(nst - 1);
  } else {
    const uint32_t id = idesc(TILE_M, NC, 1, 1);
    const int pa[6] = {0, 2, 1, 0, 1, 0}, pb[6] = {2, 0, 1, 1, 0, 0};   // the small products first
    for (int st = 0; st < nst && ok; ++st) {
      const int slot = st % WS_SLOTS;
      ok = __all_sync(0xffffffffu, mbar_wait(full + slot, (uint32_t)((st / WS_SLOTS) & 1)));
      fence_after();
      if (lane == 0 && ok) {
        const uint32_t a_s = smem_u32(smem + (size_t)slot * G::SLOT);
        // (a descriptor's address field holds 16-byte units and does not carry)
        const uint64_t a_d = desc(a_s, M * 16, 128), b_d = desc(a_s + 3 * G::A_PART, NC * 16, 128);
        const uint32_t id_hh = negated(st) ? id | IDESC_NEGATE_A : id;
        const bool first_hh = st % (2 * WS_GROUP) == 0, first_small = st % WS_SMALL == 0;
#pragma unroll
        for (int mt = 0; mt < G::MT; ++mt)
#pragma unroll
          for (int q = 0; q < 6; ++q) {
            const bool hh = q == 5;
            const uint32_t d = tmem + (uint32_t)((hh ? G::D_HI : 0) + mt * NC);
#pragma unroll
            for (int ks = 0; ks < WS_ROWS / 16; ++ks)
              mma_ss(d, a_d + (uint64_t)((pa[q] * G::A_PART + 2 * ks * (M * 16) + mt * 16 * 128) / 16),
                     b_d + (uint64_t)((pb[q] * G::B_PART + 2 * ks * (NC * 16)) / 16), hh ? id_hh : id,
                     ks > 0 || (hh ? !first_hh : !first_small || q > 0));
          }
        commit(bar + slot);
      }
      __syncwarp();
    }
  }
  if (!ok) set_device_error(err, VX_ERR_TIMEOUT);
  float* out = P.part + (size_t)range * M * NP;
  if (__syncthreads_or(bad)) {
    // a value without parts among the CTA's rows: plain FP32 sums, in the
    // order of the CUDA-core kernel
    for (int i = tid; i < M * NC; i += G::THREADS + 32) {
      const int m = i / NC, n = n0 + i % NC;
      float v = 0.f;
      if (n < P.N)
        for (int64_t r = r0; r < r1; ++r) v = fmaf(P.A[r * P.lda + m], P.B[r * P.ldb + n], v);
      out[(size_t)m * NP + n] = v;
    }
  } else if (warp < G::WARPS) {
#pragma unroll
    for (int mt = 0; mt < G::MT; ++mt) {
      const int m = mt * TILE_M + 32 * quarter + lane;
      if (m >= M) break;
#pragma unroll
      for (int b = 0; b < G::BLOCKS; ++b) {
        const int c = 16 * (G::PARTS * b + part);
        if (c >= NC) break;
#pragma unroll
        for (int e = 0; e < 16; e += 8) st_sector(out + (size_t)m * NP + n0 + c + e, acc[mt][b] + e);
      }
    }
  }
  fence_before();
  __syncthreads();
  if (warp == 0) {
    fence_after();
    dealloc(tmem, G::TM_COLS);
  }
}

bool split_wgrad_takes(const WgradParams& P, int MP, int NP) {
  const uintptr_t a16 = reinterpret_cast<uintptr_t>(P.A) | reinterpret_cast<uintptr_t>(P.B) |
                        reinterpret_cast<uintptr_t>(P.part);
  return (MP == 128 || MP == 192) && P.M == MP && (NP == MP || NP == 80 || NP == 64) && P.lda % 4 == 0 &&
         P.ldb % 4 == 0 && a16 % 16 == 0 && reinterpret_cast<uintptr_t>(P.part) % 32 == 0;
}

template <int M, int NC>
static int wgrad_go(const WgradParams& P, int NP, unsigned grid, cudaStream_t st) {
  using G = WgradGeo<M, NC>;
  const cudaError_t e =
      cudaFuncSetAttribute(split_wgrad_kernel<M, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)G::SMEM);
  if (e != cudaSuccess) return cuda_status(e);
  split_wgrad_kernel<M, NC><<<grid * (unsigned)(NP / NC), G::THREADS + 32, G::SMEM, st>>>(P, NP, (int)grid,
                                                                                   device_error_ptr());
  return launch_status();
}

int split_wgrad_launch(const WgradParams& P, int MP, int NP, unsigned grid, cudaStream_t st) {
  if (MP == 192) {
    if (NP == 192) return wgrad_go<192, 96>(P, NP, grid, st);
    return NP == 80 ? wgrad_go<192, 80>(P, NP, grid, st) : wgrad_go<192, 64>(P, NP, grid, st);
  }
  if (NP == 128) return wgrad_go<128, 128>(P, NP, grid, st);
  return NP == 80 ? wgrad_go<128, 80>(P, NP, grid, st) : wgrad_go<128, 64>(P, NP, grid, st);
}

}  // namespace mf
}  // namespace vx
