// C[M, N] = A[M, K] * W[N, K]^T (+ bias[N]) in true 32-bit: FFMA on the CUDA cores, no
// tensor cores and therefore no reduced-precision matrix mode.
//
// The order of additions is a function of N and K only, so a row's result depends neither on M nor on the row's
// place in the batch, whichever of the two kernels below computes it: K is cut into segments of SEG entries, each
// summed in index order by one chain of fused multiply-adds; the segments of a part are added in order, and the
// parts (gemm_parts, at most 8) are added in order.  (Short chains also round less than one chain over all of K.)
//
// Two kernels, because two things bound this product:
//  * few rows (up to FEW_ROWS): the weights have to be read once and everything else hides behind that.  A block owns
//    8 weight rows; all of its copies of a round of 16 segments are in flight at once (two rounds deep, 32 KB each).  A thread
//    owns one chain: (weight row, segment), for all rows of A.  More than 8 rows read the weights once per 8: 9 to 16 rows still take
//    0.53 to 0.89 of the tiles' time (weights of 64 x 64 to 151,936 x 1,024; 1.06 at 12,288 x 4,096), 17 rows 0.56 to 1.6.
//  * more rows: arithmetic.  64 x 128 tiles with 8 x 8 results a thread in packed pairs (fma.rn.f32x2: two IEEE fused
//    multiply-adds an instruction, which leaves issue slots for the loads), the parts of K in the blocks of a cluster
//    that add their tiles through shared memory, since tiles alone leave most SMs idle when N is small.
//
// Weight layout and meaning as the reference's `linear`: row-major [out, in],
// y[o] = sum_i x[i] * W[o, i] (crates/sglang-kernel/src/cpu.rs:73-108).
#include "common.cuh"

SRB_DEFINE_LAST_ERROR()
SRB_DEFINE_PDL_SWITCH()

#define SEG 64                // entries of K that one chain of additions covers
#define FEW_ROWS 16
#define FEW_FEATURES 8        // weight rows of a block
#define FEW_SEGS 16           // segments of a round: 128 threads
#define FEW_THREADS (FEW_FEATURES * FEW_SEGS)
#define ROUND_K (SEG * FEW_SEGS)
#define W_PITCH (ROUND_K + 4)                // floats; 8 neighbouring rows fall on different banks
#define X_PITCH (FEW_SEGS * (SEG + 4))       // a row's segments too

#define TILE_M 64
#define TILE_N 128
#define TILE_K 16
#define TILE_THREADS 128
#define A_PITCH (TILE_M + 4)
#define B_PITCH (TILE_N + 4)

// Parts of K: as many as make about three blocks per SM at 256 rows, each with at least one segment, equal in segments but for the last.
__host__ __device__ static inline int gemm_part_segments(int n, int k) {
  const int segments = (k + SEG - 1) / SEG;
  const int tiles = 4 * ((n + TILE_N - 1) / TILE_N);
  int parts = 1;
  while (parts < 8 && parts * 2 <= segments && tiles * parts < 444) parts *= 2;
  return (segments + parts - 1) / parts;
}

template <int BYTES>
__device__ __forceinline__ void copy_async(float* dst, const float* src, bool inside) {
  const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
  const int size = inside ? BYTES : 0;                       // 0: the destination is filled with zeros, the source is not read
  if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(size) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(src), "r"(size) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING> __device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// ---------------------------------------------------------------------------------------------- few rows
// blockIdx.x: 8 weight rows; blockIdx.y: ROWS rows of A.  WIDE: rows of both operands start on 16 bytes.
template <int ROWS, bool WIDE>
__global__ void __launch_bounds__(FEW_THREADS)
gemm_f32_few_kernel(const float* __restrict__ a, const float* __restrict__ w, const float* __restrict__ bias,
                    float* __restrict__ c, int m, int n, int k, int lda, int ldw, int ldc, int part_segments, int stages) {
  extern __shared__ __align__(16) float few_smem[];
  constexpr int STAGE = FEW_FEATURES * W_PITCH + ROWS * X_PITCH;
  constexpr int UNIT = WIDE ? 4 : 1;
  float* sums = few_smem + stages * STAGE;                   // [feature][segment][row] of a round
  const int col0 = blockIdx.x * FEW_FEATURES, row0 = blockIdx.y * ROWS;
  const int rounds = (k + ROUND_K - 1) / ROUND_K;
  const int feature = threadIdx.x & (FEW_FEATURES - 1), segment = threadIdx.x / FEW_FEATURES;

  auto load_w = [&](int round) {
    float* to = few_smem + (round % stages) * STAGE;
    const int k0 = round * ROUND_K;
    const int units = (min(k - k0, ROUND_K) + SEG - 1) / SEG * (SEG / UNIT);     // whole segments, zeros behind K
    for (int f = 0; f < FEW_FEATURES; ++f) {
      const bool live = col0 + f < n;
      const float* from = w + (size_t)(live ? col0 + f : 0) * ldw;
      for (int u = threadIdx.x; u < units; u += FEW_THREADS) {
        const int at = k0 + u * UNIT;
        const bool inside = live && at < k;
        copy_async<UNIT * 4>(to + f * W_PITCH + u * UNIT, inside ? from + at : w, inside);
      }
    }
  };
  auto load_x = [&](int round) {
    float* to = few_smem + (round % stages) * STAGE + FEW_FEATURES * W_PITCH;
    const int k0 = round * ROUND_K;
    const int units = (min(k - k0, ROUND_K) + SEG - 1) / SEG * (SEG / UNIT);
    for (int r = 0; r < ROWS; ++r) {
      const bool live = row0 + r < m;
      const float* from = a + (size_t)(live ? row0 + r : 0) * lda;
      for (int u = threadIdx.x; u < units; u += FEW_THREADS) {
        const int at = k0 + u * UNIT;
        const bool inside = live && at < k;
        const int seg = u * UNIT / SEG;
        copy_async<UNIT * 4>(to + r * X_PITCH + seg * (SEG + 4) + (u * UNIT - seg * SEG), inside ? from + at : a, inside);
      }
    }
  };

  // The weights of the first rounds are asked into L2 ahead of the wait for the kernels ahead (nothing is read yet, so it
  // does not matter who writes them); the copies follow it.
  const int early = min(stages, rounds);
  if (WIDE && threadIdx.x < FEW_FEATURES && col0 + threadIdx.x < n) {
    const int entries = min(k, early * ROUND_K);
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(w + (size_t)(col0 + threadIdx.x) * ldw), "r"(entries * 4) : "memory");
  }
  srb_launch_dependents();
  srb_grid_dependency_wait();
  for (int r = 0; r < early; ++r) {
    load_w(r);
    load_x(r);
    copy_commit();                                           // group r
  }

  float total = 0.f, part = 0.f;                             // of (feature, row) = thread, for the first 8 * ROWS threads
  constexpr int OWNED = (FEW_FEATURES * ROWS + FEW_THREADS - 1) / FEW_THREADS;
  static_assert(OWNED == 1, "a thread adds the segments of one result");
  const int own_feature = threadIdx.x / ROWS, own_row = threadIdx.x % ROWS;
  const bool owner = threadIdx.x < FEW_FEATURES * ROWS;
  for (int round = 0; round < rounds; ++round) {
    // the groups behind this round's: stages - 1 of them, or as many rounds as are left
    const int later = min(stages - 1, rounds - 1 - round);
    if (later > 0) copy_wait<1>();
    else copy_wait<0>();
    __syncthreads();
    const float* stage = few_smem + (round % stages) * STAGE;
    const int segments = (min(k - round * ROUND_K, ROUND_K) + SEG - 1) / SEG;
    if (segment < segments) {
      const float* wv = stage + feature * W_PITCH + segment * SEG;
      const float* xv = stage + FEW_FEATURES * W_PITCH + segment * (SEG + 4);
      float acc[ROWS];
#pragma unroll
      for (int r = 0; r < ROWS; ++r) acc[r] = 0.f;
#pragma unroll 8
      for (int e = 0; e < SEG; e += 4) {
        const float4 wq = *reinterpret_cast<const float4*>(wv + e);
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
          const float4 xq = *reinterpret_cast<const float4*>(xv + r * X_PITCH + e);
          acc[r] = fmaf(xq.x, wq.x, acc[r]);
          acc[r] = fmaf(xq.y, wq.y, acc[r]);
          acc[r] = fmaf(xq.z, wq.z, acc[r]);
          acc[r] = fmaf(xq.w, wq.w, acc[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < ROWS; ++r) sums[(feature * FEW_SEGS + segment) * ROWS + r] = acc[r];
    }
    __syncthreads();
    if (round + stages < rounds) {
      load_w(round + stages);
      load_x(round + stages);
      copy_commit();
    }
    if (owner) {
      for (int s = 0; s < segments; ++s) {
        part += sums[(own_feature * FEW_SEGS + s) * ROWS + own_row];
        const int done = round * FEW_SEGS + s + 1;
        if (done % part_segments == 0) {
          total += part;
          part = 0.f;
        }
      }
    }
  }
  // a last part that is shorter than the others (0 if there is none: x + 0 is x)
  total += part;
  if (owner && col0 + own_feature < n && row0 + own_row < m)
    c[(size_t)(row0 + own_row) * ldc + col0 + own_feature] = total + (bias ? bias[col0 + own_feature] : 0.f);
}

// ---------------------------------------------------------------------------------------------- more rows
typedef unsigned long long pair_t;          // two floats in a 64-bit register, for the packed instructions
__device__ __forceinline__ pair_t pack(float lo, float hi) {
  pair_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void unpack(pair_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ void fma2(pair_t& acc, pair_t x, pair_t y) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(y)); }
__device__ __forceinline__ void add2(pair_t& acc, pair_t x) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(x)); }

// blockIdx.x: 128 weight rows, blockIdx.y: 64 rows of A, blockIdx.z (the rank in the cluster): part of K
template <bool WIDE>
__global__ void __launch_bounds__(TILE_THREADS, 2)
gemm_f32_tile_kernel(const float* __restrict__ a, const float* __restrict__ w, const float* __restrict__ bias,
                     float* __restrict__ c, int m, int n, int k, int lda, int ldw, int ldc, int part_segments) {
  // two buffers of operands, [k][row]; the finished tile of a part lies over them
  __shared__ __align__(16) float smem[TILE_M * B_PITCH > 2 * TILE_K * (A_PITCH + B_PITCH) ? TILE_M * B_PITCH
                                                                                       : 2 * TILE_K * (A_PITCH + B_PITCH)];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;             // 16 x 8 threads
  const int row0 = blockIdx.y * TILE_M, col0 = blockIdx.x * TILE_N;
  const int k_begin = blockIdx.z * part_segments * SEG, k_end = min(k, k_begin + part_segments * SEG);
  const int steps = max(0, (k_end - k_begin + TILE_K - 1) / TILE_K);
  srb_launch_dependents();
  srb_grid_dependency_wait();

  // a thread brings 4 neighbouring entries of K of 2 rows of A and of 4 rows of W
  const int quad = (tid & 3) * 4, line = tid >> 2;                       // 32 lines
  float4 held[6];
  auto fetch = [&](int step) {
    const int at = k_begin + step * TILE_K + quad;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const int row = i < 2 ? row0 + line + 32 * i : col0 + line + 32 * (i - 2);
      const bool live = row < (i < 2 ? m : n);
      const float* from = i < 2 ? a + (size_t)row * lda + at : w + (size_t)row * ldw + at;
      if (WIDE) {
        held[i] = live && at < k_end ? *reinterpret_cast<const float4*>(from) : make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
        held[i].x = live && at + 0 < k_end ? from[0] : 0.f;
        held[i].y = live && at + 1 < k_end ? from[1] : 0.f;
        held[i].z = live && at + 2 < k_end ? from[2] : 0.f;
        held[i].w = live && at + 3 < k_end ? from[3] : 0.f;
      }
    }
  };
  auto put = [&](int buffer) {
    float* at_a = smem + buffer * TILE_K * (A_PITCH + B_PITCH);
    float* at_b = at_a + TILE_K * A_PITCH;
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      float* to = i < 2 ? at_a + quad * A_PITCH + line + 32 * i : at_b + quad * B_PITCH + line + 32 * (i - 2);
      const int pitch = i < 2 ? A_PITCH : B_PITCH;
      to[0] = held[i].x; to[pitch] = held[i].y; to[2 * pitch] = held[i].z; to[3 * pitch] = held[i].w;
    }
  };

  pair_t acc[8][4], sum[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = sum[i][j] = 0ull;

  if (steps > 0) {
    fetch(0);
    put(0);
  }
  __syncthreads();
  for (int step = 0; step < steps; ++step) {
    const float* at_a = smem + (step & 1) * TILE_K * (A_PITCH + B_PITCH);
    const float* at_b = at_a + TILE_K * A_PITCH;
    if (step + 1 < steps) fetch(step + 1);
#pragma unroll
    for (int e = 0; e < TILE_K; ++e) {
      const float4 a0 = *reinterpret_cast<const float4*>(at_a + e * A_PITCH + ty * 4);
      const float4 a1 = *reinterpret_cast<const float4*>(at_a + e * A_PITCH + 32 + ty * 4);
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(at_b + e * B_PITCH + tx * 4);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(at_b + e * B_PITCH + 64 + tx * 4);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const pair_t x = pack(av[i], av[i]);
        fma2(acc[i][0], x, b0.x);
        fma2(acc[i][1], x, b0.y);
        fma2(acc[i][2], x, b1.x);
        fma2(acc[i][3], x, b1.y);
      }
    }
    if ((step + 1) % (SEG / TILE_K) == 0 || step + 1 == steps) {         // a segment is complete
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          add2(sum[i][j], acc[i][j]);
          acc[i][j] = 0ull;
        }
    }
    if (step + 1 < steps) put((step + 1) & 1);
    __syncthreads();
  }

  const int parts = gridDim.z;
  if (parts > 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float* to = smem + ((i >> 2) * 32 + ty * 4 + (i & 3)) * B_PITCH + tx * 4;
      *reinterpret_cast<ulonglong2*>(to) = make_ulonglong2(sum[i][0], sum[i][1]);
      *reinterpret_cast<ulonglong2*>(to + 64) = make_ulonglong2(sum[i][2], sum[i][3]);
    }
    srb_cluster_sync();
    // block r of the cluster adds rows r, r + parts, ... of the tile over all parts, in part order
    for (int r = blockIdx.z; r < TILE_M; r += parts) {
      const int row = row0 + r, col = col0 + tid;
      if (row >= m) break;
      if (col >= n) continue;
      float v = 0.f;
      for (int b = 0; b < parts; ++b) v += srb_load_peer_shared(smem + r * B_PITCH + tid, b);
      c[(size_t)row * ldc + col] = v + (bias ? bias[col] : 0.f);
    }
    srb_cluster_sync();                                                  // nobody leaves while its tile may still be read
    return;
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = row0 + (i >> 2) * 32 + ty * 4 + (i & 3);
    if (row >= m) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = col0 + (j >> 1) * 64 + tx * 4 + (j & 1) * 2;
      float lo, hi;
      unpack(sum[i][j], lo, hi);
      if (col < n) c[(size_t)row * ldc + col] = 0.f + lo + (bias ? bias[col] : 0.f);
      if (col + 1 < n) c[(size_t)row * ldc + col + 1] = 0.f + hi + (bias ? bias[col + 1] : 0.f);
    }
  }
}

template <int ROWS, bool WIDE>
static int launch_few(const float* a, const float* w, const float* bias, float* c, int m, int n, int k, int lda, int ldw, int ldc,
                      int part_segments, cudaStream_t s) {
  constexpr size_t STAGE = (size_t)(FEW_FEATURES * W_PITCH + ROWS * X_PITCH) * sizeof(float);
  const int rounds = (k + ROUND_K - 1) / ROUND_K, stages = rounds < 2 ? rounds : 2;
  const size_t smem = stages * STAGE + (size_t)FEW_FEATURES * FEW_SEGS * ROWS * sizeof(float);
  SRB_CUDA_CALL(cudaFuncSetAttribute(gemm_f32_few_kernel<ROWS, WIDE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)(2 * STAGE + FEW_FEATURES * FEW_SEGS * ROWS * sizeof(float))));
  dim3 grid((n + FEW_FEATURES - 1) / FEW_FEATURES, (m + ROWS - 1) / ROWS);
  SRB_CUDA_CALL(srb_launch(gemm_f32_few_kernel<ROWS, WIDE>, grid, dim3(FEW_THREADS), smem, s, a, w, bias, c, m, n, k, lda, ldw, ldc,
                           part_segments, stages));
  return SRB_OK;
}

template <bool WIDE>
static int dispatch(const float* a, const float* w, const float* bias, float* c, int m, int n, int k, int lda, int ldw, int ldc,
                    cudaStream_t s) {
  const int part_segments = gemm_part_segments(n, k);
  if (m == 1) return launch_few<1, WIDE>(a, w, bias, c, m, n, k, lda, ldw, ldc, part_segments, s);
  if (m == 2) return launch_few<2, WIDE>(a, w, bias, c, m, n, k, lda, ldw, ldc, part_segments, s);
  if (m <= 4) return launch_few<4, WIDE>(a, w, bias, c, m, n, k, lda, ldw, ldc, part_segments, s);
  if (m <= FEW_ROWS) return launch_few<8, WIDE>(a, w, bias, c, m, n, k, lda, ldw, ldc, part_segments, s);
  const int segments = (k + SEG - 1) / SEG;
  dim3 grid((n + TILE_N - 1) / TILE_N, (m + TILE_M - 1) / TILE_M, (segments + part_segments - 1) / part_segments);
  if (grid.y > 65535) SRB_FAIL("gemm_f32: %d rows exceed one launch", m);
  SRB_CUDA_CALL(srb_launch_clustered(gemm_f32_tile_kernel<WIDE>, grid, dim3(TILE_THREADS), 0, s, dim3(1, 1, grid.z), a, w, bias, c,
                                     m, n, k, lda, ldw, ldc, part_segments));
  return SRB_OK;
}

extern "C" int srb_gemm_f32(const float* a, const float* w, const float* bias, float* c, int m, int n, int k,
                            int lda, int ldw, int ldc, void* stream) {
  if (m <= 0 || n <= 0) return SRB_OK;
  if (k <= 0) SRB_FAIL("gemm_f32: inner size %d must be positive", k);
  if (lda < k || ldw < k || ldc < n) SRB_FAIL("gemm_f32: a leading dimension is smaller than its row");
  if ((m + 63) / 64 > 65535) SRB_FAIL("gemm_f32: %d rows exceed one launch", m);
  const bool wide = k % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0;
  return wide ? dispatch<true>(a, w, bias, c, m, n, k, lda, ldw, ldc, (cudaStream_t)stream)
              : dispatch<false>(a, w, bias, c, m, n, k, lda, ldw, ldc, (cudaStream_t)stream);
}
