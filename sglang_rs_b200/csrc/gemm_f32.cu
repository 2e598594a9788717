// C[M, N] = A[M, K] * W[N, K]^T (+ bias[N]) to 32-bit precision on the 5th-generation tensor cores.
//
// A float is the sum of three bfloat16 numbers: its upper six bits of precision to nearest, the upper eight of what is left to nearest, and
// the rest.  A product of two floats is then nine products of bfloat16 numbers, which are exact in 32 bits; the smallest (2^-30 of the
// product) is left out, the eight others go to tcgen05.mma.  The unit truncates what it adds, so nothing is left in it for long: of every
// 64 entries of K the products of the upper parts have a sum of their own and the seven others another; both start from zero and are
// added to the result in registers, rounded to nearest.  Products of six bits by six leave twelve bits of a sum to grow into: with eight
// bits in the upper parts, the truncations of positive operands came to 3.3e-8 of the result even in sums of 32 entries; now 1.6e-8.
// Against 64 bits (2-norm, 450 rows) the error of normal operands is 3.5e-8 to 1.2e-7 at K = 63 to 12,288 (chains of 64 fused
// multiply-adds, what this kernel replaced, 1.4e-7 to 2.1e-7), of positive operands 4.1e-8 to 5.8e-8 (5.2e-8 to 1.1e-7), of normal operands
// whose rows span 2^40 1.1e-7 to 1.6e-7 (1.1e-7 to 1.9e-7).
//
// The order of additions is a function of N and K only, so a row's result depends neither on M nor on the row's place in the
// batch: sums of 64 entries are added in order to a part, and the parts (gemm_parts, at most 8) in order or in pairs to the result.
//
// The weights are the M side of the instruction.  Up to 16 rows of A: a block owns 128 rows of W and one, two or all parts of K.  More
// rows: a pair of blocks on neighbouring SMs (cta_group::2) owns 256 rows of W and TOKENS (32, 64 or 128) rows of A, of which each block
// brings 128 and TOKENS / 2, and one, two or all parts of K.  The blocks of a tile are a cluster and add their sums through shared memory.
// Warps of a block: eight bring both operands (plain loads: rows may start on any float; a thread asks for its pieces of the next chunk
// while it splits those of the one before) and leave the parts in the swizzled layout that the unit reads; one issues the products (of the
// pair, in its even block); the others read finished sums out of tensor memory and add them up.  No barrier spans the block in between.
//
// The parts of an entry below 2^-126 lose bits, or all; products below that may be lost; infinities have no parts.  The loaders keep the
// largest magnitude of each row of A and of a block's rows of W (two instructions to four entries; 2 us of 43 at 450 x 4,096 x 1,024).  A
// result that is not large enough to hide what may be lost (K 2^-97 times the sum of both magnitudes leaves 2^-27 of it; rows of zeros are
// exact), or whose operands have entries of 2^40 and more, is computed again in fused multiply-adds by a warp; one whose operands have an
// entry that is not a number is not a number.  450 x 4,096 x 1,024 on one set of weights: 38 us; with a row that is not a number 42, all rows
// 45; with a row of infinities or of entries above 2^40 97; a tenth of the entries below 2^-40 39; 250 rows of zeros 46.  (A thread a
// result that is not finite: 105 for a row that is not a number, 15,700 for all.)
//
// What bounds it: of some 3,800 cycles a chunk (450 rows) the products take 2,100 and the loaders 2,800, which split floats and wait for
// L2; and a start and end of some 11,000.  Times in us, behind another product; in brackets six products in sums of 32 entries without
// regard for ranges, then fused multiply-adds over tiles in shared memory: 450 x 4,096 x 1,024 43 (50, 124), 450 x 6,144 x 1,024 79 (79,
// 173), 450 x 1,024 x 3,072 59 (60, 94), 64 x 4,096 x 1,024 23 (25, 38), 2,048 x 4,096 x 1,024 160 (198, 456), 2,048 x 1,024 x 3,072, where
// pairs of blocks have two parts each whatever the number of tiles, 155 (110, 350).
// One and two rows are bound by latencies and by the unit's reads of W (eight per piece of it: 1,400 cycles a chunk), and slower than fused
// multiply-adds, which could not give the same bits for all row counts: 2 x 4,096 x 1,024 9.5 us (8.9, 7.9), 2 x 1,024 x 2,048 7.4 (7.2, 5.5),
// 2 x 6,144 x 1,024 11.4 (10.4, 9.1), 2 x 1,024 x 3,072 9.3 (9.9, 7.8), 2 x 151,936 x 1,024 150 (141, 160) with constant weights, as the step
// executor's are; 9.4, 8.6, 12.3, 10.3 and 148 where they are read behind the wait for the kernels ahead.  A life of one request at
// the 0.6B shape (a prompt of 8 tokens, eight decoded) takes 14.7 ms (13.9, 13.4); with six products in this form it would take 13.9.
//
// Weight layout and meaning as the reference's `linear`: row-major [out, in],
// y[o] = sum_i x[i] * W[o, i] (crates/sglang-kernel/src/cpu.rs:73-108).
//
// Every wait is bounded; if one runs out the block's warps leave their loops once the products in flight are done, its results are not
// numbers, and the error word says so.
#include "common.cuh"
#include "tcgen05_helpers.cuh"
#include <algorithm>
#include <type_traits>

SRB_DEFINE_LAST_ERROR()
SRB_DEFINE_PDL_SWITCH()

#define F32_FEATURES 128      // weight rows of a block
#define F32_CHUNK 64          // entries of K in a buffer of shared memory: a swizzled row of 128 bytes
#define F32_PLANES 3          // bfloat16 parts of a float
#define F32_EARLY_CHUNKS 4    // of the weights, that are asked into L2 ahead of the wait for the kernels ahead
#define F32_MAX_PARTS 8
#define F32_MAX_BLOCKS 8      // blocks of a cluster (16 where two share a part)

// Blocks along K for up to 16 rows, and parts of K, whose sums are rounded apart and then added.  Blocks: as many (a power of two) as are
// resident at once, two to an SM, each of at least two chunks.  Eight parts of eight blocks are added in neighbouring pairs (a sequence
// of eight roundings was 5 % less exact on positive operands than multiply-adds), for which a pair of blocks that walks all of K has no room,
// so there are four where an SM has more than one block.  Longer sums have more parts: twice as many as blocks, or up to eight of at least
// eight chunks (of positive operands, 20,000 x 4,096, the error is 5.2e-8 in eight parts and was 1.5e-7 in one).  Parts of four or six
// chunks are shared by two blocks where those are resident at once too: the second leaves the sums of its chunks apart, so that the
// order of additions stays (two rows, 1,024 x 3,072: 10.9 us by a block a part, 9.2 by two; 6,144 x 1,024, whose 384 blocks are not: 11.4 and 16).
struct F32Parts { int count, chunks, blocks; };      // parts, the chunks of each but the last, blocks (twice the parts: each shares one)
static inline F32Parts gemm_parts(int n, int k) {
  const int chunks = (k + F32_CHUNK - 1) / F32_CHUNK, tiles = (n + F32_FEATURES - 1) / F32_FEATURES;
  int blocks = 1;
  while (blocks < 4 && blocks * 4 <= chunks && tiles * blocks * 2 <= 296) blocks *= 2;
  if (blocks == 4 && chunks >= 16 && tiles * 8 <= 148) blocks = 8;
  int parts = blocks;
  if (blocks == 4 && chunks > 64) parts = 8;
  while (blocks < 4 && parts < (blocks == 1 ? F32_MAX_PARTS : 2 * blocks) && parts * 16 <= chunks) parts *= 2;
  while (parts > 1 && (parts - 1) * ((chunks + parts - 1) / parts) >= chunks) parts /= 2;        // no part is empty
  const int part_chunks = (chunks + parts - 1) / parts;
  if (parts == blocks && parts >= 4 && (part_chunks == 4 || part_chunks == 6) && chunks == parts * part_chunks && tiles * parts * 2 <= 296)
    return {parts, part_chunks, 2 * parts};
  return {parts, part_chunks, std::min(blocks, parts)};
}

struct F32Args {
  const float *a, *w, *bias;
  float* c;
  int m, n, k, lda, ldw, ldc;
  int parts, part_chunks;     // of K; chunks of a part
  int block_parts;            // parts that a block adds up: all, two or one
  int in_pairs;               // neighbouring parts are added first
  int halved;                 // two blocks share a part of four or six chunks; the second leaves the sums of its chunks apart
  float unit;                 // K * 2^-97
  int constant;               // no kernel ahead writes w
  int* error_word;            // or null
};

// TOKENS rows of A of a block, or of a pair of blocks
template <int TOKENS, bool PAIR>
struct F32Shape {
  static constexpr int X_ROWS = PAIR ? TOKENS / 2 : TOKENS;              // rows of A that a block brings
  static constexpr int LOADERS = 256;                                    // threads that bring the operands: warps 0 to 7
  static constexpr int ADDERS = PAIR ? 256 : 128;                        // threads that add up: warps 8 and up
  static constexpr int THREADS = LOADERS + ADDERS + 32;                  // the last warp issues the products
  static constexpr unsigned W_PLANE = F32_FEATURES * 128, X_PLANE = X_ROWS * 128;
  static constexpr unsigned BUFFER = F32_PLANES * (W_PLANE + X_PLANE);
  static constexpr unsigned LEVEL = PAIR ? TOKENS * F32_FEATURES * 4 : 0;      // sums of earlier parts
  static constexpr unsigned SMEM = 2 * BUFFER + LEVEL + 1024;
  static constexpr unsigned TMEM = 4 * TOKENS;                           // two sums of a chunk, two buffers of them
  static constexpr int BLOCKS = PAIR ? 1 : 2;                            // an SM
};

__host__ __device__ constexpr unsigned f32_idesc(int m, int n) {         // D float, A and B bfloat16, both K-major
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(m >> 4) << 24);
}

// ---- the forms of the instructions for one block and for a pair
template <bool PAIR>
__device__ __forceinline__ void f32_tmem_alloc(unsigned holder, unsigned columns) {
  if (!PAIR) { tmem_alloc(holder, columns); return; }
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(holder), "r"(columns) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
template <bool PAIR>
__device__ __forceinline__ void f32_tmem_dealloc(unsigned address, unsigned columns) {
  if (!PAIR) { tmem_dealloc(address, columns); return; }
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(address), "r"(columns) : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void f32_umma(unsigned tmem_d, unsigned long long w, unsigned long long x, unsigned idesc, unsigned accumulate) {
  if (!PAIR) { umma_bf16(tmem_d, w, x, idesc, accumulate); return; }
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               ::"r"(tmem_d), "l"(w), "l"(x), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on the barrier (in both blocks of the pair) once the products issued so far are done
template <bool PAIR>
__device__ __forceinline__ void f32_commit(unsigned bar, unsigned short pair_mask) {
  if (!PAIR) { umma_commit(bar); return; }
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(pair_mask) : "memory");
}
// arrives on the barrier of the block that issues the products
template <bool PAIR>
__device__ __forceinline__ void f32_arrive(unsigned bar, unsigned rank) {
  if (!PAIR) { mbar_arrive(bar); return; }
  asm volatile("{\n.reg .b32 remote;\nmapa.shared::cluster.u32 remote, %0, %1;\n"
               "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [remote];\n}\n" ::"r"(bar), "r"(rank) : "memory");
}
// twice 8 columns of this thread's lane of tensor memory, in pairs
typedef unsigned long long pair_t;          // two floats in a 64-bit register, for the packed instructions
__device__ __forceinline__ void tmem_load_2x8(unsigned first, unsigned second, pair_t (&v)[4], pair_t (&u)[4]) {
  unsigned r[16];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%16];\n"
               "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%17];\n"
               "tcgen05.wait::ld.sync.aligned;"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(first), "r"(second) : "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = ((pair_t)r[2 * i + 1] << 32) | r[2 * i];
    u[i] = ((pair_t)r[9 + 2 * i] << 32) | r[8 + 2 * i];
  }
}
__device__ __forceinline__ void add2(pair_t& acc, pair_t x) { asm volatile("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(x)); }
__device__ __forceinline__ pair_t pack2(float low, float high) {
  pair_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(low), "f"(high));
  return v;
}
__device__ __forceinline__ float low_of(pair_t v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float high_of(pair_t v) { return __uint_as_float((unsigned)(v >> 32)); }

// Four neighbouring entries of a row, zeros outside of it.  WIDE: rows start on 16 bytes and K is a multiple of 4.
template <bool WIDE>
__device__ __forceinline__ float4 load_four(const float* row, int at, int k, bool live) {
  float4 v;
  if (WIDE) {
    asm volatile(
        "{\n.reg .pred p;\nsetp.ne.b32 p, %5, 0;\nmov.b32 %0, 0;\nmov.b32 %1, 0;\nmov.b32 %2, 0;\nmov.b32 %3, 0;\n"
        "@p ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];\n}\n"
        : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w) : "l"(row + at), "r"((int)(live && at < k)) : "memory");
  } else {
    v.x = live && at < k ? row[at] : 0.f;
    v.y = live && at + 1 < k ? row[at + 1] : 0.f;
    v.z = live && at + 2 < k ? row[at + 2] : 0.f;
    v.w = live && at + 3 < k ? row[at + 3] : 0.f;
  }
  return v;
}

__device__ __forceinline__ unsigned pack_rn(float low, float high) {
  unsigned r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(high), "f"(low));
  return r;
}
__device__ __forceinline__ float upper_of(float v) { return __uint_as_float(__float_as_uint(v) & 0xffff0000u); }

// the three parts of two floats, packed: six bits to nearest, eight of what is left to nearest, the rest
__device__ __forceinline__ void split_two(float x, float y, unsigned (&part)[F32_PLANES]) {
  const unsigned ux = (__float_as_uint(x) + 0x20000u) & 0xfffc0000u, uy = (__float_as_uint(y) + 0x20000u) & 0xfffc0000u;
  part[0] = __byte_perm(ux, uy, 0x7632);
  const float rx = x - __uint_as_float(ux), ry = y - __uint_as_float(uy);        // exact
  part[1] = pack_rn(rx, ry);
  part[2] = pack_rn(rx - __uint_as_float(part[1] << 16), ry - upper_of(__uint_as_float(part[1])));
}
// Notes on a row of W: it has an entry
#define F32_LARGE 1u          // of 2^40 or more, or infinite
#define F32_NAN 2u            // that is not a number
#define F32_LIMIT 0x53800000u // the bits of 2^40
// the largest magnitude so far, or not a number
__device__ __forceinline__ void take_largest(float& high, float4 v) {
  asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(high) : "f"(v.x), "f"(v.y));
  asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(high) : "f"(v.z), "f"(v.w));
}
__device__ __noinline__ void note_row(float4 v, unsigned* row_notes) {
  float high = 0.f;
  take_largest(high, v);
  if (!(high < 0x1p40f)) atomicOr(row_notes, high != high ? F32_NAN : F32_LARGE);
}

// The parts of four neighbouring entries of row `row` into the planes of a swizzled tile (rows of 64 entries, 128 bytes; the
// 16-byte pieces of a row change places with its number), planes `plane_bytes` apart.
__device__ __forceinline__ void put_four(unsigned tile, unsigned plane_bytes, int row, int quad, float4 v, float& high) {
  unsigned p[F32_PLANES], q[F32_PLANES];
  split_two(v.x, v.y, p);
  split_two(v.z, v.w, q);
  take_largest(high, v);
  const unsigned at = tile + row * 128 + ((((unsigned)quad >> 1) ^ ((unsigned)row & 7u)) << 4) + ((unsigned)quad & 1u) * 8;
#pragma unroll
  for (int i = 0; i < F32_PLANES; ++i)
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + i * plane_bytes), "r"(p[i]), "r"(q[i]) : "memory");
}

// one element by a warp: a chain of fused multiply-adds a lane, their sums in a tree
__device__ __noinline__ float plain_element(const float* a, const float* w, int k, int lane) {
  float v = 0.f;
#pragma unroll 4
  for (int i = lane; i < k; i += 32) v = fmaf(a[i], w[i], v);
  return srb_warp_sum(v);
}

// blockIdx.x: 128 weight rows (neighbours are a pair), blockIdx.y: TOKENS rows of A, blockIdx.z: a range of K
template <int TOKENS, bool PAIR, bool WIDE>
__global__ void __launch_bounds__(F32Shape<TOKENS, PAIR>::THREADS, F32Shape<TOKENS, PAIR>::BLOCKS) gemm_f32_kernel(F32Args args) {
  using S = F32Shape<TOKENS, PAIR>;
  constexpr int LOADER_WARPS = S::LOADERS / 32, ADDER_WARPS = S::ADDERS / 32, ISSUE_WARP = LOADER_WARPS + ADDER_WARPS;
  constexpr int OWN = TOKENS / (S::ADDERS / 128);                        // an adder warp has a quarter of the lanes and OWN tokens
  constexpr int W_LOADS = F32_FEATURES * 16 / S::LOADERS, X_LOADS = S::X_ROWS * 16 / S::LOADERS, LINES = S::LOADERS / 16;
  constexpr unsigned PAIRED = PAIR ? 2 : 1;
  static_assert(X_LOADS >= 1 && OWN % 8 == 0 && S::TMEM >= 32 && S::TMEM <= 512, "shapes");
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_unaligned + 1023) & ~(uintptr_t)1023);
  // of the buffers of shared memory: filled (in the issuing block), their products done; of the sums: taken out (in the issuing block)
  __shared__ __align__(8) unsigned long long full_bar[2], done_bar[2], sum_empty[2], drain_bar;
  // the largest magnitude (as bits) of each row of A and of W, there 2^40 at most with the upper bit for rows that have notes; whether one of
  // them, of a pair in any block of the cluster, is 2^40 or more or not a number
  __shared__ unsigned x_most[S::X_ROWS], w_most, w_notes[F32_FEATURES], large;
  __shared__ unsigned tmem_holder;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const unsigned rank = srb_cluster_rank(), leader = PAIR ? rank & ~1u : rank;
  const int feature0 = blockIdx.x * F32_FEATURES, token0 = blockIdx.y * TOKENS;
  const int all_chunks = (args.k + F32_CHUNK - 1) / F32_CHUNK;
  const int half_chunks = args.part_chunks / 2;
  const int chunk0 = !PAIR && args.halved ? blockIdx.z * half_chunks : blockIdx.z * args.block_parts * args.part_chunks;
  const int chunks = !PAIR && args.halved ? half_chunks : min(all_chunks, chunk0 + args.block_parts * args.part_chunks) - chunk0;

  float4 held_w[W_LOADS];
  const int row = tid >> 4, quad = tid & 15;                             // of a loader's first load; the next ones are LINES rows on
  auto load_w = [&](int i, int chunk) {
    const int r = feature0 + row + i * LINES;
    held_w[i] = load_four<WIDE>(args.w + (size_t)r * args.ldw, (chunk0 + chunk) * F32_CHUNK + quad * 4, args.k, r < args.n && chunk < chunks);
  };
  if (warp < LOADER_WARPS && args.constant) {                            // (beside the set-up)
#pragma unroll
    for (int i = 0; i < W_LOADS; ++i) load_w(i, 0);
  }
  for (int i = tid; i < F32_FEATURES; i += S::THREADS) w_notes[i] = 0;
  if (tid == 0) {
    abort_flag = 0;
    large = 0;
    w_most = 0;
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&full_bar[b]), PAIRED * LOADER_WARPS);          // one lane of each warp, of both blocks
      mbar_init(smem_u32(&done_bar[b]), 1);
      mbar_init(smem_u32(&sum_empty[b]), PAIRED * ADDER_WARPS);
    }
    mbar_init(smem_u32(&drain_bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == ISSUE_WARP) f32_tmem_alloc<PAIR>(smem_u32(&tmem_holder), S::TMEM);
  tc_fence_before();
  if (PAIR) srb_cluster_sync();                                          // both blocks' barriers exist before anyone signals them
  else __syncthreads();
  tc_fence_after();
  const unsigned tmem_base = tmem_holder;
  const unsigned smem_base = smem_u32(smem);
  float* level = reinterpret_cast<float*>(smem + (PAIR ? 2 * S::BUFFER : TOKENS * F32_FEATURES * 4));
  // sums of an adder's feature (its lane of tensor memory)
  const int quarter = warp & 3, group = (warp - LOADER_WARPS) >> 2;
  pair_t part[OWN / 2];
  pair_t held[PAIR ? 1 : OWN / 2], middle[PAIR ? 1 : OWN / 2];           // few rows: the sums of earlier parts, or of chunks
  srb_launch_dependents();

  if (warp < LOADER_WARPS) {
    float4 held_x[X_LOADS];
    float w_high = 0.f, x_high[X_LOADS] = {};
    auto load_x = [&](int i, int chunk) {
      const int r = token0 + (int)(rank - leader) * S::X_ROWS + row + i * LINES;
      held_x[i] = load_four<WIDE>(args.a + (size_t)r * args.lda, (chunk0 + chunk) * F32_CHUNK + quad * 4, args.k, r < args.m && chunk < chunks);
    };
    // A chunk's operands are split and put in place while the next one's travel.  The second half of those is asked for only
    // behind the fence, which would wait for loads that have just been issued.
    constexpr int EARLY = W_LOADS / 2;
    auto put_w = [&](int chunk) {
#pragma unroll
      for (int i = 0; i < W_LOADS; ++i) {
        put_four(smem_base + (chunk & 1) * S::BUFFER, S::W_PLANE, row + i * LINES, quad, held_w[i], w_high);
        if (i < EARLY) load_w(i, chunk + 1);
      }
    };
    auto load_late_w = [&](int chunk) {
#pragma unroll
      for (int i = EARLY; i < W_LOADS; ++i) load_w(i, chunk);
    };
    auto put_x = [&](int chunk) {
#pragma unroll
      for (int i = 0; i < X_LOADS; ++i) {
        put_four(smem_base + (chunk & 1) * S::BUFFER + F32_PLANES * S::W_PLANE, S::X_PLANE, row + i * LINES, quad, held_x[i], x_high[i]);
      }
      fence_proxy_async_shared();
      __syncwarp();
      if (lane == 0) f32_arrive<PAIR>(smem_u32(&full_bar[chunk & 1]), leader);
#pragma unroll
      for (int i = 0; i < X_LOADS; ++i) load_x(i, chunk + 1);
    };
    auto tell_large = [&]() {
      if (!PAIR) { large = 1; return; }
      for (unsigned b = 0; b < 2 * gridDim.z; ++b)
        asm volatile("{\n.reg .b32 remote;\nmapa.shared::cluster.u32 remote, %0, %1;\nst.shared::cluster.u32 [remote], %2;\n}\n"
                     ::"r"(smem_u32(&large)), "r"(b), "r"(1u) : "memory");
    };
    int chunk = 0;
    if (args.constant) {
      // Weights that no kernel ahead writes: both buffers' share of them is split ahead of the wait.
      put_w(0);
      load_late_w(1);
      if (chunks > 1) {
        put_w(1);
        load_late_w(2);
      }
      srb_grid_dependency_wait();
#pragma unroll
      for (int i = 0; i < X_LOADS; ++i) load_x(i, 0);
      put_x(0);
      if (chunks > 1) put_x(1);
      chunk = min(2, chunks);
    } else {
      srb_grid_dependency_wait();
#pragma unroll
      for (int i = 0; i < X_LOADS; ++i) load_x(i, 0);
#pragma unroll
      for (int i = 0; i < W_LOADS; ++i) load_w(i, 0);
    }
    for (; chunk < chunks; ++chunk) {
      // the products of the chunk before the last have read this buffer
      if (chunk >= 2 && !mbar_wait_warp(smem_u32(&done_bar[chunk & 1]), ((unsigned)(chunk >> 1) & 1u) ^ 1u, &abort_flag)) break;
      put_w(chunk);
      put_x(chunk);
      load_late_w(chunk + 1);
    }
#pragma unroll
    for (int i = 0; i < X_LOADS; ++i) {                                  // (the sixteen lanes of a row are its only readers)
      const unsigned most = __reduce_max_sync(lane < 16 ? 0xffffu : 0xffff0000u, __float_as_uint(x_high[i]));
      if (quad == 0) {
        x_most[row + i * LINES] = most;
        if (most >= F32_LIMIT) tell_large();
      }
    }
    const unsigned most = __reduce_max_sync(0xffffffffu, min(__float_as_uint(w_high), F32_LIMIT));
    if (lane == 0) atomicMax(&w_most, most);
    if (!(w_high < 0x1p40f)) {                                           // which rows: in a second look
      atomicMax(&w_most, 0x80000000u | F32_LIMIT);
      tell_large();
#pragma unroll 1
      for (int i = 0; i < W_LOADS; ++i) {
        const int r = feature0 + row + i * LINES;
#pragma unroll 1
        for (chunk = 0; chunk < chunks; ++chunk)
          note_row(load_four<WIDE>(args.w + (size_t)r * args.ldw, (chunk0 + chunk) * F32_CHUNK + quad * 4, args.k, r < args.n), &w_notes[row + i * LINES]);
      }
    }
  } else if (warp == ISSUE_WARP) {
    if (rank == leader) {
      constexpr unsigned idesc = f32_idesc(PAIR ? 2 * F32_FEATURES : F32_FEATURES, TOKENS);
      const unsigned short pair_mask = (unsigned short)(3u << leader);
      const unsigned long long w_desc = smem_descriptor(smem_base), x_desc = smem_descriptor(smem_base + F32_PLANES * S::W_PLANE);
      constexpr unsigned long long W2 = S::W_PLANE >> 4, X2 = S::X_PLANE >> 4, W3 = 2 * W2, X3 = 2 * X2;
      srb_grid_dependency_wait();                                        // the limit of the waits counts from here, as for the loaders
      bool ok = true;
      auto issue = [&](auto buffer, int chunk) {
        constexpr int b = decltype(buffer)::value;
        if (!mbar_wait_warp(smem_u32(&full_bar[b]), (unsigned)(chunk >> 1) & 1u, &abort_flag) ||
            !mbar_wait_warp(smem_u32(&sum_empty[b]), ((unsigned)(chunk >> 1) & 1u) ^ 1u, &abort_flag))
          return false;
        tc_fence_after();
        if (elect_one()) {
          const unsigned upper = tmem_base + b * 2 * TOKENS, others = upper + TOKENS;
#pragma unroll
          for (int s = 0; s < F32_CHUNK / 16; ++s) {
            const unsigned long long w = w_desc + ((b * S::BUFFER) >> 4) + s * 2, x = x_desc + ((b * S::BUFFER) >> 4) + s * 2;
            f32_umma<PAIR>(upper, w, x, idesc, s > 0 ? 1u : 0u);
            f32_umma<PAIR>(others, w + W3, x + X2, idesc, s > 0 ? 1u : 0u);
            f32_umma<PAIR>(others, w + W2, x + X3, idesc, 1u);
            f32_umma<PAIR>(others, w + W3, x, idesc, 1u);
            f32_umma<PAIR>(others, w, x + X3, idesc, 1u);
            f32_umma<PAIR>(others, w + W2, x + X2, idesc, 1u);
            f32_umma<PAIR>(others, w + W2, x, idesc, 1u);
            f32_umma<PAIR>(others, w, x + X2, idesc, 1u);
          }
          f32_commit<PAIR>(smem_u32(&done_bar[b]), pair_mask);
        }
        __syncwarp();
        return true;
      };
      for (int chunk = 0; chunk < chunks && ok; chunk += 2) {
        ok = issue(std::integral_constant<int, 0>(), chunk);
        if (ok && chunk + 1 < chunks) ok = issue(std::integral_constant<int, 1>(), chunk + 1);
      }
      if (!ok) {                                                         // products that were issued may still read and write
        if (elect_one()) f32_commit<PAIR>(smem_u32(&drain_bar), (unsigned short)(1u << leader));
        __syncwarp();
        mbar_wait_timed(smem_u32(&drain_bar), 0u);
      }
    }
    srb_grid_dependency_wait();
  } else {
    if (WIDE && !(PAIR && args.constant) && tid - S::LOADERS < F32_FEATURES && feature0 + tid - S::LOADERS < args.n) {
      // The weights of the first chunks are asked into L2 (nothing is read yet, so it does not matter who writes them).
      const int first = chunk0 * F32_CHUNK, entries = min(args.k - first, min(chunks, F32_EARLY_CHUNKS) * F32_CHUNK);
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(args.w + (size_t)(feature0 + tid - S::LOADERS) * args.ldw + first), "r"(entries * 4) : "memory");
    }
    srb_grid_dependency_wait();                                          // the output may still be read by a kernel ahead
    const unsigned column = tmem_base + ((unsigned)(quarter * 32) << 16) + group * OWN;
#pragma unroll
    for (int j = 0; j < OWN / 2; ++j) part[j] = 0ull;
    bool ok = true;
    float* own_level = level + group * OWN * F32_FEATURES + quarter * 32 + lane;
    int parts_done = 0;
    for (int chunk = 0; chunk < chunks && ok; ++chunk) {
      const int b = chunk & 1;
      ok = mbar_wait_warp(smem_u32(&done_bar[b]), (unsigned)(chunk >> 1) & 1u, &abort_flag);
      if (!ok) break;
      tc_fence_after();
#pragma unroll
      for (int j0 = 0; j0 < OWN; j0 += 8) {
        pair_t upper[4], others[4];
        tmem_load_2x8(column + b * 2 * TOKENS + j0, column + b * 2 * TOKENS + TOKENS + j0, upper, others);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          add2(upper[j], others[j]);
          add2(part[j0 / 2 + j], upper[j]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) f32_arrive<PAIR>(smem_u32(&sum_empty[b]), leader);
      if (!PAIR && args.halved) {
        if (chunk + 1 < chunks && (blockIdx.z & 1)) {
#pragma unroll
          for (int j = 0; j < OWN / 2; ++j) {
            if (chunk == 0) held[PAIR ? 0 : j] = part[j];
            else middle[PAIR ? 0 : j] = part[j];
            part[j] = 0ull;
          }
        }
        continue;
      }
      if (args.block_parts == 1 || ((chunk0 + chunk + 1) % args.part_chunks != 0 && chunk + 1 != chunks)) continue;
      // A block with all parts keeps their running sum; one with two leaves the first beside the second.
      const bool last = chunk + 1 == chunks;
      if (!last || args.block_parts == args.parts) {
#pragma unroll
        for (int j = 0; j < OWN / 2; ++j) {
          if (PAIR) {
            float* at = own_level + 2 * j * F32_FEATURES;
            if (parts_done > 0) part[j] = pack2(at[0] + low_of(part[j]), at[F32_FEATURES] + high_of(part[j]));
            if (!last) {
              at[0] = low_of(part[j]);
              at[F32_FEATURES] = high_of(part[j]);
              part[j] = 0ull;
            }
          } else {
            if (parts_done > 0) add2(part[j], held[PAIR ? 0 : j]);
            if (!last) {
              held[PAIR ? 0 : j] = part[j];
              part[j] = 0ull;
            }
          }
        }
      }
      ++parts_done;
    }
  }
  __syncwarp();
  __syncthreads();                                                       // every role has left its loop: the buffers take sums
  const bool lost = abort_flag != 0;
  if (tid == 0 && lost && args.error_word) atomicOr(args.error_word, SRB_FLAG_WAIT_TIMEOUT);

  // This block's sums as [token][128 features], of two parts one behind the other.  The block of the cluster with range z of K adds rows
  // z, z + blocks, ... over all ranges.
  const int blocks = gridDim.z;
  const bool two = blocks > 1 && (args.block_parts == 2 || (!PAIR && args.halved));
  float* tile = reinterpret_cast<float*>(smem);
  if (warp >= LOADER_WARPS && warp < ISSUE_WARP) {
    const bool noted_here = large != 0;
#pragma unroll
    for (int j = 0; j < OWN; ++j) {
      const int at = (group * OWN + j) * F32_FEATURES + quarter * 32 + lane;
      tile[at] = lost ? __int_as_float(0x7fffffff) : j & 1 ? high_of(part[j / 2]) : low_of(part[j / 2]);
      // few rows: what has notes is not a number in this block's sums, whoever adds them (a pair's blocks are told)
      if (!PAIR && noted_here && (x_most[(group * OWN + j) % S::X_ROWS] >= F32_LIMIT || w_notes[quarter * 32 + lane])) tile[at] = __int_as_float(0x7fffffff);
      if (!PAIR && two) level[at] = j & 1 ? high_of(held[PAIR ? 0 : j / 2]) : low_of(held[PAIR ? 0 : j / 2]);
      if (!PAIR && args.halved && half_chunks == 3)
        level[TOKENS * F32_FEATURES + at] = j & 1 ? high_of(middle[PAIR ? 0 : j / 2]) : low_of(middle[PAIR ? 0 : j / 2]);
    }
  }
  __syncwarp();
  if (PAIR || blocks > 1) srb_cluster_sync();
  else __syncthreads();
  const unsigned first_rank = rank - blockIdx.z * PAIRED - (rank - leader);                  // of the blocks that share the tile
  auto noted = [&](const unsigned* word, unsigned peer) {
    return __float_as_uint(srb_load_peer_shared(reinterpret_cast<const float*>(word), peer));
  };
  auto store = [&](int r, int f, float v) {
    const int row = token0 + r, col = feature0 + f;
    if (row < args.m && col < args.n) args.c[(size_t)row * args.ldc + col] = v + (args.bias ? args.bias[col] : 0.f);
  };
  // Results below this may lack what the parts lose of small entries: 3 * 2^-126 an entry and 2^-126 a product.
  auto least = [&](unsigned x, unsigned w) { return args.unit * (__uint_as_float(x) + __uint_as_float(w & 0x7fffffffu) + 2.f); };
  // The first look, without the other blocks' notes: no entry is above 2^40 then.
  const float at_most_least = args.unit * 0x1.1p41f;
  auto unsure = [&](float smallest) { return (PAIR && large) || __any_sync(0xffffffffu, !(smallest >= at_most_least)); };
  // A result that may not be sure, by a whole warp with one row and 32 neighbouring columns.
  auto reconsidered = [&](int r, int f, float v) {
    const int row = token0 + r, col = feature0 + f;
    unsigned notes = 0, x = 0, w = 0;                                    // the largest magnitude of the row, and of W
    if (lane < blocks) {
      x = noted(&x_most[r % S::X_ROWS], first_rank + lane * PAIRED + r / S::X_ROWS);
      w = noted(&w_most, first_rank + lane * PAIRED + (rank - leader));
    }
    x = __reduce_max_sync(0xffffffffu, x);
    w = __reduce_max_sync(0xffffffffu, w);
    for (int b = 0; (w >> 31) && b < blocks; ++b) notes |= noted(&w_notes[f], first_rank + b * PAIRED + (rank - leader));
    const bool none = x > 0x7f800000u || (notes & F32_NAN);
    const bool again = row < args.m && col < args.n && !none && (x >= F32_LIMIT || notes || (x != 0 && fabsf(v) < least(x, w)));
    if (none) v = __int_as_float(0x7fffffff);
    for (unsigned left = __ballot_sync(0xffffffffu, again); left; left &= left - 1) {
      const int owner = __ffs(left) - 1;
      const float sum = plain_element(args.a + (size_t)row * args.lda, args.w + (size_t)(col - lane + owner) * args.ldw, args.k, lane);
      if (lane == owner) v = sum;
    }
    return v;
  };
  constexpr int LINES_AT_ONCE = S::THREADS / F32_FEATURES;
  const int col = tid & (F32_FEATURES - 1), line = tid / F32_FEATURES, first_row = (int)blockIdx.z + line * blocks;
  const int limit = min(TOKENS, args.m - token0);
  const bool live = feature0 + col < args.n;
  if (line < LINES_AT_ONCE && first_row < limit) {
    if (blocks == 1) {
      constexpr int AT_ONCE = 4;
      for (int r0 = first_row; r0 < limit; r0 += LINES_AT_ONCE * AT_ONCE) {
        float v[AT_ONCE];
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i) v[i] = r0 + i * LINES_AT_ONCE < limit ? tile[(r0 + i * LINES_AT_ONCE) * F32_FEATURES + col] : 0.f;
        float smallest = INFINITY;
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i)
          if (live && r0 + i * LINES_AT_ONCE < limit) smallest = fabsf(v[i]) < smallest || v[i] != v[i] ? fabsf(v[i]) : smallest;
        if (unsure(smallest)) {
#pragma unroll 1
          for (int i = 0; i < AT_ONCE; ++i) {
            const int r = r0 + i * LINES_AT_ONCE;
            if (r < limit) store(r, col, reconsidered(r, col, tile[r * F32_FEATURES + col]));
          }
          continue;
        }
#pragma unroll
        for (int i = 0; i < AT_ONCE; ++i)
          if (r0 + i * LINES_AT_ONCE < limit) store(r0 + i * LINES_AT_ONCE, col, v[i]);
      }
    } else {
      constexpr int MOST = PAIR ? F32_MAX_BLOCKS / 2 : F32_MAX_BLOCKS;
      for (int r = first_row; r < limit; r += LINES_AT_ONCE * blocks) {
        float v = 0.f;
        if (!PAIR && args.halved) {
          float half[F32_MAX_PARTS], one[F32_MAX_PARTS], more[F32_MAX_PARTS], last[F32_MAX_PARTS];
          const int at = r * F32_FEATURES + col;
#pragma unroll
          for (int b = 0; b < F32_MAX_PARTS; ++b) {
            half[b] = one[b] = more[b] = last[b] = 0.f;
            if (b < args.parts) {
              half[b] = srb_load_peer_shared(tile + at, first_rank + 2 * b);
              one[b] = srb_load_peer_shared(level + at, first_rank + 2 * b + 1);
              if (half_chunks == 3) more[b] = srb_load_peer_shared(level + TOKENS * F32_FEATURES + at, first_rank + 2 * b + 1);
              last[b] = srb_load_peer_shared(tile + at, first_rank + 2 * b + 1);
            }
          }
#pragma unroll
          for (int b = 0; b < F32_MAX_PARTS; ++b) half[b] = half_chunks == 3 ? half[b] + one[b] + more[b] + last[b] : half[b] + one[b] + last[b];
          if (args.in_pairs) {
#pragma unroll
            for (int b = 0; b < F32_MAX_PARTS; b += 2) v = b == 0 ? half[0] + half[1] : v + (half[b] + half[b + 1]);
          } else {
#pragma unroll
            for (int b = 0; b < F32_MAX_PARTS; ++b) v = b == 0 ? half[0] : b < args.parts ? v + half[b] : v;
          }
        } else {
          float first[MOST], second[MOST];
#pragma unroll
          for (int b = 0; b < MOST; ++b) {
            const unsigned peer = first_rank + b * PAIRED + (rank - leader);
            first[b] = second[b] = 0.f;
            if (b < blocks) {
              if (two) first[b] = srb_load_peer_shared(level + r * F32_FEATURES + col, peer);
              second[b] = srb_load_peer_shared(tile + r * F32_FEATURES + col, peer);
            }
          }
          if (args.in_pairs) {
            if (two) {
#pragma unroll
              for (int b = 0; b < MOST; ++b) v = b == 0 ? first[0] + second[0] : b < blocks ? v + (first[b] + second[b]) : v;
            } else {
#pragma unroll
              for (int b = 0; b < MOST; b += 2) v = b == 0 ? second[0] + second[1] : b < blocks ? v + (second[b] + second[b + 1]) : v;
            }
          } else {
            v = two ? first[0] + second[0] : second[0];
#pragma unroll
            for (int b = 1; b < MOST; ++b) {
              if (b < blocks) {
                if (two) v += first[b];
                v += second[b];
              }
            }
          }
        }
        if (unsure(live ? fabsf(v) : INFINITY)) v = reconsidered(r, col, v);
        store(r, col, v);
      }
    }
  }
  __syncwarp();
  if (PAIR || blocks > 1) {
    // Nobody leaves while its sums may still be read.  (What was read has arrived, as it was stored: no fence, which would wait for the
    // stores.)
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (warp == ISSUE_WARP) {
    tc_fence_after();
    f32_tmem_dealloc<PAIR>(tmem_base, S::TMEM);
  }
}

template <int TOKENS, bool PAIR, bool WIDE>
static int launch(F32Args args, int blocks, cudaStream_t s) {
  using S = F32Shape<TOKENS, PAIR>;
  auto kernel = gemm_f32_kernel<TOKENS, PAIR, WIDE>;
  SRB_CUDA_CALL(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
  if (blocks > F32_MAX_BLOCKS) SRB_CUDA_CALL(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  args.block_parts = std::max(1, args.parts / blocks);
  args.halved = blocks > args.parts;
  const unsigned features = (args.n + F32_FEATURES - 1) / F32_FEATURES;
  dim3 grid(PAIR ? (features + 1) / 2 * 2 : features, (args.m + TOKENS - 1) / TOKENS, blocks);
  if (grid.y > 65535) SRB_FAIL("gemm_f32: %d rows exceed one launch", args.m);
  SRB_CUDA_CALL(srb_launch_clustered(kernel, grid, dim3(S::THREADS), S::SMEM, s, dim3(PAIR ? 2 : 1, 1, blocks), args));
  return SRB_OK;
}

template <int TOKENS, bool WIDE>
static int launch_pairs(const F32Args& args, cudaStream_t s) {
  // Pairs that share a tile: one that takes all of K, or as many as there are parts or half of that (4 at most), whichever ends first if
  // a pair takes its chunks and some six more for its start and end.
  const long long pairs = std::max(1, srb_sm_count() / 2);
  const long long tiles = (long long)((args.n + 2 * F32_FEATURES - 1) / (2 * F32_FEATURES)) * ((args.m + TOKENS - 1) / TOKENS);
  int blocks = 1;
  long long best = -1;
  for (int b : {1, args.parts / 2, args.parts}) {
    if (b < 1 || b > F32_MAX_BLOCKS / 2 || (args.in_pairs && b != args.parts / 2)) continue;      // (two parts that are added first)
    const long long cost = (tiles * b + pairs - 1) / pairs * ((long long)args.parts / b * args.part_chunks + 6);
    if (best < 0 || cost < best) {
      best = cost;
      blocks = b;
    }
  }
  return launch<TOKENS, true, WIDE>(args, blocks, s);
}

template <bool WIDE>
static int dispatch(const F32Args& args, int few_blocks, cudaStream_t s) {
  if (args.m <= 16) return launch<16, false, WIDE>(args, few_blocks, s);
  if (args.m <= 32) return launch_pairs<32, WIDE>(args, s);
  if (args.m <= 64) return launch_pairs<64, WIDE>(args, s);
  return launch_pairs<128, WIDE>(args, s);
}

// `constant_weights`: no kernel that the stream may still run writes w (the weights of a model), so it may be read before those are done.
// `error_word` (or null) receives SRB_FLAG_WAIT_TIMEOUT.
extern "C" int srb_gemm_f32(const float* a, const float* w, const float* bias, float* c, int m, int n, int k,
                            int lda, int ldw, int ldc, int constant_weights, int* error_word, void* stream) {
  if (m <= 0 || n <= 0) return SRB_OK;
  if (k <= 0) SRB_FAIL("gemm_f32: inner size %d must be positive", k);
  if (lda < k || ldw < k || ldc < n) SRB_FAIL("gemm_f32: a leading dimension is smaller than its row");
  const F32Parts parts = gemm_parts(n, k);
  F32Args args = {};
  args.a = a; args.w = w; args.bias = bias; args.c = c;
  args.m = m; args.n = n; args.k = k; args.lda = lda; args.ldw = ldw; args.ldc = ldc;
  args.parts = parts.count; args.part_chunks = parts.chunks;
  args.in_pairs = parts.count == 8 && parts.blocks >= 8; args.constant = constant_weights; args.error_word = error_word;
  args.unit = ldexpf((float)k, -97);
  const bool wide = k % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)a | (uintptr_t)w) & 15) == 0;
  return wide ? dispatch<true>(args, parts.blocks, (cudaStream_t)stream) : dispatch<false>(args, parts.blocks, (cudaStream_t)stream);
}
