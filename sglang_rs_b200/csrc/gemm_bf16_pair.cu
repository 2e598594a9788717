// Y = X W^T in bfloat16 for many tokens (prompt portions): tiles of 256 tokens x 256 weight rows computed
// by pairs of CTAs on neighbouring SMs with tcgen05.mma.cta_group::2, in a persistent loop.
//
// The pair is a thread-block cluster of two.  The tokens are the M side: CTA r of the pair brings 128 tokens of X and
// 128 rows of W (its half of the N side) into its own shared memory by TMA; one thread of the even CTA issues the
// products for both, and each CTA's tensor memory receives the accumulator of its own tokens, a token per lane.  Per
// product step a CTA reads 8 KB of operands from shared memory and the pair asks L2 for 1 byte per 131 FLOP (a single
// CTA with a 128 x 256 tile: 12 KB and 1 byte per 85 FLOP).  The kernel is persistent: 74 pairs walk the tiles, the
// accumulator has two buffers in tensor memory, and the epilogue of a tile runs while the products of the next one are
// issued.  Six stages of 32 KB keep 160 KB of operands in flight per CTA.
//
// A token per lane is what the epilogue wants: in the gated mode the even CTA brings gate rows and the odd one the up
// rows of the same features, so a lane finds both in its own columns, and a lane's results are neighbours in the output
// row.  Eight epilogue warps (a quarter of the lanes and half of the columns each) work on their own: tensor memory ->
// registers -> a swizzled 4 KB tile of 32 tokens x 128 bytes -> one TMA store, no barrier between warps.  With the weight
// rows in the lanes (gate and up 64 lanes apart) they met through shared memory behind a barrier every 32 tokens and half
// of the four warps computed: 19 us a tile, twice what its products take at K = 2,048.
// Gate/up of 2,048 tokens: 117 -> 71 us at 2,048 x 12,288 (1,450 TFLOP/s; 384 tiles are 5.2 rounds of 74 pairs), 286 -> 244 to
// 256 us at 4,096 x 24,576 (1,610 to 1,690).  The tensor pipe under the chip's power limit bounds it, and rounds that are not full.
//
// Warps of each CTA: 0 copies (TMA), 1 issues products (even CTA only) and owns the tensor memory,
// 2-9 epilogue.  Barriers: full[s] lives in the even CTA and counts the bytes of both CTAs' copies;
// empty[s] and acc_full[b] live in both and are signalled by tcgen05.commit with a multicast to the
// pair; acc_empty[b] lives in the even CTA and is signalled by the epilogue warps of both.
// Every wait is bounded; a wait that runs out flags SRB_FLAG_WAIT_TIMEOUT and every role leaves its
// loop.  No TMA load uses multicast.
//
// Modes: bfloat16 store, with an activation or without; float store; act(gate) * up.  Each of them also over grouped rows
// (routed experts, GROUPED): the rows of X are slots in the order of their experts, a tile is up to `tile_slots` slots of one
// expert (moe_plan_kernel's list, read on the device: pairs walk as many tiles as there are) and its weight rows are that expert's.
#include "common.cuh"
#include "tcgen05_helpers.cuh"
#include "activations.cuh"
#include <algorithm>
#include <mutex>

SRB_DEFINE_LAST_ERROR()
SRB_DEFINE_PDL_SWITCH()

#define PAIR_ROWS 128         // tokens, and weight rows, per CTA (256 of each per pair)
#define PAIR_T 256            // tokens per tile (128 copied by each CTA)
#define PAIR_K 64
#define PAIR_STAGES 6
#define PAIR_EPILOGUE_WARPS 8
#define PAIR_THREADS (64 + 32 * PAIR_EPILOGUE_WARPS)
#define PAIR_BOX_BYTES 4096   // a warp's piece of the output on its way: 32 tokens x 128 bytes, swizzled
#define PAIR_EPI_BF16 0
#define PAIR_EPI_F32 1
#define PAIR_EPI_SILU 2
#define PAIR_EPI_ACT 5        // out = activation(x w^T): the plain kernel with an activation in its epilogue

struct PairArgs {
  void* out;                 // bfloat16, or float (PAIR_EPI_F32)
  int tokens, features, k, ldo, up_row_offset;
  float act_param;           // the activation's parameter, for those that have one
  int activation;            // which SRB_ACT_* the gated mode applies to the gate half, or the plain mode to its result (-1: none)
  int tiles_t, tiles_f;
  int* error_word;
  // GROUPED: [number of row tiles, first slot of every expert (experts + 1), then (expert, first slot) per row tile]
  const int* plan;
  int tile_slots, experts, expert_rows;
  const float* slot_weight;  // a factor on the input of every slot (its sums are multiplied by it), or null
};

// ---- the cta_group::2 forms of the instructions
__device__ __forceinline__ void tmem_alloc_pair(unsigned holder, unsigned columns) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(holder), "r"(columns) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(unsigned address, unsigned columns) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(address), "r"(columns) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(unsigned tmem_d, unsigned long long a_desc, unsigned long long b_desc,
                                               unsigned idesc, unsigned accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(tmem_d), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives on the barrier at this shared-memory offset in both CTAs of the pair once the products issued so far are done
__device__ __forceinline__ void umma_commit_pair(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"((unsigned short)3) : "memory");
}
// a tile copy whose bytes are counted by the barrier of the even CTA of the pair (bit 24 of a shared
// address names the odd CTA)
__device__ __forceinline__ void tma_load_2d_pair(unsigned dst, const CUtensorMap* map, unsigned bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar & 0xFEFFFFFFu), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void mbar_arrive_remote(unsigned bar, unsigned rank) {
  asm volatile("{\n.reg .b32 remote;\nmapa.shared::cluster.u32 remote, %0, %1;\n"
               "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [remote];\n}\n" ::"r"(bar), "r"(rank) : "memory");
}

__host__ __device__ constexpr unsigned pair_idesc() {
  // D float, A and B bfloat16, both K-major, M = 256 (the pair), N = 256
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(2 * PAIR_ROWS >> 3) << 17) | ((unsigned)(PAIR_T >> 4) << 24);
}

// A tile of 32 rows x 128 bytes of shared memory to the tensor of `map`; rows and columns beyond its extents are not written.
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, unsigned src, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(map), "r"(src), "r"(x), "r"(y) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void tma_stores_have_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ unsigned pack_bf16(float low, float high) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(low, high);
  return *reinterpret_cast<const unsigned*>(&v);
}

// What a tile is, the same in every role of both CTAs.
struct PairTile {
  int feature0, token0;      // the first output feature; the first token (or slot)
  int limit;                 // tokens (or slots of the expert) end here
  int w_row0;                // the expert's first weight row, or 0
};

template <int EPI, bool GROUPED>
__device__ __forceinline__ PairTile pair_tile(const PairArgs& args, int tile) {
  constexpr int FEATURES = EPI == PAIR_EPI_SILU ? PAIR_ROWS : 2 * PAIR_ROWS;
  PairTile t;
  if (GROUPED) {
    // the features of one row tile follow one another: its rows stay in L2, and an expert's weights are streamed once
    const int* first_slot = args.plan + 1;
    const int* tiles = first_slot + args.experts + 1;
    const int rt = tile / args.tiles_f;
    const int expert = tiles[2 * rt];
    t.feature0 = (tile % args.tiles_f) * FEATURES;
    t.token0 = tiles[2 * rt + 1];
    t.limit = min(t.token0 + args.tile_slots, first_slot[expert + 1]);
    t.w_row0 = expert * args.expert_rows;
  } else {
    t.feature0 = tile / args.tiles_t * FEATURES;
    t.token0 = tile % args.tiles_t * PAIR_T;
    t.limit = args.tokens;
    t.w_row0 = 0;
  }
  return t;
}

template <int EPI, bool GROUPED>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                      const __grid_constant__ CUtensorMap map_out, PairArgs args) {
  constexpr int A_BYTES = PAIR_ROWS * PAIR_K * 2;            // 16 KB: this CTA's tokens of X
  constexpr int B_BYTES = PAIR_ROWS * PAIR_K * 2;            // 16 KB: this CTA's rows of W
  constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_unaligned + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) unsigned long long full_bar[PAIR_STAGES], empty_bar[PAIR_STAGES], acc_full[2], acc_empty[2];
  __shared__ unsigned tmem_holder;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned rank = srb_cluster_rank();                  // 0: the CTA that issues the products
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int total_kb = (args.k + PAIR_K - 1) / PAIR_K;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < PAIR_STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&acc_full[b]), 1);
      mbar_init(smem_u32(&acc_empty[b]), 2 * PAIR_EPILOGUE_WARPS);      // one lane of each epilogue warp of both CTAs
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) tmem_alloc_pair(smem_u32(&tmem_holder), 512);
  tc_fence_before();
  srb_cluster_sync();                                        // both CTAs' barriers exist before anyone signals them
  tc_fence_after();
  const unsigned tmem_base = tmem_holder;
  srb_launch_dependents();
  srb_grid_dependency_wait();                                // x and the plan are written by kernels ahead
  const int num_tiles = GROUPED ? args.plan[0] * args.tiles_f : args.tiles_t * args.tiles_f;

  if (warp == 0) {
    // copies: both CTAs, each its own halves, into its own stages; the bytes count on the even CTA's barrier
    int issued = 0;
    long long round = 0;
    bool ok = true;
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      const PairTile t = pair_tile<EPI, GROUPED>(args, tile);
      // gated: the even CTA brings the gate rows, the odd one the up rows of the same features
      const int w_row = t.w_row0 + t.feature0 + (int)rank * (EPI == PAIR_EPI_SILU ? args.up_row_offset : PAIR_ROWS);
      const int token = t.token0 + (int)rank * PAIR_ROWS;
      for (int kb = 0; kb < total_kb && ok; ++kb, ++round) {
        const int s = (int)(round % PAIR_STAGES);
        const unsigned phase = (unsigned)(round / PAIR_STAGES) & 1u;
        ok = mbar_wait_warp(smem_u32(&empty_bar[s]), phase ^ 1u, &abort_flag);
        if (!ok) break;
        const unsigned bar = smem_u32(&full_bar[s]);
        const unsigned stage = smem_u32(smem) + s * STAGE_BYTES;
        const int kx = kb * PAIR_K;
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(bar, 2 * STAGE_BYTES);
          tma_load_2d_pair(stage, &map_x, bar, kx, token);
          tma_load_2d_pair(stage + A_BYTES, &map_w, bar, kx, w_row);
        }
        ++issued;
      }
    }
    // copies that were still in flight when a wait ran out write into this CTA's memory: give them time to land
    if (abort_flag && issued > 0) {
      const long long start = clock64();
      while (clock64() - start < 4000000ll) {}
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // products of the pair, issued by one elected lane of the even CTA
      constexpr unsigned idesc = pair_idesc();
      const unsigned long long a_desc0 = smem_descriptor(smem_u32(smem));
      const unsigned long long b_desc0 = smem_descriptor(smem_u32(smem) + A_BYTES);
      long long round = 0;
      int local_tile = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs, ++local_tile) {
        const int b = local_tile & 1;
        // the epilogue warps of both CTAs have read this accumulator buffer (two tiles ago)
        ok = mbar_wait_warp(smem_u32(&acc_empty[b]), (((unsigned)(local_tile >> 1)) & 1u) ^ 1u, &abort_flag);
        if (!ok) break;
        tc_fence_after();
        const unsigned acc = tmem_base + b * 2 * PAIR_ROWS;
        for (int kb = 0; kb < total_kb && ok; ++kb, ++round) {
          const int s = (int)(round % PAIR_STAGES);
          const unsigned phase = (unsigned)(round / PAIR_STAGES) & 1u;
          ok = mbar_wait_warp(smem_u32(&full_bar[s]), phase, &abort_flag);
          if (!ok) break;
          tc_fence_after();
          const unsigned long long stage_step = (unsigned long long)((s * STAGE_BYTES) >> 4);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < PAIR_K / 16; ++k) {
              const unsigned long long step = stage_step + (unsigned long long)((k * 16 * 2) >> 4);
              umma_bf16_pair(acc, a_desc0 + step, b_desc0 + step, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            }
            umma_commit_pair(smem_u32(&empty_bar[s]));       // frees the stage in both CTAs
            if (kb == total_kb - 1) umma_commit_pair(smem_u32(&acc_full[b]));
          }
          __syncwarp();
        }
      }
    }
  } else {
    // epilogue: warp w reads TMEM lanes 32 * (w % 4) .. + 32 of its own CTA, and one half of the columns
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const unsigned lane_address = tmem_base + ((unsigned)(quarter * 32) << 16);
    unsigned char* box = smem + PAIR_STAGES * STAGE_BYTES + (warp - 2) * PAIR_BOX_BYTES;
    constexpr int BOX_FEATURES = EPI == PAIR_EPI_F32 ? 32 : 64;         // 128 bytes of an output row
    constexpr int HALF_FEATURES = EPI == PAIR_EPI_SILU ? PAIR_ROWS / 2 : PAIR_ROWS;
    int local_tile = 0;
    for (int tile = pair; tile < num_tiles; tile += num_pairs, ++local_tile) {
      const int b = local_tile & 1;
      const PairTile t = pair_tile<EPI, GROUPED>(args, tile);
      const int token = t.token0 + (int)rank * PAIR_ROWS + quarter * 32;                // of lane 0
      const int live = min(t.limit - token, 32);
      const float weight = GROUPED && EPI != PAIR_EPI_F32 && args.slot_weight && lane < live ? args.slot_weight[token + lane] : 1.0f;
      if (!mbar_wait_warp(smem_u32(&acc_full[b]), ((unsigned)(local_tile >> 1)) & 1u, &abort_flag)) break;
      tc_fence_after();
      if (GROUPED && live <= 0) {
        // none of this warp's tokens is the expert's: nothing to compute or to store.  (With the padding computed, and its zeros behind
        // the last slot divided the slow way, gate/up of 130 slots of 16 experts, 1,024 x 4,096, took 66 us; 42 us now.)
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(smem_u32(&acc_empty[b]), 0);
        continue;
      }
#pragma unroll 1
      for (int c = 0; c < HALF_FEATURES; c += BOX_FEATURES) {
        const unsigned column = lane_address + b * 2 * PAIR_ROWS + half * HALF_FEATURES + c;
        // the row's 128 bytes as eight pieces; a piece goes where the 128-byte swizzle of the store expects it
        const unsigned row = smem_u32(box) + lane * 128;
        const int turn = lane & 7;
#pragma unroll
        for (int part = 0; part < BOX_FEATURES; part += 32) {
          float acc[32];
          unsigned packed[16];
          tmem_load_32(column + part, acc);
          if (EPI == PAIR_EPI_SILU) {
            float up[32];
            tmem_load_32(column + PAIR_ROWS + part, up);
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              // (a lane without a token computes with 1: a sum of 0, behind the last slot, is a division's slow case)
              if (GROUPED) { acc[j] = lane < live ? acc[j] * weight : 1.0f; up[j] *= weight; }
              acc[j] = srb_gated<GROUPED>(args.activation, acc[j], up[j], args.act_param);
            }
          } else if (EPI == PAIR_EPI_BF16 && args.activation >= 0) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              acc[j] = srb_gated<GROUPED>(args.activation, GROUPED ? (lane < live ? acc[j] * weight : 1.0f) : acc[j], 1.0f, args.act_param);
          }
          if (part == 0) {
            // the store of the box before has read it
            if (lane == 0) tma_stores_have_read();
            __syncwarp();
          }
          if (EPI == PAIR_EPI_F32) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row + ((i ^ turn) << 4)), "r"(__float_as_uint(acc[4 * i])),
                           "r"(__float_as_uint(acc[4 * i + 1])), "r"(__float_as_uint(acc[4 * i + 2])), "r"(__float_as_uint(acc[4 * i + 3])) : "memory");
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) packed[j] = pack_bf16(acc[2 * j], acc[2 * j + 1]);
#pragma unroll
            for (int i = 0; i < 4; ++i)
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(row + (((part / 8 + i) ^ turn) << 4)), "r"(packed[4 * i]),
                           "r"(packed[4 * i + 1]), "r"(packed[4 * i + 2]), "r"(packed[4 * i + 3]) : "memory");
          }
        }
        if (c + BOX_FEATURES >= HALF_FEATURES) {
          // the accumulator buffer is free for the tile after next
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_remote(smem_u32(&acc_empty[b]), 0);
        }
        const int feature = t.feature0 + half * HALF_FEATURES + c;
        if (feature >= args.features || live <= 0) continue;
        if (!GROUPED || live == 32) {
          fence_proxy_async_shared();
          __syncwarp();
          if (lane == 0) tma_store_2d(&map_out, smem_u32(box), feature, token);
        } else {
          // the rows behind the expert's last slot belong to the next one: only the live rows, 16 bytes a lane
          __syncwarp();
          constexpr int ELEMENT = EPI == PAIR_EPI_F32 ? 4 : 2;
          const int piece = lane & 7;
          for (int r = lane >> 3; r < live; r += 4) {
            if (feature + piece * (16 / ELEMENT) >= args.features) continue;        // whole pieces: features are a multiple of 8
            const uint4 v = *reinterpret_cast<const uint4*>(box + r * 128 + ((piece ^ (r & 7)) << 4));
            *reinterpret_cast<uint4*>(reinterpret_cast<unsigned char*>(args.out) +
                                      ((size_t)(token + r) * args.ldo + feature) * ELEMENT + piece * 16) = v;
          }
          __syncwarp();
        }
      }
    }
    if (lane == 0) tma_stores_have_read();                   // before this block's shared memory goes
    tc_fence_before();
  }
  __syncwarp();
  srb_cluster_sync();                                        // nobody leaves while the other CTA may still signal or read
  if (threadIdx.x == 0 && abort_flag) atomicOr(args.error_word, SRB_FLAG_WAIT_TIMEOUT);
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* entry = nullptr;
    cudaDriverEntryPointQueryResult result;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &entry, 12000, cudaEnableDefault, &result) ==
            cudaSuccess && result == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(entry);
  });
  return fn;
}

// A row-major matrix [rows, columns] (row pitch in elements) cut into boxes of [box_rows, 128 bytes] with 128-byte swizzle.
static int make_map(CUtensorMap* map, const void* base, long long rows, long long columns, long long pitch, int box_rows,
                    bool floats = false) {
  EncodeTiledFn fn = encode_tiled();
  if (!fn) SRB_FAIL("gemm_bf16_pair: the driver does not offer cuTensorMapEncodeTiled");
  const cuuint64_t dims[2] = {(cuuint64_t)columns, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)pitch * (floats ? 4 : 2)};
  const cuuint32_t box[2] = {(cuuint32_t)(floats ? 32 : 64), (cuuint32_t)box_rows};
  const cuuint32_t elem[2] = {1, 1};
  const CUresult status = fn(map, floats ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base),
                             dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (status != CUDA_SUCCESS) SRB_FAIL("gemm_bf16_pair: cuTensorMapEncodeTiled failed with %d", (int)status);
  return SRB_OK;
}

template <int EPI, bool GROUPED>
static int launch_pair(const CUtensorMap& map_w, const CUtensorMap& map_x, const CUtensorMap& map_out, const PairArgs& args,
                       int max_tiles, cudaStream_t s) {
  const int pairs = std::max(1, std::min(srb_sm_count() / 2, max_tiles));
  // the stages, a box per epilogue warp, alignment
  const size_t smem = (size_t)PAIR_STAGES * 2 * PAIR_ROWS * PAIR_K * 2 + PAIR_EPILOGUE_WARPS * PAIR_BOX_BYTES + 1024;
  auto kernel = gemm_bf16_pair_kernel<EPI, GROUPED>;
  SRB_CUDA_CALL(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  SRB_CUDA_CALL(srb_launch_clustered(kernel, dim3(2 * pairs), dim3(PAIR_THREADS), smem, s, dim3(2, 1, 1), map_w, map_x, map_out, args));
  return SRB_OK;
}

// x [tokens, k] (row pitch ldx), w [rows_of_w, k] (row pitch ldw), out [tokens, ldo], all bfloat16; k and the
// pitches multiples of 8.  mode 0: out = x w^T over `features` rows of w.  mode 5: out = activation(x w^T).  mode 2: w stacks gate rows
// [0, features) and up rows [up_row_offset, up_row_offset + features); out = act(x gate^T) * (x up^T), act being SRB_ACT_* `activation` (activations.cuh).
// `act_param`: the parameter of an activation that has one.
extern "C" int srb_gemm_bf16_pair_param(const void* x, const void* w, void* out, int tokens, int features, int k, int ldx,
                                        int ldw, int ldo, int rows_of_w, int up_row_offset, int mode, int activation,
                                        float act_param, int* error_word, void* stream) {
  if (tokens <= 0 || features <= 0) return SRB_OK;
  if (k <= 0 || k % 8 != 0 || ldx % 8 != 0 || ldw % 8 != 0 || ldo % 8 != 0)
    SRB_FAIL("gemm_bf16_pair: inner size %d and the row pitches %d, %d, %d must be positive multiples of 8", k, ldx, ldw,
             ldo);
  if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) & 15) SRB_FAIL("gemm_bf16_pair: operands must be 16-byte aligned");
  if (mode != PAIR_EPI_BF16 && mode != PAIR_EPI_SILU && mode != PAIR_EPI_ACT) SRB_FAIL("gemm_bf16_pair: unknown mode %d", mode);
  if (mode == PAIR_EPI_BF16) activation = -1;
  else if (activation < 0 || activation >= SRB_ACT_COUNT) SRB_FAIL("gemm_bf16_pair: unknown activation %d", activation);
  if (mode == PAIR_EPI_ACT) mode = PAIR_EPI_BF16;            // the plain kernel; its epilogue applies `activation`
  if (mode == PAIR_EPI_SILU && up_row_offset + features > rows_of_w)
    SRB_FAIL("gemm_bf16_pair: the up rows lie outside the %d rows of w", rows_of_w);
  if (mode == PAIR_EPI_BF16 && features > rows_of_w) SRB_FAIL("gemm_bf16_pair: %d features exceed %d rows of w", features, rows_of_w);
  CUtensorMap map_w, map_x, map_out;
  if (make_map(&map_w, w, rows_of_w, k, ldw, PAIR_ROWS) != SRB_OK || make_map(&map_x, x, tokens, k, ldx, PAIR_ROWS) != SRB_OK ||
      make_map(&map_out, out, tokens, features, ldo, 32) != SRB_OK)
    return SRB_ERR_INVALID;
  const int features_per_tile = mode == PAIR_EPI_SILU ? PAIR_ROWS : 2 * PAIR_ROWS;
  PairArgs args = {};
  args.out = out; args.tokens = tokens; args.features = features; args.k = k; args.ldo = ldo;
  args.up_row_offset = up_row_offset; args.activation = activation; args.act_param = act_param; args.error_word = error_word;
  args.tiles_t = (tokens + PAIR_T - 1) / PAIR_T;
  args.tiles_f = (features + features_per_tile - 1) / features_per_tile;
  const int tiles = args.tiles_t * args.tiles_f;
  cudaStream_t s = (cudaStream_t)stream;
  if (mode == PAIR_EPI_SILU) return launch_pair<PAIR_EPI_SILU, false>(map_w, map_x, map_out, args, tiles, s);
  return launch_pair<PAIR_EPI_BF16, false>(map_w, map_x, map_out, args, tiles, s);
}

extern "C" int srb_gemm_bf16_pair(const void* x, const void* w, void* out, int tokens, int features, int k, int ldx,
                                  int ldw, int ldo, int rows_of_w, int up_row_offset, int mode, int activation,
                                  int* error_word, void* stream) {
  if (mode != PAIR_EPI_BF16 && activation == SRB_ACT_SWIGLU_CLAMP)
    SRB_FAIL("gemm_bf16_pair: an activation with a parameter comes with its parameter");
  return srb_gemm_bf16_pair_param(x, w, out, tokens, features, k, ldx, ldw, ldo, rows_of_w, up_row_offset, mode, activation, 0.f,
                                  error_word, stream);
}

// ---- grouped: one weight matrix per expert, rows grouped by expert ---------------------------------------------
// x [slots, k]: the rows in slot order (the slots of an expert are consecutive); w [experts * expert_rows, k]; `plan` (device)
// as in PairArgs, with row tiles of `tile_slots` slots (256 at most).  mode 1: out float [slots, ldo] = x w_e^T over `features`
// rows of the expert's matrix; mode 2: the expert's matrix stacks gate rows [0, features) over up rows [up_row_offset,
// + features), out bf16 [slots, ldo] = act(gate) * up; mode 5: out bf16 = act(x w_e^T).  `slot_weight` (float [slots], or
// null): a factor on the input of every slot, taken on the 32-bit sums (modes 2 and 5).  The activations are computed with the
// full-precision exponential.
extern "C" int srb_gemm_bf16_pair_grouped(const void* x, const void* w, void* out, const int* plan, int tile_slots, int slots,
                                          int experts, int expert_rows, int features, int k, int ldo, int up_row_offset, int mode,
                                          int activation, float act_param, const float* slot_weight, int* error_word, void* stream) {
  if (slots <= 0 || features <= 0) return SRB_OK;
  if (tile_slots != 128 && tile_slots != 256) SRB_FAIL("gemm_bf16_pair_grouped: tiles of %d slots are not 128 or 256", tile_slots);
  if (k <= 0 || k % 8 != 0 || features % 8 != 0 || ldo % 8 != 0)
    SRB_FAIL("gemm_bf16_pair_grouped: the sizes %d, %d and the pitch %d must be positive multiples of 8", k, features, ldo);
  if (((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) & 15) SRB_FAIL("gemm_bf16_pair_grouped: operands must be 16-byte aligned");
  if (mode != PAIR_EPI_F32 && mode != PAIR_EPI_SILU && mode != PAIR_EPI_ACT)
    SRB_FAIL("gemm_bf16_pair_grouped: mode %d is not float, gated or activated", mode);
  if (mode != PAIR_EPI_F32 && (activation < 0 || activation >= SRB_ACT_COUNT))
    SRB_FAIL("gemm_bf16_pair_grouped: unknown activation %d", activation);
  if (!plan || experts <= 0 || expert_rows <= 0) SRB_FAIL("gemm_bf16_pair_grouped: a plan and the experts' sizes are needed");
  if ((mode == PAIR_EPI_SILU ? up_row_offset + features : features) > expert_rows)
    SRB_FAIL("gemm_bf16_pair_grouped: %d features do not fit the %d rows of an expert", features, expert_rows);
  if (ldo < features) SRB_FAIL("gemm_bf16_pair_grouped: output pitch %d is smaller than %d features", ldo, features);
  CUtensorMap map_w, map_x, map_out;
  if (make_map(&map_w, w, (long long)experts * expert_rows, k, k, PAIR_ROWS) != SRB_OK || make_map(&map_x, x, slots, k, k, PAIR_ROWS) != SRB_OK ||
      make_map(&map_out, out, slots, features, ldo, 32, mode == PAIR_EPI_F32) != SRB_OK)
    return SRB_ERR_INVALID;
  const int features_per_tile = mode == PAIR_EPI_SILU ? PAIR_ROWS : 2 * PAIR_ROWS;
  PairArgs args = {};
  args.out = out; args.tokens = slots; args.features = features; args.k = k; args.ldo = ldo;
  args.up_row_offset = up_row_offset; args.activation = activation; args.act_param = act_param; args.error_word = error_word;
  args.plan = plan; args.tile_slots = tile_slots; args.experts = experts; args.expert_rows = expert_rows; args.slot_weight = slot_weight;
  args.tiles_f = (features + features_per_tile - 1) / features_per_tile;
  const int max_tiles = (slots / tile_slots + experts) * args.tiles_f;
  cudaStream_t s = (cudaStream_t)stream;
  if (mode == PAIR_EPI_F32) return launch_pair<PAIR_EPI_F32, true>(map_w, map_x, map_out, args, max_tiles, s);
  if (mode == PAIR_EPI_SILU) return launch_pair<PAIR_EPI_SILU, true>(map_w, map_x, map_out, args, max_tiles, s);
  return launch_pair<PAIR_EPI_BF16, true>(map_w, map_x, map_out, args, max_tiles, s);
}
