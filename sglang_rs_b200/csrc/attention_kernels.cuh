// Attention over the paged cache, generic form: any head_dim, any number of query heads per kv
// head, any page size, optional window, optional sink per query head, values as wide as the keys or
// narrower, 32-bit arithmetic throughout.  T is the storage type of q, the pages and the
// output.  It is the whole attention of the 32-bit path and the fallback of the bfloat16
// path for sizes its tensor-core kernels refuse.
//
// Formula (crates/sglang-kernel/src/cpu.rs:475-517): kv head = q head / (n_q / n_kv);
// s_t = (q . k_t) * scale over the keys the row may see; softmax with the maximum
// subtracted; o = sum_t p_t v_t.  The mask is by length only: a row at position pos sees
// keys max(0, pos - window + 1) .. pos (crates/sglang-srt/src/cuda_attention.rs:285-297 for
// the causal length).  The running maximum and denominator follow the online form of
// cuda_attention.rs:137-151.
//
// Two terms that other designs add, both off by default:
//  * a sink: `sinks` holds one float per query head; exp(sink_h) is added to the softmax's denominator and to nothing
//    else.  It belongs to no key, gets no share of the values, is taken as it is (the score scale does not apply), and is
//    added exactly one time per row, also when the row's keys are split over several blocks (the merge adds it);
//  * a gate: `gates` holds one float per (row, query head) that multiplies the head's result (a mixer's output gate,
//    already passed through its sigmoid), applied where the result is normalised and written;
//  * a place inside wider rows: `out_pitch` elements lie between rows of the output, and `out_scale` multiplies every
//    result (a mixer beside another one writes its columns of the row that one output product reads);
//  * values of another width than the keys: the output and the value rows are `value_dim` wide.  With
//    `shared_values` the value of a key is the first `value_dim` entries of its key row (a cache that
//    keeps one latent row per token serves as key and as value), and v_pool is not read;
//  * first tokens that a window keeps: with `keep_first` > 0 a row also sees the sequence's first keep_first keys, however
//    far behind its window they lie;
//  * a cap on the scores: with `softcap` > 0 a score s becomes softcap * tanh(s / softcap), taken in 32-bit;
//  * two maps per head (differential attention): with `maps` 2 a head's query row and its key row are two halves,
//    [map 1 | map 2]; each map is an attention of its own over the same values, and the head's result is
//    o = a_1 - map_lambda * a_2, divided by its own root mean square and multiplied by map_scale.  The kernels see twice as
//    many query heads (`n_q`): number 2 h + t is map t of head h, whose query is the head's row with the other half taken
//    as zero; `q` itself holds each head's row once.  The generic kernel writes the maps' results as floats
//    (`float_out`) and srb_map_combine (attention.cu) joins them; the tensor-core kernels join them in their last step.
//
// Work split: one block per (row, kv head and chunk of its query heads, split); the block's warp w
// owns query head kv_head * G + chunk * heads_per_block + w (at most 32 warps, 15 for values wider than 512
// entries, so more query heads per kv head go in several chunks).  Keys are visited in blocks of 32 aligned to absolute multiples of 32,
// and a split covers `split_size` keys aligned to absolute multiples of split_size, so a
// row's arithmetic depends on its own position only, never on how the step was cut or
// what else is in the batch.  With split_size == 0 the block walks all keys and writes
// the output; otherwise it writes an unnormalised partial (acc, m, l) to scratch memory
// and srb_attention_combine merges the partials in split order.
#pragma once
#include "common.cuh"
#include <algorithm>
#include <math.h>
#include <type_traits>

#define KEY_BLOCK 32

struct AttnParams {
  const int* positions;      // [rows] position of the row in its sequence
  const int* row_request;    // [rows] index of the row's request in the block table
  const int* block_table;    // [requests, table_stride] page ids, -1 where none
  int table_stride;
  int n_q, n_kv, head_dim, page_size, num_pages;
  int window;                // 0 = all keys
  int chunk;                 // > 0: a row sees only the keys of its own chunk of `chunk` positions, counted from position 0
  int split_size;            // 0 = no split
  int max_splits;
  float scale;
  int* error_word;
  const float* sinks;        // [n_q] or null
  int value_dim;             // width of a value row and of the output
  int shared_values;         // 1: values are the first value_dim entries of the key rows
  int head_chunks;           // blocks per (row, kv head, split) along the query heads
  int heads_per_block;
  const float* gates = nullptr;   // [rows, n_q] or null: a factor on the result of every (row, query head)
  float out_scale = 1.0f;         // a factor on every result, taken in 32-bit before it is rounded
  long long out_pitch = 0;        // elements between rows of the output (a head's results are always dense); 0: n_q * value_dim
  int keep_first = 0;             // with a window: the sequence's first keys that stay visible behind it
  float softcap = 0.f;            // > 0: s -> softcap * tanh(s / softcap)
  int maps = 1;                   // 2: two maps per head, n_q counts maps
  float map_lambda = 0.f, map_scale = 1.f, map_eps = 0.f;
  int float_out = 0;              // the generic kernel's results are floats
  int steady_arrays = 0;          // no kernel that the stream may still run writes the index arrays
};

// What a caller may ask for beyond the arguments that every attention has (null pointer: nothing of it).
struct AttnTerms {
  int keep_first;
  float softcap;
  int maps;
  float map_lambda, map_scale, map_eps;
  int float_out;
};

// Takes the terms over and checks them against the mask; an error text or null.
static inline const char* srb_apply_terms(AttnParams& p, const AttnTerms* terms) {
  if (!terms) return nullptr;
  if (terms->keep_first < 0 || (terms->keep_first > 0 && p.chunk > 0)) return "first tokens are kept behind a window, not behind a chunk";
  if (!(terms->softcap >= 0.f)) return "the cap on the scores must be positive, or 0 for none";
  if (terms->maps != 1 && terms->maps != 2) return "a head has one map or two";
  if (terms->maps == 2 && (p.sinks || p.gates || p.n_q % 2 || p.head_dim % 2)) return "two maps come without sink and gate, with rows of two halves";
  p.keep_first = p.window > 0 ? terms->keep_first : 0;
  p.softcap = terms->softcap; p.maps = terms->maps;
  p.map_lambda = terms->map_lambda; p.map_scale = terms->map_scale; p.map_eps = terms->map_eps; p.float_out = terms->float_out;
  return nullptr;
}

// The pieces of `size` keys, cut at absolute multiples of `size`, that a row or tile walks: first those that hold kept first
// tokens and lie ahead of the window's first piece, then the window's.  Piece number i of the walk is piece
// srb_piece(i, ...) of the sequence.
__host__ __device__ __forceinline__ int srb_kept_pieces(int keep_first, int size, int first_piece) {
  const int kept = (keep_first + size - 1) / size;
  return kept < first_piece ? kept : first_piece;
}
__host__ __device__ __forceinline__ int srb_piece(int i, int kept_pieces, int first_piece) {
  return i < kept_pieces ? i : first_piece + i - kept_pieces;
}

// cap * tanh(x / cap) from x / cap: tanh(y) = 1 - 2 / (e^(2y) + 1), finite for every y
__device__ __forceinline__ float srb_capped(float y, float cap) { return cap * (1.0f - 2.0f / (expf(2.0f * y) + 1.0f)); }

// The first key that a row at `pos` may see: the start of its window, or of its chunk of positions, whichever is later.
// It never falls as pos grows, so the first row of a tile has the lowest first key of the tile.
__host__ __device__ __forceinline__ int srb_first_visible(int pos, int window, int chunk) {
  int begin = (window > 0 && pos + 1 > window) ? pos + 1 - window : 0;
  if (chunk > 0) {
    const int start = pos / chunk * chunk;
    begin = begin > start ? begin : start;
  }
  return begin;
}

__device__ __forceinline__ void row_key_range(const AttnParams& p, int pos, int split, int& lo, int& hi) {
  const int begin = srb_first_visible(pos, p.window, p.chunk);
  const int end = pos + 1;
  if (p.split_size == 0) {
    lo = p.keep_first > 0 ? 0 : begin;
    hi = end;
    return;
  }
  const int first = begin / p.split_size;
  const int piece = srb_piece(split, srb_kept_pieces(p.keep_first, p.split_size, first), first) * p.split_size;
  lo = piece < p.keep_first ? piece : max(begin, piece);
  hi = min(end, piece + p.split_size);
}

__device__ __forceinline__ int row_split_count(const AttnParams& p, int pos) {
  if (p.split_size == 0) return 1;
  const int begin = srb_first_visible(pos, p.window, p.chunk);
  const int first = begin / p.split_size;
  return pos / p.split_size - first + 1 + srb_kept_pieces(p.keep_first, p.split_size, first);
}

// Four neighbouring elements, 32-bit.
__device__ __forceinline__ float4 load_four(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load_four(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// The rows of a key block into a tile with `pitch` floats a row: a warp takes whole rows, four at a time, so that a lane
// has four loads in flight and no index needs a division.  `offset`: of the keys' rows, in rows of `width`; -1: zeros.
template <typename T>
__device__ __forceinline__ void load_rows(float* tile, int pitch, const T* pool, int width, const long long* offset) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int e = lane * 4; e < width; e += 128) {
    for (int first = warp * 4; first < KEY_BLOCK; first += warps * 4) {
      float4 v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const long long at = offset[first + i];
        v[i] = at < 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : load_four(pool + at * width + e);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(tile + (first + i) * pitch + e) = v[i];
    }
  }
}

// Floats: a block's tile as asynchronous copies of 16 bytes, one group: 32 key rows `k_pitch` floats apart, behind them the value rows
// (`v_pool` null: none).  `offset`: lane l has the row of the pool that holds key l, -1: zeros.  A warp takes whole rows.
__device__ __forceinline__ void copy_tile_async(float* tile, int k_pitch, const float* k_pool, const float* v_pool, int d, int vd,
                                                long long offset) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  auto copy = [](float* to, const float* from, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from), "r"(bytes) : "memory");
  };
  for (int key = warp; key < KEY_BLOCK; key += warps) {
    const long long at = __shfl_sync(0xffffffffu, offset, key);
    const int bytes = at < 0 ? 0 : 16;
    for (int e = lane * 4; e < d; e += 128) copy(tile + key * k_pitch + e, k_pool + (at < 0 ? 0 : at * d + e), bytes);
    if (v_pool)
      for (int e = lane * 4; e < vd; e += 128) copy(tile + KEY_BLOCK * k_pitch + key * vd + e, v_pool + (at < 0 ? 0 : at * vd + e), bytes);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// FORM: how a tile of 32 keys and values comes.  ATTN_NARROW: one element at a time, whatever the sizes.  ATTN_WIDE: rows of
// keys and values are multiples of four elements and start on four elements' borders; they move four elements at a time
// through registers, and a score is four chains of additions (entries 0, 4, .. / 1, 5, .. / 2, 6, .. / 3, 7, ..).  ATTN_ASYNC (floats,
// which need no conversion): the same rows as asynchronous copies, all of a tile in flight at once, into two tiles that
// take turns, so that the copies of a tile run under the arithmetic of the one before (two rows of some 230 keys in splits of 128, 16 heads
// on 8 of 128: 17 us, through registers with four loads in flight 31; such splits now go to paged_attention_split_kernel).
// A warp per query head that shares the kv head: up to 32 of them, 15 where values are wider than 512 entries (registers;
// the dispatch cuts the heads into chunks by the same numbers).
#define ATTN_WIDE_VALUE_WARPS 15
#define ATTN_NARROW 0
#define ATTN_WIDE 1
#define ATTN_ASYNC 2
template <typename T, int DIM_PER_LANE, int FORM>
__global__ void __launch_bounds__(DIM_PER_LANE <= 16 ? 1024 : 32 * ATTN_WIDE_VALUE_WARPS)
paged_attention_kernel(const T* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool, T* __restrict__ out,
                       float* __restrict__ part_acc, float* __restrict__ part_ml, AttnParams p) {
  extern __shared__ __align__(16) float smem[];
  const int d = p.head_dim, vd = p.value_dim;
  const int groups = p.n_q / p.n_kv;
  constexpr bool WIDE = FORM != ATTN_NARROW, ASYNC = FORM == ATTN_ASYNC;
  const int k_pitch = d + (WIDE ? 4 : 1);                // a lane per key: neighbouring keys on different banks
  float* k_tile = smem;                                  // [32][k_pitch]
  float* v_tile = k_tile + KEY_BLOCK * k_pitch;          // [32][vd], or the key tile itself
  const int tile_floats = KEY_BLOCK * (k_pitch + (p.shared_values ? 0 : vd));
  float* q_tile = smem + (ASYNC ? 2 : 1) * tile_floats;  // [heads_per_block][d]
  const int v_stride = p.shared_values ? k_pitch : vd;
  if (p.shared_values) v_tile = k_tile;
  __shared__ long long key_offset[KEY_BLOCK];            // which row of the pool each key's is, -1 = masked

  const int row = blockIdx.z, kv_head = blockIdx.y / p.head_chunks, chunk = blockIdx.y % p.head_chunks;
  const int split = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pos = p.positions[row];
  int lo, hi;
  row_key_range(p, pos, split, lo, hi);
  if (lo >= hi) return;
  const int request = p.row_request[row];
  const int first_head = chunk * p.heads_per_block;      // within the kv head's group
  const int here = min(p.heads_per_block, groups - first_head);
  const bool live = warp < here;                         // a warp beyond the group's heads only helps to load
  const int q_head = kv_head * groups + first_head + (live ? warp : 0);

  if (p.maps == 2) {
    // number 2 h + t: the head's row, of which map t is one half
    for (int i = threadIdx.x; i < here * d; i += blockDim.x) {
      const int number = kv_head * groups + first_head + i / d, e = i % d;
      const bool mine = (e >= (d >> 1)) == (number & 1);
      q_tile[i] = mine ? srb_to_float(q[((size_t)row * (p.n_q >> 1) + (number >> 1)) * d + e]) : 0.f;
    }
  } else {
    for (int i = threadIdx.x; i < here * d; i += blockDim.x)
      q_tile[i] = srb_to_float(q[((size_t)row * p.n_q + (size_t)kv_head * groups + first_head) * d + i]);
  }
  const int begin = srb_first_visible(pos, p.window, p.chunk);
  // the entries of a row that its score sums over: all, or one map's half
  const int e_begin = p.maps == 2 ? (q_head & 1) * (d >> 1) : 0, e_end = p.maps == 2 ? e_begin + (d >> 1) : d;

  float m = -INFINITY, l = 0.f;
  float acc[DIM_PER_LANE];
#pragma unroll
  for (int j = 0; j < DIM_PER_LANE; ++j) acc[j] = 0.f;

  // the tile after `base`: blocks without a visible key are passed over
  auto following = [&](int base) {
    const int next = base + KEY_BLOCK;
    return next >= p.keep_first && next < (begin & ~(KEY_BLOCK - 1)) ? begin & ~(KEY_BLOCK - 1) : next;
  };
  // the row of the pool that holds a key, -1 = masked
  auto pool_row = [&](int key, bool report) {
    long long offset = -1;
    if (key >= lo && key < hi && (key >= begin || key < p.keep_first)) {
      const int page = p.block_table[(size_t)request * p.table_stride + key / p.page_size];
      if (page < 0 || page >= p.num_pages) {
        if (report) atomicOr(p.error_word, SRB_FLAG_BAD_PAGE);
      } else {
        offset = ((long long)page * p.n_kv + kv_head) * p.page_size + key % p.page_size;
      }
    }
    return offset;
  };
  int base = lo & ~(KEY_BLOCK - 1), turn = 0;
  long long my_row = -1;                                 // ASYNC: of key `lane` of the tile at hand
  if constexpr (ASYNC) {
    my_row = pool_row(base + lane, warp == 0);
    copy_tile_async(smem, k_pitch, k_pool, p.shared_values ? nullptr : v_pool, d, vd, my_row);
  }
  for (int next; base < hi; base = next, turn ^= 1) {
    next = following(base);
    long long next_row = -1;
    if constexpr (ASYNC) {
      if (next < hi) {
        next_row = pool_row(next + lane, warp == 0);
        // (read last a turn ago, behind the barrier at the end of the loop)
        copy_tile_async(smem + (turn ^ 1) * tile_floats, k_pitch, k_pool, p.shared_values ? nullptr : v_pool, d, vd, next_row);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      k_tile = smem + turn * tile_floats;
      v_tile = p.shared_values ? k_tile : k_tile + KEY_BLOCK * k_pitch;
      __syncthreads();                                   // everybody's copies of this tile have landed
    } else {
      __syncthreads();                                   // previous tile fully consumed
      if (threadIdx.x < KEY_BLOCK) key_offset[threadIdx.x] = pool_row(base + threadIdx.x, true);
      __syncthreads();
    }
    float s = 0.f;
    const float* qv = q_tile + (live ? warp : 0) * d;
    const float* kv = k_tile + lane * k_pitch;
    if (WIDE) {
      if (!ASYNC) {
        load_rows(k_tile, k_pitch, k_pool, d, key_offset);
        if (!p.shared_values) load_rows(v_tile, vd, v_pool, vd, key_offset);
        __syncthreads();
      }
      // one key per lane
      float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
      for (int e = e_begin; e < e_end; e += 4) {
        const float4 x = load_four(qv + e), y = load_four(kv + e);
        s4[0] += x.x * y.x; s4[1] += x.y * y.y; s4[2] += x.z * y.z; s4[3] += x.w * y.w;
      }
      s = (s4[0] + s4[1]) + (s4[2] + s4[3]);
    } else {
      for (int i = threadIdx.x; i < KEY_BLOCK * d; i += blockDim.x) {
        const int key = i / d, e = i - key * d;
        const long long offset = key_offset[key];
        k_tile[key * k_pitch + e] = offset < 0 ? 0.f : srb_to_float(k_pool[offset * d + e]);
      }
      if (!p.shared_values) {
        for (int i = threadIdx.x; i < KEY_BLOCK * vd; i += blockDim.x) {
          const int key = i / vd, e = i - key * vd;
          const long long offset = key_offset[key];
          v_tile[key * vd + e] = offset < 0 ? 0.f : srb_to_float(v_pool[offset * vd + e]);
        }
      }
      __syncthreads();
      // one key per lane: the dot product runs over the head in index order
      for (int e = e_begin; e < e_end; ++e) s += qv[e] * kv[e];
    }
    s *= p.scale;
    if (p.softcap > 0.f) s = srb_capped(s / p.softcap, p.softcap);
    if ((ASYNC ? my_row : key_offset[lane]) < 0) s = -INFINITY;

    const float m_new = fmaxf(m, srb_warp_max(s));       // finite: the tile holds a visible key
    const float correction = expf(m - m_new);            // exp(-inf) = 0 on the first tile
    const float prob = expf(s - m_new);                  // 0 for masked keys
    l = l * correction + srb_warp_sum(prob);
    m = m_new;
#pragma unroll
    for (int j = 0; j < DIM_PER_LANE; ++j) acc[j] *= correction;
#pragma unroll 8
    for (int key = 0; key < KEY_BLOCK; ++key) {
      const float pk = __shfl_sync(0xffffffffu, prob, key);
#pragma unroll
      for (int j = 0; j < DIM_PER_LANE; ++j) {
        const int e = lane + 32 * j;
        if (e < vd) acc[j] += pk * v_tile[key * v_stride + e];
      }
    }
    if (ASYNC) {
      my_row = next_row;
      __syncthreads();                                   // this tile may be written again
    }
  }
  if (!live) return;

  if (p.split_size == 0) {
    if (p.sinks) {
      // the sink joins the denominator as one more term: exp(sink - M) with M the larger maximum
      const float sink = p.sinks[q_head];
      const float m_new = fmaxf(m, sink);
      const float correction = expf(m - m_new);
      l = l * correction + expf(sink - m_new);
#pragma unroll
      for (int j = 0; j < DIM_PER_LANE; ++j) acc[j] *= correction;
    }
    const float inv = (p.gates ? p.gates[(size_t)row * p.n_q + q_head] * p.out_scale : p.out_scale) / l;
#pragma unroll
    for (int j = 0; j < DIM_PER_LANE; ++j) {
      const int e = lane + 32 * j;
      if (e >= vd) continue;
      const size_t at = (size_t)row * p.out_pitch + (size_t)q_head * vd + e;
      if (p.float_out) reinterpret_cast<float*>(out)[at] = acc[j] * inv;
      else out[at] = srb_from_float<T>(acc[j] * inv);
    }
  } else {
    const size_t slot = ((size_t)row * p.n_q + q_head) * p.max_splits + split;
#pragma unroll
    for (int j = 0; j < DIM_PER_LANE; ++j) {
      const int e = lane + 32 * j;
      if (e < vd) part_acc[slot * vd + e] = acc[j];
    }
    if (lane == 0) {
      part_ml[slot * 2] = m;
      part_ml[slot * 2 + 1] = l;
    }
  }
}

// Rows of prompt portions in floats: as paged_attention_kernel in its ATTN_ASYNC form, tile by tile the same arithmetic, but a
// block takes ROW_WARPS / (heads per kv head) neighbouring rows, a warp per (row, head), which read the same tiles while they
// belong to the same request.  With one row per block and two query heads per kv head six warps an SM had work and every row's
// keys were copied again: 227 us for two prompts of 225 tokens and 16
// heads of 128, 95 us this way.
#define ROW_WARPS 8
template <int DIM_PER_LANE>
__global__ void __launch_bounds__(ROW_WARPS * 32)
paged_attention_rows_kernel(const float* __restrict__ q, const float* __restrict__ k_pool, const float* __restrict__ v_pool,
                            float* __restrict__ out, int rows, AttnParams p) {
  extern __shared__ __align__(16) float smem[];
  const int d = p.head_dim, vd = p.value_dim, groups = p.n_q / p.n_kv, per_block = ROW_WARPS / groups;
  const int k_pitch = d + 4, v_stride = p.shared_values ? k_pitch : vd;
  const int tile_floats = KEY_BLOCK * (k_pitch + (p.shared_values ? 0 : vd));
  float* q_tile = smem + 2 * tile_floats;                // [row][head][d]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, kv_head = blockIdx.y;
  const int row0 = blockIdx.x * per_block, row_end = min(rows, row0 + per_block);
  const int row = row0 + warp / groups, q_head = kv_head * groups + warp % groups;
  const bool mine = row < row_end;
  const int pos = mine ? p.positions[row] : -1;          // a row before position 0 is padding
  const int begin = srb_first_visible(pos, p.window, p.chunk), hi = pos + 1;
  for (int i = threadIdx.x; i < (row_end - row0) * groups * d; i += blockDim.x)
    q_tile[i] = q[((size_t)(row0 + i / (groups * d)) * p.n_q + (size_t)kv_head * groups) * d + i % (groups * d)];

  float m = -INFINITY, l = 0.f;
  float acc[DIM_PER_LANE];
#pragma unroll
  for (int j = 0; j < DIM_PER_LANE; ++j) acc[j] = 0.f;

  // a run: the block's neighbouring rows of one request; its tiles span what any of them sees
  for (int first = row0, last; first < row_end; first = last) {
    const int request = p.row_request[first];
    int low = 0x7fffffff, high = 0;
    for (last = first; last < row_end && p.row_request[last] == request; ++last) {
      const int at = p.positions[last];
      if (at < 0) continue;
      low = min(low, srb_first_visible(at, p.window, p.chunk));
      high = max(high, at + 1);
    }
    const bool in_run = mine && row >= first && row < last && pos >= 0;
    auto pool_row = [&](int key) {
      long long offset = -1;
      if (key >= low && key < high) {
        const int page = p.block_table[(size_t)request * p.table_stride + key / p.page_size];
        if (page < 0 || page >= p.num_pages) {
          if (warp == 0) atomicOr(p.error_word, SRB_FLAG_BAD_PAGE);
        } else {
          offset = ((long long)page * p.n_kv + kv_head) * p.page_size + key % p.page_size;
        }
      }
      return offset;
    };
    int base = high > 0 ? low & ~(KEY_BLOCK - 1) : 0, turn = 0;
    __syncthreads();                                     // q is there, and the run before has read its last tile
    long long my_row = -1;
    if (base < high) {
      my_row = pool_row(base + lane);
      copy_tile_async(smem, k_pitch, k_pool, p.shared_values ? nullptr : v_pool, d, vd, my_row);
    }
    for (; base < high; base += KEY_BLOCK, turn ^= 1) {
      long long next_row = -1;
      if (base + KEY_BLOCK < high) {
        next_row = pool_row(base + KEY_BLOCK + lane);
        copy_tile_async(smem + (turn ^ 1) * tile_floats, k_pitch, k_pool, p.shared_values ? nullptr : v_pool, d, vd, next_row);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncthreads();                                   // everybody's copies of this tile have landed
      // Only the keys that this row sees: the tile holds those of the block's other rows too, and their values, times a probability
      // of 0, would bring their infinities and NaN into this row.
      const int from = max(begin - base, 0), to = min(hi - base, KEY_BLOCK);
      auto tile = [&](auto whole) {
        const float* k_tile = smem + turn * tile_floats;
        const float* v_tile = p.shared_values ? k_tile : k_tile + KEY_BLOCK * k_pitch;
        const float* qv = q_tile + warp * d;
        const float* kv = k_tile + lane * k_pitch;
        float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
        for (int e = 0; e < d; e += 4) {
          const float4 x = load_four(qv + e), y = load_four(kv + e);
          s4[0] += x.x * y.x; s4[1] += x.y * y.y; s4[2] += x.z * y.z; s4[3] += x.w * y.w;
        }
        float s = (s4[0] + s4[1]) + (s4[2] + s4[3]);
        s *= p.scale;
        if (p.softcap > 0.f) s = srb_capped(s / p.softcap, p.softcap);
        if (my_row < 0 || (!whole.value && (lane < from || lane >= to))) s = -INFINITY;

        const float m_new = fmaxf(m, srb_warp_max(s));   // finite: the tile holds a visible key
        const float correction = expf(m - m_new);        // exp(-inf) = 0 on the first tile
        const float prob = expf(s - m_new);              // 0 for masked keys
        l = l * correction + srb_warp_sum(prob);
        m = m_new;
#pragma unroll
        for (int j = 0; j < DIM_PER_LANE; ++j) acc[j] *= correction;
        auto add_value = [&](int k) {
          const float pk = __shfl_sync(0xffffffffu, prob, k);
#pragma unroll
          for (int j = 0; j < DIM_PER_LANE; ++j) {
            const int e = lane + 32 * j;
            if (e < vd) acc[j] += pk * v_tile[k * v_stride + e];
          }
        };
        if constexpr (whole.value) {
#pragma unroll 8
          for (int k = 0; k < KEY_BLOCK; ++k) add_value(k);
        } else {
          for (int k = from; k < to; ++k) add_value(k);
        }
      };
      if (in_run && from < to) {
        if (from == 0 && to == KEY_BLOCK) tile(std::true_type());
        else tile(std::false_type());
      }
      my_row = next_row;
      __syncthreads();                                   // this tile may be written again
    }
  }
  if (!mine || pos < 0) return;
  if (p.sinks) {
    const float sink = p.sinks[q_head];
    const float m_new = fmaxf(m, sink);
    const float correction = expf(m - m_new);
    l = l * correction + expf(sink - m_new);
#pragma unroll
    for (int j = 0; j < DIM_PER_LANE; ++j) acc[j] *= correction;
  }
  const float inv = (p.gates ? p.gates[(size_t)row * p.n_q + q_head] * p.out_scale : p.out_scale) / l;
#pragma unroll
  for (int j = 0; j < DIM_PER_LANE; ++j) {
    const int e = lane + 32 * j;
    if (e < vd) out[(size_t)row * p.out_pitch + (size_t)q_head * vd + e] = acc[j] * inv;
  }
}

// Decoded rows in floats, a split of SPLIT_TILES * 32 keys a block: its tiles side by side, a warp per (tile, head), and the warps' results
// joined at the end in the order of the tiles.  All keys of the split are on their way at once, and its values beside them: one tile after
// the other by a warp per head, the latencies of four tiles add up (two rows of some 230 keys, 16 heads on 8 of 128, 17.1 us a layer then,
// 9.1 now).  IN_TURNS, the values follow into the memory of the keys once the scores are there, so that two to three times as many blocks
// share an SM and cover each other's loads: for launches that do not fit the SMs at once.  The arithmetic is the same, so a row's bits do
// not depend on the rows beside it.  16 heads on 8 of 128, rows x keys, us side by side / in turns / one tile after the other: 1 x 2,048 15.4
// / 18.3 / 23.1 (128 blocks), 16 x 230 21.4 / 17.4 / 23.6 (256), 8 x 2,048 67 / 47 / 69, 64 x 2,048 475 / 244 / 385 (4.4 TB/s of keys); 8
// heads of 64, three blocks an SM side by side: 8 x 512 16.9 / 19.3 / 19.8 (256), 16 x 512 29.7 / 21.1 / 23.3 (512), 64 x 2,048 252 / 160 / 214.
#define SPLIT_TILES 4
#define SPLIT_MAX_HEADS 4                                // that share a kv head
template <int DIM_PER_LANE, bool IN_TURNS>
__global__ void __launch_bounds__(32 * SPLIT_TILES * SPLIT_MAX_HEADS)
paged_attention_split_kernel(const float* __restrict__ q, const float* __restrict__ k_pool, const float* __restrict__ v_pool,
                             float* __restrict__ out, float* __restrict__ part_acc, float* __restrict__ part_ml, AttnParams p) {
  extern __shared__ __align__(16) float smem[];
  __shared__ float tile_m[SPLIT_TILES * SPLIT_MAX_HEADS], tile_l[SPLIT_TILES * SPLIT_MAX_HEADS];
  const int d = p.head_dim, vd = p.value_dim, groups = p.n_q / p.n_kv;
  const int k_pitch = d + 4, v_stride = p.shared_values ? k_pitch : vd;
  float* k_rows = smem;                                  // [128][k_pitch], behind them the values' rows
  float* v_rows = IN_TURNS || p.shared_values ? k_rows : k_rows + SPLIT_TILES * KEY_BLOCK * k_pitch;
  float* q_rows = k_rows + SPLIT_TILES * KEY_BLOCK * (IN_TURNS || p.shared_values ? max(k_pitch, v_stride) : k_pitch + vd);
  const int split = blockIdx.x, kv_head = blockIdx.y, row = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tile = warp / groups, head = warp % groups;
  srb_launch_dependents();
  if (!p.steady_arrays) srb_grid_dependency_wait();
  const int pos = p.positions[row];
  int lo, hi;
  row_key_range(p, pos, split, lo, hi);
  if (lo >= hi) {
    srb_grid_dependency_wait();
    return;
  }
  const int request = p.row_request[row];
  // the key of this lane, and the row of the pool that holds it: -1 = masked
  const int key0 = lo / p.split_size * p.split_size + tile * KEY_BLOCK, key = key0 + lane;
  const bool some = key0 < hi && key0 + KEY_BLOCK > lo;  // a key of this tile is visible
  long long at = -1;
  if (key >= lo && key < hi) {
    const int page = p.block_table[(size_t)request * p.table_stride + key / p.page_size];
    if (page < 0 || page >= p.num_pages) {
      if (head == 0) atomicOr(p.error_word, SRB_FLAG_BAD_PAGE);
    } else {
      at = ((long long)page * p.n_kv + kv_head) * p.page_size + key % p.page_size;
    }
  }
  srb_grid_dependency_wait();
  auto copy_rows = [&](float* to, int pitch, const float* pool, int width) {
    if (some) {
      for (int k = head; k < KEY_BLOCK; k += groups) {
        const long long from = __shfl_sync(0xffffffffu, at, k);
        const int bytes = from < 0 ? 0 : 16;             // 0: zeros
        for (int e = lane * 4; e < width; e += 128)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(
                           to + (size_t)(tile * KEY_BLOCK + k) * pitch + e)), "l"(pool + (from < 0 ? 0 : from * width + e)), "r"(bytes) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  copy_rows(k_rows, k_pitch, k_pool, d);
  if (IN_TURNS || p.shared_values) asm volatile("cp.async.commit_group;" ::: "memory");
  else copy_rows(v_rows, vd, v_pool, vd);
  for (int i = threadIdx.x; i < groups * d; i += blockDim.x)
    q_rows[i] = q[((size_t)row * p.n_q + (size_t)kv_head * groups) * d + i];
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  __syncthreads();

  float m = -INFINITY, l = 0.f, prob = 0.f;
  if (some) {
    // one key per lane, four chains
    const float* qv = q_rows + head * d;
    const float* kv = k_rows + (size_t)(tile * KEY_BLOCK + lane) * k_pitch;
    float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
    for (int e = 0; e < d; e += 4) {
      const float4 x = load_four(qv + e), y = load_four(kv + e);
      s4[0] += x.x * y.x; s4[1] += x.y * y.y; s4[2] += x.z * y.z; s4[3] += x.w * y.w;
    }
    float s = ((s4[0] + s4[1]) + (s4[2] + s4[3])) * p.scale;
    if (p.softcap > 0.f) s = srb_capped(s / p.softcap, p.softcap);
    if (at < 0) s = -INFINITY;
    m = srb_warp_max(s);
    prob = s == -INFINITY && m == -INFINITY ? 0.f : expf(s - m);         // 0 for masked keys
    l = srb_warp_sum(prob);
  }
  if (IN_TURNS) {
    __syncthreads();                                     // the keys are read
    copy_rows(v_rows, vd, v_pool, vd);
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float acc[DIM_PER_LANE];
#pragma unroll
  for (int j = 0; j < DIM_PER_LANE; ++j) acc[j] = 0.f;
  if (some) {
#pragma unroll 8
    for (int k = 0; k < KEY_BLOCK; ++k) {
      const float pk = __shfl_sync(0xffffffffu, prob, k);
#pragma unroll
      for (int j = 0; j < DIM_PER_LANE; ++j) {
        const int e = lane + 32 * j;
        if (e < vd) acc[j] += pk * v_rows[(size_t)(tile * KEY_BLOCK + k) * v_stride + e];
      }
    }
  }
  __syncthreads();                                       // the tiles are read: the results of the warps lie over them
  float* results = smem;                                 // [tile][head][vd]
#pragma unroll
  for (int j = 0; j < DIM_PER_LANE; ++j) {
    const int e = lane + 32 * j;
    if (e < vd) results[warp * vd + e] = acc[j];
  }
  if (lane == 0) {
    tile_m[warp] = m;
    tile_l[warp] = l;
  }
  __syncthreads();
  // a warp joins the tiles of one head
  if (warp >= groups) return;
  float most = -INFINITY;
#pragma unroll
  for (int t = 0; t < SPLIT_TILES; ++t) most = fmaxf(most, tile_m[t * groups + warp]);
  float factor[SPLIT_TILES], sum = 0.f;
#pragma unroll
  for (int t = 0; t < SPLIT_TILES; ++t) {
    const float mine = tile_m[t * groups + warp], mass = tile_l[t * groups + warp];
    factor[t] = mine == -INFINITY ? (mass == 0.f ? 0.f : 1.f) : expf(mine - most);        // (a mass that is not a number stays)
    sum += mass * factor[t];
  }
  const int q_head = kv_head * groups + warp;
  if (p.max_splits == 1) {
    // the one split of a short context: what attention_combine_kernel makes of it, which is not launched then
    if (row_split_count(p, pos) > 1 && q_head == 0 && lane == 0 && p.error_word) atomicOr(p.error_word, SRB_FLAG_TOO_FEW_SPLITS);
    const float top = p.sinks ? fmaxf(p.sinks[q_head], most) : most;
    const float scale = expf(most - top), mass = (p.sinks ? expf(p.sinks[q_head] - top) : 0.f) + sum * scale;
    const float inv = (p.gates ? p.gates[(size_t)row * p.n_q + q_head] * p.out_scale : p.out_scale) / mass;
#pragma unroll
    for (int j = 0; j < DIM_PER_LANE; ++j) {
      const int e = lane + 32 * j;
      if (e >= vd) continue;
      float v = 0.f;
#pragma unroll
      for (int t = 0; t < SPLIT_TILES; ++t) v += results[(t * groups + warp) * vd + e] * factor[t];
      out[(size_t)row * p.out_pitch + (size_t)q_head * vd + e] = v * scale * inv;
    }
    return;
  }
  const size_t slot = ((size_t)row * p.n_q + q_head) * p.max_splits + split;
#pragma unroll
  for (int j = 0; j < DIM_PER_LANE; ++j) {
    const int e = lane + 32 * j;
    if (e >= vd) continue;
    float v = 0.f;
#pragma unroll
    for (int t = 0; t < SPLIT_TILES; ++t) v += results[(t * groups + warp) * vd + e] * factor[t];
    part_acc[slot * vd + e] = v;
  }
  if (lane == 0) {
    part_ml[slot * 2] = most;
    part_ml[slot * 2 + 1] = sum;
  }
}

// Merges a row's partials in split order: M = max m_s, out = sum acc_s e^(m_s - M) / sum l_s e^(m_s - M).
template <typename T>
__global__ void attention_combine_kernel(const float* __restrict__ part_acc, const float* __restrict__ part_ml,
                                         T* __restrict__ out, AttnParams p) {
  const int row = blockIdx.x, q_head = blockIdx.y;
  srb_launch_dependents();
  srb_grid_dependency_wait();
  const int pos = p.positions[row];
  if (pos < 0) return;                                   // a padding row: no block wrote partials for it
  const int wanted = row_split_count(p, pos);
  if (wanted > p.max_splits) {
    // the launch has too few blocks along the splits for this row: its newest keys were left out
    if (q_head == 0 && threadIdx.x == 0 && p.error_word) atomicOr(p.error_word, SRB_FLAG_TOO_FEW_SPLITS);
  }
  const int count = min(wanted, p.max_splits);
  const size_t first = ((size_t)row * p.n_q + q_head) * p.max_splits;
  float m = p.sinks ? p.sinks[q_head] : -INFINITY;
  for (int s = 0; s < count; ++s) m = fmaxf(m, part_ml[(first + s) * 2]);
  float l = p.sinks ? expf(p.sinks[q_head] - m) : 0.f;   // the sink counts once, whatever the number of splits
  for (int s = 0; s < count; ++s) l += part_ml[(first + s) * 2 + 1] * expf(part_ml[(first + s) * 2] - m);
  const float inv = (p.gates ? p.gates[(size_t)row * p.n_q + q_head] * p.out_scale : p.out_scale) / l;
  for (int e = threadIdx.x; e < p.value_dim; e += blockDim.x) {
    float acc = 0.f;
    for (int s = 0; s < count; ++s)
      acc += part_acc[(first + s) * p.value_dim + e] * expf(part_ml[(first + s) * 2] - m);
    const size_t at = (size_t)row * p.out_pitch + (size_t)q_head * p.value_dim + e;
    if (p.float_out) reinterpret_cast<float*>(out)[at] = acc * inv;
    else out[at] = srb_from_float<T>(acc * inv);
  }
}

// Shared memory that a block may ask for.  The limit set ahead of a launch is the kernel's and not the launch's, so it is the same number
// in every call: another thread's call of another size does not lower it in between.
#define ATTN_SHARED_MOST (227 * 1024 - KEY_BLOCK * 8)    // beside the keys' rows
#define ATTN_SHARED_TWO_BLOCKS (113 * 1024)

static thread_local int attention_launches = 0;          // kernels that this thread's last call launched

template <typename T, int DIM_PER_LANE>
static int launch_attention(const void* q, const void* k_pool, const void* v_pool, void* out, float* part_acc,
                            float* part_ml, const AttnParams& p, int rows, cudaStream_t s) {
  auto bytes = [&p](int extra, int tiles) {
    return (tiles * ((size_t)KEY_BLOCK * (p.head_dim + extra) + (p.shared_values ? 0 : (size_t)KEY_BLOCK * p.value_dim)) +
            (size_t)p.heads_per_block * p.head_dim) * sizeof(float);
  };
  // rows of whole groups of four elements on four elements' borders (each half of a key row of two maps too)
  const size_t group = 4 * sizeof(T);
  const bool wide = p.head_dim % (p.maps == 2 ? 8 : 4) == 0 && p.value_dim % 4 == 0 &&
                    ((uintptr_t)k_pool | (uintptr_t)v_pool) % group == 0 && bytes(4, 1) <= ATTN_SHARED_MOST;
  // two tiles in flight while a second block still fits beside this one (values up to some 200 entries wide; those of
  // more than 512, with which two tiles take at least 131 KB, never)
  constexpr bool MAY_ASYNC = sizeof(T) == 4 && DIM_PER_LANE <= 16;
  const bool async = MAY_ASYNC && wide && bytes(4, 2) <= ATTN_SHARED_TWO_BLOCKS;
  if constexpr (MAY_ASYNC) {
    // rows of prompts, up to four query heads per kv head: two rows a block and more
    const int groups = p.n_q / p.n_kv;
    const size_t shared = bytes(4, 2) + (size_t)(ROW_WARPS - p.heads_per_block) * p.head_dim * sizeof(float);
    if (async && p.split_size == 0 && p.maps == 1 && p.keep_first == 0 && groups <= ROW_WARPS / 2 && p.n_kv <= 65535 && shared <= ATTN_SHARED_TWO_BLOCKS) {
      auto rows_kernel = paged_attention_rows_kernel<DIM_PER_LANE>;
      if (shared > 48 * 1024)
        SRB_CUDA_CALL(cudaFuncSetAttribute(rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATTN_SHARED_TWO_BLOCKS));
      const int per_block = ROW_WARPS / groups;
      rows_kernel<<<dim3((rows + per_block - 1) / per_block, p.n_kv), ROW_WARPS * 32, shared, s>>>(
          (const float*)q, (const float*)k_pool, (const float*)v_pool, (float*)out, rows, p);
      SRB_LAUNCH_CHECK("paged_attention rows");
      ++attention_launches;
      return SRB_OK;
    }
  }
  bool side_by_side = false;
  if constexpr (MAY_ASYNC) {
    // splits of four tiles whose keys and values fit a block together
    const int groups = p.n_q / p.n_kv;
    const size_t shared = bytes(4, SPLIT_TILES);
    side_by_side = wide && p.split_size == SPLIT_TILES * KEY_BLOCK && p.maps == 1 && p.keep_first == 0 && groups <= SPLIT_MAX_HEADS &&
                   p.n_kv <= 65535 && shared <= ATTN_SHARED_MOST - 1024;
    if (side_by_side) {
      // more blocks than are resident at once
      const long long resident = (long long)srb_sm_count() * (228 * 1024 / (shared + 1024));
      const bool in_turns = !p.shared_values && (long long)p.max_splits * p.n_kv * rows > resident;
      const size_t most = !in_turns ? shared
                                    : (SPLIT_TILES * KEY_BLOCK * (size_t)std::max(p.head_dim + 4, p.value_dim) + (size_t)groups * p.head_dim) * sizeof(float);
      auto split_kernel = in_turns ? paged_attention_split_kernel<DIM_PER_LANE, true> : paged_attention_split_kernel<DIM_PER_LANE, false>;
      SRB_CUDA_CALL(cudaFuncSetAttribute(split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATTN_SHARED_MOST - 1024));
      SRB_CUDA_CALL(srb_launch(split_kernel, dim3(p.max_splits, p.n_kv, rows), dim3(32 * SPLIT_TILES * groups), most, s, (const float*)q,
                               (const float*)k_pool, (const float*)v_pool, (float*)out, part_acc, part_ml, p));
      ++attention_launches;
      if (p.max_splits == 1) return SRB_OK;
    }
  }
  const size_t smem = bytes(wide ? 4 : 1, async ? 2 : 1);
  if (smem > ATTN_SHARED_MOST) SRB_FAIL("paged_attention: %zu bytes of shared memory exceed %d", smem, ATTN_SHARED_MOST);
  auto kernel = async ? paged_attention_kernel<T, DIM_PER_LANE, MAY_ASYNC ? ATTN_ASYNC : ATTN_WIDE>
                      : wide ? paged_attention_kernel<T, DIM_PER_LANE, ATTN_WIDE> : paged_attention_kernel<T, DIM_PER_LANE, ATTN_NARROW>;
  if (smem > 48 * 1024)
    SRB_CUDA_CALL(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, async ? ATTN_SHARED_TWO_BLOCKS : ATTN_SHARED_MOST));
  dim3 grid(p.split_size == 0 ? 1 : p.max_splits, p.n_kv * p.head_chunks, rows);
  if (grid.y > 65535) SRB_FAIL("paged_attention: %d blocks along the heads exceed 65535", (int)grid.y);
  // at least four warps bring the rows, whatever the number of heads that share them
  if (!side_by_side) {
    kernel<<<grid, (p.heads_per_block < 4 ? 4 : p.heads_per_block) * 32, smem, s>>>(
        (const T*)q, (const T*)k_pool, (const T*)v_pool, (T*)out, part_acc, part_ml, p);
    SRB_LAUNCH_CHECK("paged_attention");
    ++attention_launches;
  }
  if (p.split_size != 0) {
    dim3 cgrid(rows, p.n_q);
    SRB_CUDA_CALL(srb_launch(attention_combine_kernel<T>, cgrid, dim3(64), 0, s, (const float*)part_acc, (const float*)part_ml, (T*)out, p));
    SRB_LAUNCH_CHECK("attention_combine");
    ++attention_launches;
  }
  return SRB_OK;
}

// Checks the sizes and launches; shared by every entry point.  Scratch (only when split_size > 0):
// part_acc holds rows * n_q * max_splits * value_dim floats and part_ml rows * n_q * max_splits * 2.
// `sinks` null: no sink.  `value_dim` 0: as wide as the keys.  `v_pool` null: the values are the first
// value_dim entries of the key rows.
// `chunk` > 0: a row sees only keys of its own chunk of positions (see AttnParams).
static int paged_attention_dispatch_masked(const void* q, const void* k_pool, const void* v_pool, void* out,
                                           float* part_acc, float* part_ml, const int* positions,
                                           const int* row_request, const int* block_table, int table_stride, int rows,
                                           int n_q, int n_kv, int head_dim, int page_size, int num_pages, int window,
                                           int chunk, int split_size, int max_splits, float scale, int* error_word,
                                           int dtype, const float* sinks, int value_dim, void* stream,
                                           const float* gates = nullptr, long long out_pitch = 0, float out_scale = 1.0f,
                                           const AttnTerms* terms = nullptr, bool steady_arrays = false) {
  attention_launches = 0;
  if (rows <= 0) return SRB_OK;
  if (chunk < 0) SRB_FAIL("paged_attention: the chunk size must be non-negative");
  if (n_q <= 0 || n_kv <= 0 || n_q % n_kv != 0)
    SRB_FAIL("paged_attention: %d query heads are not a multiple of %d kv heads", n_q, n_kv);
  if (head_dim <= 0) SRB_FAIL("paged_attention: head_dim %d must be positive", head_dim);
  if (value_dim == 0) value_dim = head_dim;
  if (value_dim < 0 || value_dim > 1024 || (!v_pool && value_dim > head_dim))
    SRB_FAIL("paged_attention: values of %d entries must be positive, at most 1024 and, if they are the head of the key "
             "rows (%d entries), no wider than those", value_dim, head_dim);
  if (page_size <= 0 || num_pages <= 0 || table_stride <= 0)
    SRB_FAIL("paged_attention: page size, page count and table stride must be positive");
  if (window < 0 || split_size < 0) SRB_FAIL("paged_attention: window and split size must be non-negative");
  if (split_size != 0 && (max_splits <= 0 || !part_acc || !part_ml))
    SRB_FAIL("paged_attention: a split run needs scratch memory and max_splits > 0");
  if (rows > 65535) {
    // grid.z is limited to 65535 blocks
    SRB_FAIL("paged_attention: %d rows exceed 65535 in one launch", rows);
  }
  AttnParams p;
  p.positions = positions; p.row_request = row_request; p.block_table = block_table;
  p.table_stride = table_stride; p.n_q = n_q; p.n_kv = n_kv; p.head_dim = head_dim;
  p.page_size = page_size; p.num_pages = num_pages; p.window = window; p.chunk = chunk; p.split_size = split_size;
  p.max_splits = split_size == 0 ? 1 : max_splits; p.scale = scale; p.error_word = error_word;
  p.sinks = sinks; p.value_dim = value_dim; p.shared_values = v_pool == nullptr; p.gates = gates;
  p.out_pitch = out_pitch ? out_pitch : (long long)n_q * value_dim; p.out_scale = out_scale;
  p.steady_arrays = steady_arrays;
  if (p.out_pitch < (long long)n_q * value_dim) SRB_FAIL("paged_attention: rows of the output overlap");
  if (const char* fault = srb_apply_terms(p, terms)) SRB_FAIL("paged_attention: %s", fault);
  if (p.maps == 2 && !p.float_out) SRB_FAIL("paged_attention: the results of two maps are floats that srb_map_combine joins");
  const int groups = n_q / n_kv;
  const int most = value_dim > 512 ? ATTN_WIDE_VALUE_WARPS : 32;       // heads, a warp each, that a block may have
  p.head_chunks = (groups + most - 1) / most;
  p.heads_per_block = (groups + p.head_chunks - 1) / p.head_chunks;
  cudaStream_t s = (cudaStream_t)stream;
  const int per_lane = (value_dim + 31) / 32;
#define SRB_ATTN_CASE(T, N) \
  return launch_attention<T, N>(q, k_pool, v_pool, out, part_acc, part_ml, p, rows, s)
#define SRB_ATTN_DISPATCH(T)                        \
  if (per_lane <= 1) { SRB_ATTN_CASE(T, 1); }       \
  else if (per_lane <= 2) { SRB_ATTN_CASE(T, 2); }  \
  else if (per_lane <= 4) { SRB_ATTN_CASE(T, 4); }  \
  else if (per_lane <= 8) { SRB_ATTN_CASE(T, 8); }  \
  else if (per_lane <= 16) { SRB_ATTN_CASE(T, 16); } \
  else { SRB_ATTN_CASE(T, 32); }
  if (dtype == SRB_DTYPE_F32) { SRB_ATTN_DISPATCH(float) }
  if (dtype == SRB_DTYPE_BF16) { SRB_ATTN_DISPATCH(__nv_bfloat16) }
  SRB_FAIL("paged_attention: unknown dtype %d", dtype);
}

static int paged_attention_dispatch_ex(const void* q, const void* k_pool, const void* v_pool, void* out,
                                       float* part_acc, float* part_ml, const int* positions,
                                       const int* row_request, const int* block_table, int table_stride, int rows,
                                       int n_q, int n_kv, int head_dim, int page_size, int num_pages, int window,
                                       int split_size, int max_splits, float scale, int* error_word, int dtype,
                                       const float* sinks, int value_dim, void* stream) {
  return paged_attention_dispatch_masked(q, k_pool, v_pool, out, part_acc, part_ml, positions, row_request, block_table,
                                         table_stride, rows, n_q, n_kv, head_dim, page_size, num_pages, window, 0,
                                         split_size, max_splits, scale, error_word, dtype, sinks, value_dim, stream);
}

static int paged_attention_dispatch(const void* q, const void* k_pool, const void* v_pool, void* out,
                                   float* part_acc, float* part_ml, const int* positions,
                                   const int* row_request, const int* block_table, int table_stride, int rows,
                                   int n_q, int n_kv, int head_dim, int page_size, int num_pages, int window,
                                   int split_size, int max_splits, float scale, int* error_word, int dtype,
                                   void* stream) {
  if (!v_pool) SRB_FAIL("paged_attention: the value pool is missing");
  return paged_attention_dispatch_ex(q, k_pool, v_pool, out, part_acc, part_ml, positions, row_request, block_table,
                                     table_stride, rows, n_q, n_kv, head_dim, page_size, num_pages, window, split_size,
                                     max_splits, scale, error_word, dtype, nullptr, 0, stream);
}
