// Paged grouped-query attention over the block table, 32-bit arithmetic throughout, one kernel
// for every segment length: a whole prompt, a portion of one, or a single decoded token.
//
//   s_j = (q . K_j) * scale          for keys j <= p and (window == 0 or p - j < window or j < keep_first)
//                                    and (mask_chunk == 0 or floor(j / mask_chunk) == floor(p / mask_chunk))
//   o   = sum_j softmax(s)_j V_j     (layover/model.py:59,90-96; layover/kernels/triton_decode.py:89-119)
//
// where p is the query's absolute position (a chunked mask lets a query see only the keys of its own
// chunk of mask_chunk positions, counted from position 0 of the sequence; `keep_first` keeps the first keys
// of a sequence visible behind a window, at their own positions). Three optional generalisations, each off with a null
// pointer or an equal size: values of another size than keys (`vdim`, out is [T, q_heads * vdim]);
// a learned sink per query head, a score without key or value that only enlarges the softmax's
// denominator, o = sum_j exp(s_j) V_j / (exp(sink_h) + sum_j exp(s_j)); and a gate per (token,
// head), a 32-bit factor on the head's output. Two more: a soft cap, s_j <- cap * tanh(s_j / cap), and a factor
// `out_scale` on every output. Keys are walked in tiles of 32 aligned to absolute
// positions (tile i holds keys [32 i, 32 i + 32)), four tiles are a chunk. Within a chunk each score is a dot product
// of four interleaved chains and the running maximum / sum / output follow the same recurrence for every row, starting
// anew with the chunk; then the chunks' results are merged in their order. So a row's result does not depend on how the
// tokens were cut into steps, on which other rows share its block, or on how many blocks share its keys.
// Keys outside [first needed key, context length) are never used: their scores are replaced,
// not multiplied, and their values are read as zero, so stale or non-finite contents of a page
// cannot leak.
//
// Work is a list of tiles made on the host: tile w covers queries [tile_q0[w], +BQ) of sequence
// tile_seq[w]. Query t of sequence s is row cu_q[s] + t of q and out, at absolute position ctx_len[s] - q_len(s) + t. A
// row is one query of one query head; the rows of a tile that share a key/value head share every load of its keys and
// values: a block takes 4 R of them (R a warp, `rows_per_warp`), and with few blocks (a decode step) the chunks of a row are dealt to
// `splits` blocks, which leave each chunk's maximum, sum and output in scratch memory for a second kernel to merge.
// What bounds it: a decode step the latency of a tile (scores, softmax, output: about a thousand cycles for its 32 KB), which
// more blocks hide; a prompt the reads of shared memory, one of 16 bytes per 4 R fused multiply-adds.
// Measured (one B200, 32 query heads of 128 over 8, per layer): four decoding requests of 900 keys 386 -> 24.5 us and 3.6 for the
// merge, a prompt of 261 tokens 205 -> 114 and 18 us (against a block per 16 queries of one head, a chain per score).
#include <math.h>

#include "common.cuh"

namespace {
constexpr int BQ = 16;      // queries per tile
constexpr int BKEYS = 32;   // keys per tile (one per lane)
constexpr int CHUNK_TILES = 4;
constexpr int WARPS = 4;
constexpr int MAX_DIM = 640, MAX_QUADS = MAX_DIM / 128;      // value sizes up to 128 keep one quad of the output a lane, the largest five

// four neighbouring elements with one load (the head size is a multiple of 4 and rows are 16-byte aligned)
template <typename T> struct Quad;
template <> struct Quad<float> {
  static __device__ __forceinline__ float4 load(const float* p) { return *reinterpret_cast<const float4*>(p); }
};
template <> struct Quad<bf16> {
  static __device__ __forceinline__ float4 load(const bf16* p) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&r.x), b = *reinterpret_cast<const __nv_bfloat162*>(&r.y);
    return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
  }
};
// a key's or value's row of `size` channels (a lane four of every 128) into shared memory, or zeros: asynchronously where no
// conversion is needed, else with all its loads on their way before the first is stored
template <int QUADS>
__device__ __forceinline__ void fetch_row(float* dst, const float* src, int size, bool valid, int lane) {
#pragma unroll
  for (int n = 0; n < QUADS; ++n) {
    const int c = 4 * (lane + 32 * n);
    if (c >= size) break;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + c)), "l"(src + c),
                 "r"(valid ? 16 : 0) : "memory");
  }
}
template <int QUADS>
__device__ __forceinline__ void load_row(uint2 (&row)[QUADS], const bf16* src, int size, bool valid, int lane) {
#pragma unroll
  for (int n = 0; n < QUADS; ++n) {
    const int c = 4 * (lane + 32 * n);
    row[n] = valid && c < size ? *reinterpret_cast<const uint2*>(src + c) : make_uint2(0, 0);
  }
}
template <int QUADS>
__device__ __forceinline__ void widen_row(float* dst, const uint2 (&row)[QUADS], int size, int lane) {
#pragma unroll
  for (int n = 0; n < QUADS; ++n) {
    const int c = 4 * (lane + 32 * n);
    if (c < size)
      *reinterpret_cast<float4*>(dst + c) = make_float4(__uint_as_float(row[n].x << 16), __uint_as_float(row[n].x & 0xffff0000u),
                                                        __uint_as_float(row[n].y << 16), __uint_as_float(row[n].y & 0xffff0000u));
  }
}

template <typename T> struct Attention {
  const T *q, *k_pool, *v_pool;
  T* out;
  const int *block_table, *cu_q, *ctx_len, *tile_seq, *tile_q0;
  const float *sinks, *gates;
  float* partials;            // [item][row of the item][chunk][2 + vdim]; null: a block walks all of its rows' chunks
  int chunk_room;             // chunks there is room for: all that a block table can hold
  int table_width, q_heads, kv_heads, dim, key_pitch, vdim, page_tokens, window, mask_chunk, keep_first, row_groups, stages;
  bool q_quads;               // q's rows begin where four elements can be read at once
  float scale, cap, out_scale;
  long out_stride;
};

// What a block works on: rows first_row .. of a tile (row = query * group + query head of the group).
struct Item {
  int seq, row0, start, n_rows, group, kv_head, first_row;      // row0: the tile's first query in q; start: its position
  template <typename T, int ROWS> static __device__ __forceinline__ Item at(const Attention<T>& a) {
    Item item;
    item.seq = a.tile_seq[blockIdx.x];
    const int q0 = a.tile_q0[blockIdx.x], begin = a.cu_q[item.seq], q_len = a.cu_q[item.seq + 1] - begin;
    item.group = a.q_heads / a.kv_heads;
    item.row0 = begin + q0;
    item.start = a.ctx_len[item.seq] - q_len + q0;
    item.n_rows = min(BQ, q_len - q0) * item.group;
    item.kv_head = blockIdx.y / a.row_groups;
    item.first_row = blockIdx.y % a.row_groups * ROWS;
    return item;
  }
  __device__ __forceinline__ int position(int row) const { return start + row / group; }
};

// One chunk's result joins those of the chunks before it; explicit roundings, the same bits wherever it happens.
__device__ __forceinline__ float merge_scale(float& m, float& l, float chunk_m, float chunk_l, float& chunk_scale) {
  const float top = fmaxf(m, chunk_m), keep = m == -INFINITY ? 0.f : expf(m - top);
  chunk_scale = expf(chunk_m - top);
  l = fmaf(chunk_l, chunk_scale, __fmul_rn(l, keep));
  m = top;
  return keep;
}
__device__ __forceinline__ void merge_quad(float4& total, const float4& chunk, float keep, float chunk_scale) {
  total.x = fmaf(chunk.x, chunk_scale, __fmul_rn(total.x, keep));
  total.y = fmaf(chunk.y, chunk_scale, __fmul_rn(total.y, keep));
  total.z = fmaf(chunk.z, chunk_scale, __fmul_rn(total.z, keep));
  total.w = fmaf(chunk.w, chunk_scale, __fmul_rn(total.w, keep));
}

template <typename T, int NV>
__device__ __forceinline__ void store_row(const Attention<T>& a, const Item& item, int row, float m, float l, const float4 (&total)[NV], int lane) {
  const int token = item.row0 + row / item.group, head = item.kv_head * item.group + row % item.group;
  float denominator = l, keep = 1.f;
  if (a.sinks) {                                   // the sink joins the denominator only; m is finite (a row sees itself)
    const float sink = a.sinks[head], top = fmaxf(m, sink);
    keep = expf(m - top);
    denominator = l * keep + expf(sink - top);
  }
  const float gate = a.gates ? a.gates[(size_t)token * a.q_heads + head] : 1.f;
  T* o = a.out + (size_t)token * a.out_stride + head * a.vdim;
#pragma unroll
  for (int n = 0; n < NV; ++n) {
    const int d = 4 * (lane + 32 * n);
    if (d >= a.vdim) continue;
    const float v[4] = {total[n].x, total[n].y, total[n].z, total[n].w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float value = a.sinks ? v[e] * keep / denominator : v[e] / l;
      if (a.gates) value *= gate;
      value *= a.out_scale;
      Elem<T>::store(o + d + e, value);
    }
  }
}

// NV: quads of a value that a lane accumulates. Row i of a warp is row 4 i + warp of the block's, so that few rows spread
// over the warps.
template <typename T, int NV, int R>
__global__ void __launch_bounds__(WARPS * 32)
attention_rows_kernel(const Attention<T> a) {
  extern __shared__ __align__(16) float smem[];
  constexpr int ROWS = WARPS * R;
  pdl_launch_dependents();
  pdl_wait();
  const Item item = Item::at<T, ROWS>(a);
  if (item.first_row >= item.n_rows) return;
  const int dim = a.dim, vdim = a.vdim, pitch = a.key_pitch;
  float* q_s = smem;                                             // [ROWS][dim]
  float* p_s = q_s + ROWS * dim;                                 // [WARPS][R][BKEYS]
  float* k_s = p_s + ROWS * BKEYS;                               // [stages][BKEYS][pitch]
  float* v_s = k_s + a.stages * BKEYS * pitch;                   // [stages][BKEYS][vdim]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = min(ROWS, item.n_rows - item.first_row);      // live rows of the block
  const int mine = rows > warp ? (rows - warp + WARPS - 1) / WARPS : 0;       // and of the warp
  const int* table = a.block_table + (size_t)item.seq * a.table_width;

  for (int r = warp; r < rows; r += WARPS) {
    const int row = item.first_row + r;
    const T* src = a.q + ((size_t)(item.row0 + row / item.group) * a.q_heads + item.kv_head * item.group + row % item.group) * dim;
    if (a.q_quads) {
      for (int c = 4 * lane; c < dim; c += 128) *reinterpret_cast<float4*>(q_s + r * dim + c) = Quad<T>::load(src + c);
    } else {
      for (int c = lane; c < dim; c += 32) q_s[r * dim + c] = Elem<T>::load(src + c);
    }
  }
  const int p_first = item.position(item.first_row), p_last = item.position(item.first_row + rows - 1);
  int key_lo = a.window > 0 ? max(0, p_first - a.window + 1) : 0;            // first key any row here may see
  if (a.mask_chunk > 0) key_lo = max(key_lo, p_first / a.mask_chunk * a.mask_chunk);
  const int tile_lo = key_lo / BKEYS, tile_hi = p_last / BKEYS;
  // the tiles of the kept first keys come first, then the window's; tiles between the two are skipped
  const int kept_keys = a.window > 0 ? min(a.keep_first, key_lo) : 0;        // kept keys that lie before the window
  const int kept_tiles = min((kept_keys + BKEYS - 1) / BKEYS, tile_lo);
  const int chunks = tile_hi / CHUNK_TILES + 1, per_block = (chunks + gridDim.z - 1) / gridDim.z;
  const int chunk_begin = blockIdx.z * per_block, chunk_end = min(chunks, chunk_begin + per_block);
  if (chunk_begin >= chunk_end) return;
  const int tile_end = min(tile_hi + 1, chunk_end * CHUNK_TILES);
  auto seen_tile = [&](int tile) { return tile >= kept_tiles && tile < tile_lo ? tile_lo : tile; };
  float* left = nullptr;                                         // where the warp's rows leave their chunks' results
  if (a.partials) {
    left = a.partials + ((size_t)(blockIdx.x * gridDim.y + blockIdx.y) * ROWS + warp) * a.chunk_room * (vdim + 2);
    if (lane == 0)
      for (int r = 0; r < mine; ++r)
        for (int c = chunk_begin; c < chunk_end; ++c) left[((size_t)r * WARPS * a.chunk_room + c) * (vdim + 2)] = -INFINITY;
  }

  auto fetch = [&](int tile, int stage) {
    // the pages of the warp's keys in one load, a lane each: a copy that waits for its own page every time takes as many trips
    // to memory as the warp has keys
    constexpr int EACH = BKEYS / WARPS;
    const int my_key = tile * BKEYS + warp + (lane % EACH) * WARPS;
    const bool my_valid = (my_key >= key_lo || my_key < kept_keys) && my_key <= p_last;
    const int my_page = my_valid ? table[my_key / a.page_tokens] : -1;
#pragma unroll 2
    for (int i = 0; i < EACH; ++i) {
      const int j = warp + i * WARPS, key = tile * BKEYS + j, page = __shfl_sync(0xffffffffu, my_page, i);
      const bool valid = page >= 0;
      const size_t at = valid ? ((size_t)page * a.kv_heads + item.kv_head) * a.page_tokens + key % a.page_tokens : 0;
      const T *k_from = a.k_pool + at * dim, *v_from = a.v_pool + at * vdim;
      float *k_to = k_s + (stage * BKEYS + j) * pitch, *v_to = v_s + (stage * BKEYS + j) * vdim;
      if constexpr (sizeof(T) == 4) {
        fetch_row<MAX_QUADS>(k_to, k_from, dim, valid, lane);
        fetch_row<MAX_QUADS>(v_to, v_from, vdim, valid, lane);
      } else {
        uint2 k_row[MAX_QUADS], v_row[NV];
        load_row(k_row, k_from, dim, valid, lane);
        load_row(v_row, v_from, vdim, valid, lane);
        widen_row(k_to, k_row, dim, lane);
        widen_row(v_to, v_row, vdim, lane);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float m[R], l[R], total_m[R], total_l[R];
  float4 acc[R][NV], total[R][NV];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    m[r] = total_m[r] = -INFINITY;
    l[r] = total_l[r] = 0.f;
#pragma unroll
    for (int n = 0; n < NV; ++n) acc[r][n] = total[r][n] = make_float4(0.f, 0.f, 0.f, 0.f);
  }

  int tile = seen_tile(chunk_begin * CHUNK_TILES), stage = 0;
  if (tile < tile_end) fetch(tile, 0);
  while (tile < tile_end) {
    const int next = seen_tile(tile + 1);
    if (a.stages > 1 && next < tile_end) {
      fetch(next, stage ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();                                             // the tile (and q_s) is complete
    const float* k_row = k_s + (stage * BKEYS + lane) * pitch;
    float4 s4[R];
#pragma unroll
    for (int r = 0; r < R; ++r) s4[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
    for (int c = 0; c < dim; c += 4) {
      const float4 k = *reinterpret_cast<const float4*>(k_row + c);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (R > 1 && r >= mine) break;
        const float4 qv = *reinterpret_cast<const float4*>(q_s + (WARPS * r + warp) * dim + c);
        s4[r].x = fmaf(qv.x, k.x, s4[r].x);
        s4[r].y = fmaf(qv.y, k.y, s4[r].y);
        s4[r].z = fmaf(qv.z, k.z, s4[r].z);
        s4[r].w = fmaf(qv.w, k.w, s4[r].w);
      }
    }
    const int key = tile * BKEYS + lane;
    float* p_row = p_s + warp * R * BKEYS;
    unsigned active = 0;                                         // rows that see something of this tile
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (r >= mine) break;                                      // uniform over the warp
      const int p = item.position(item.first_row + WARPS * r + warp);
      const bool seen = key <= p && (a.window <= 0 || p - key < a.window || key < a.keep_first) &&
                        (a.mask_chunk <= 0 || key >= p / a.mask_chunk * a.mask_chunk);
      float s = __fadd_rn(__fadd_rn(s4[r].x, s4[r].y), __fadd_rn(s4[r].z, s4[r].w));
      s = __fmul_rn(s, a.scale);
      if (a.cap > 0.f) s = a.cap * tanhf(s / a.cap);
      s = seen ? s : -INFINITY;
      const float tile_max = warp_max(s);
      if (tile_max == -INFINITY) continue;
      active |= 1u << r;
      const float top = fmaxf(m[r], tile_max), prob = seen ? expf(s - top) : 0.f;
      const float alpha = m[r] == -INFINITY ? 0.f : expf(m[r] - top);
      l[r] = __fadd_rn(__fmul_rn(l[r], alpha), warp_sum(prob));
      m[r] = top;
      p_row[r * BKEYS + lane] = prob;
#pragma unroll
      for (int n = 0; n < NV; ++n) {
        acc[r][n].x *= alpha; acc[r][n].y *= alpha; acc[r][n].z *= alpha; acc[r][n].w *= alpha;
      }
    }
    __syncwarp();
#pragma unroll 2
    for (int j = 0; j < BKEYS; j += 4) {
      float4 p4[R];
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (active >> r & 1) p4[r] = *reinterpret_cast<const float4*>(p_row + r * BKEYS + j);
#pragma unroll
      for (int n = 0; n < NV; ++n) {
        const int d = 4 * (lane + 32 * n);
        if (d >= vdim) break;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float4 v = *reinterpret_cast<const float4*>(v_s + (stage * BKEYS + j + e) * vdim + d);
#pragma unroll
          for (int r = 0; r < R; ++r) {
            if (!(active >> r & 1)) continue;
            const float p = e == 0 ? p4[r].x : e == 1 ? p4[r].y : e == 2 ? p4[r].z : p4[r].w;
            acc[r][n].x = fmaf(p, v.x, acc[r][n].x);
            acc[r][n].y = fmaf(p, v.y, acc[r][n].y);
            acc[r][n].z = fmaf(p, v.z, acc[r][n].z);
            acc[r][n].w = fmaf(p, v.w, acc[r][n].w);
          }
        }
      }
    }
    if (next >= tile_end || next / CHUNK_TILES != tile / CHUNK_TILES) {        // the chunk is done
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (r >= mine) break;
        if (m[r] == -INFINITY) continue;                         // nothing of it is seen by this row
        if (left) {
          float* at = left + ((size_t)r * WARPS * a.chunk_room + tile / CHUNK_TILES) * (vdim + 2);
          if (lane == 0) { at[0] = m[r]; at[1] = l[r]; }
#pragma unroll
          for (int n = 0; n < NV; ++n) {
            const int d = 4 * (lane + 32 * n);
            if (d < vdim) {
              reinterpret_cast<float2*>(at + 2 + d)[0] = make_float2(acc[r][n].x, acc[r][n].y);
              reinterpret_cast<float2*>(at + 2 + d)[1] = make_float2(acc[r][n].z, acc[r][n].w);
            }
          }
        } else {
          float chunk_scale;
          const float keep = merge_scale(total_m[r], total_l[r], m[r], l[r], chunk_scale);
#pragma unroll
          for (int n = 0; n < NV; ++n) merge_quad(total[r][n], acc[r][n], keep, chunk_scale);
        }
        m[r] = -INFINITY;
        l[r] = 0.f;
#pragma unroll
        for (int n = 0; n < NV; ++n) acc[r][n] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    __syncthreads();                                             // the tile is read
    if (a.stages == 1 && next < tile_end) fetch(next, 0);
    if (a.stages > 1) stage ^= 1;
    tile = next;
  }
  if (!left) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (r < mine) store_row<T, NV>(a, item, item.first_row + WARPS * r + warp, total_m[r], total_l[r], total[r], lane);
  }
}

// Merges the chunks' results of every row in their order: a warp per row, four chunks' loads on their way at once.
template <typename T, int NV, int R>
__global__ void __launch_bounds__(WARPS * 32)
merge_chunks_kernel(const Attention<T> a) {
  constexpr int ROWS = WARPS * R;
  pdl_launch_dependents();
  pdl_wait();
  const Item item = Item::at<T, ROWS>(a);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rows = min(ROWS, item.n_rows - item.first_row);
  if (rows <= 0) return;
  const int chunks = item.position(item.first_row + rows - 1) / BKEYS / CHUNK_TILES + 1;
  for (int row = warp; row < rows; row += WARPS) {
    const float* left = a.partials + ((size_t)(blockIdx.x * gridDim.y + blockIdx.y) * ROWS + row) * a.chunk_room * (a.vdim + 2);
    float m = -INFINITY, l = 0.f;
    float4 total[NV];
#pragma unroll
    for (int n = 0; n < NV; ++n) total[n] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c0 = 0; c0 < chunks; c0 += 4) {
      float2 ml[4];
      float4 part[4][NV];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float* at = left + (size_t)(c0 + c) * (a.vdim + 2);
        ml[c] = c0 + c < chunks ? make_float2(at[0], at[1]) : make_float2(-INFINITY, 0.f);
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          const int d = 4 * (lane + 32 * n);
          part[c][n] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (c0 + c < chunks && d < a.vdim) {
            const float2 lo = reinterpret_cast<const float2*>(at + 2 + d)[0], hi = reinterpret_cast<const float2*>(at + 2 + d)[1];
            part[c][n] = make_float4(lo.x, lo.y, hi.x, hi.y);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (ml[c].x == -INFINITY) continue;
        float chunk_scale;
        const float keep = merge_scale(m, l, ml[c].x, ml[c].y, chunk_scale);
#pragma unroll
        for (int n = 0; n < NV; ++n) merge_quad(total[n], part[c][n], keep, chunk_scale);
      }
    }
    store_row<T, NV>(a, item, item.first_row + row, m, l, total, lane);
  }
}

size_t block_smem(int rows, int stages, int dim, int key_pitch, int vdim) {
  return (size_t)(rows * (dim + BKEYS) + stages * BKEYS * (key_pitch + vdim)) * sizeof(float);
}
// rows of a key tile: a pitch of 4 floats beyond a multiple of 32 keeps the 16-byte reads of 32 keys free of bank conflicts
int pitch_of(int dim) { return dim + (36 - dim % 32) % 32; }

template <typename T, int NV, int R>
int launch_rows(Attention<T> a, int n_tiles, int max_rows, int splits, cudaStream_t stream) {
  constexpr int ROWS = WARPS * R;
  static LbPerDeviceOnce configured;
  auto kernel = attention_rows_kernel<T, NV, R>;
  if (!configured.run(LB_ALLOW_SMEM(kernel, 227 * 1024))) return lb_last_error();
  a.row_groups = (max_rows + ROWS - 1) / ROWS;
  auto smem = [&](int stages) { return block_smem(ROWS, stages, a.dim, a.key_pitch, a.vdim); };
  a.stages = sizeof(T) == 4 && smem(2) <= 227 * 1024 ? 2 : 1;      // a copy that converts is not asynchronous: a second stage waits all the same
  if (smem(a.stages) > 227 * 1024 || (long)a.kv_heads * a.row_groups > 65535) return LB_ERR_SIZE;
  const dim3 grid(n_tiles, a.kv_heads * a.row_groups, a.partials ? splits : 1);
  lb_launch(attention_rows_kernel<T, NV, R>, grid, dim3(WARPS * 32), smem(a.stages), stream, a);
  if (a.partials) lb_launch(merge_chunks_kernel<T, NV, R>, dim3(grid.x, grid.y), dim3(WARPS * 32), 0, stream, a);
  return lb_last_error();
}

// Rows of a warp: several, as far as registers go, share every read of a key or value; but one where the launch's rows, one a
// warp, and their chunks of keys find room on the SMs at once, where a tile takes a warp as long as it has rows. Results do not depend
// on it. Measured (one B200, 32-bit, us with one and with four rows a warp): 32 heads over 8, a prompt of 20 tokens 7.4 and 13.2, of 261
// 133 and 104, 64 decoding requests of 1,500 keys of 32 heads over 1 437 and 254, one of 900 21 and 44. Eight rows a warp were slower
// than four nearly everywhere (the prompt of 261: 127).
int rows_per_warp(int max_rows, int dim, int vdim, long blocks_of_tiles, int chunks, int sm_count) {
  if (max_rows <= WARPS) return 1;
  const size_t smem = block_smem(WARPS, 2, dim, pitch_of(dim), vdim);
  const long resident = smem > 0 ? (long)(227 * 1024 / smem) : 1, room = sm_count * (resident < 1 ? 1 : (resident > 3 ? 3 : resident));
  const long blocks = blocks_of_tiles * ((max_rows + WARPS - 1) / WARPS);
  if (blocks * (chunks > 1 ? chunks : 1) <= room) return 1;
  return vdim <= 256 ? 4 : 2;
}

template <typename T>
int launch_attention(const Attention<T>& a, int n_tiles, int max_rows, int rows, int splits, cudaStream_t stream) {
  if (rows == 1) {
    if (a.vdim <= 128) return launch_rows<T, 1, 1>(a, n_tiles, max_rows, splits, stream);
    return a.vdim <= 256 ? launch_rows<T, 2, 1>(a, n_tiles, max_rows, splits, stream) : launch_rows<T, 5, 1>(a, n_tiles, max_rows, splits, stream);
  }
  if (a.vdim <= 128) return launch_rows<T, 1, 4>(a, n_tiles, max_rows, splits, stream);
  return a.vdim <= 256 ? launch_rows<T, 2, 4>(a, n_tiles, max_rows, splits, stream) : launch_rows<T, 5, 2>(a, n_tiles, max_rows, splits, stream);
}
}  // namespace

LB_EXPORT int lb_attention_simt_block_queries() { return BQ; }

// Blocks that a launch has without a split, and the rows of each: what a caller needs to size the scratch (blocks * rows *
// chunks a block table can hold * (vdim + 2) floats) and to choose `splits`. `max_chunks`: chunks of the longest context (about;
// 0: unknown).
LB_EXPORT int lb_attention_simt_plan(int n_tiles, int q_heads, int kv_heads, int dim, int vdim, int max_q_len, int max_chunks, int sm_count,
                                     int* rows_of_block) {
  if (kv_heads <= 0 || q_heads % kv_heads || dim <= 0 || dim > MAX_DIM || vdim <= 0 || vdim > MAX_DIM) { *rows_of_block = 0; return 0; }
  const int max_rows = (max_q_len < BQ ? max_q_len : BQ) * (q_heads / kv_heads);
  *rows_of_block = WARPS * rows_per_warp(max_rows, dim, vdim, (long)n_tiles * kv_heads, max_chunks, sm_count);
  return n_tiles * kv_heads * ((max_rows + *rows_of_block - 1) / *rows_of_block);
}
LB_EXPORT int lb_attention_simt_chunk() { return BKEYS * CHUNK_TILES; }

// `max_q_len`: no sequence has more queries in this step (BQ or more: any number). `rows_of_block`: as `lb_attention_simt_plan`
// says for these sizes (any of its values will do). `splits` > 1: the keys of a row are dealt to
// that many blocks, `partials` has the room that `lb_attention_simt_plan` speaks of, `chunk_room` chunks a row.
LB_EXPORT int lb_attention_simt(int dtype, const void* q, const void* k_pool, const void* v_pool, void* out,
                                const int* block_table, int table_width, const int* cu_q, const int* ctx_len,
                                const int* tile_seq, const int* tile_q0, int n_tiles, int q_heads, int kv_heads,
                                int dim, int page_tokens, float scale, int window, int vdim, const float* sinks,
                                const float* gates, int mask_chunk, int keep_first, float softcap, float out_scale,
                                long out_stride, int max_q_len, int rows_of_block, int splits, float* partials, int chunk_room, cudaStream_t stream) {
  if (n_tiles <= 0) return 0;
  if (dim <= 0 || dim > MAX_DIM || dim % 4 || kv_heads <= 0 || q_heads % kv_heads || q_heads > 65535) return LB_ERR_SIZE;
  if (vdim <= 0 || vdim > MAX_DIM || vdim % 4 || keep_first < 0 || (keep_first && mask_chunk)) return LB_ERR_SIZE;
  if (!(softcap >= 0.f) || out_stride < (long)q_heads * vdim || max_q_len < 1 || (splits > 1 && !partials)) return LB_ERR_SIZE;
  const int element = dtype == LB_F32 ? 4 : 2;           // keys and values are read four elements at a time
  if ((uintptr_t)k_pool % (4 * element) || (uintptr_t)v_pool % (4 * element)) return LB_ERR_ALIGN;
  const int max_rows = (max_q_len < BQ ? max_q_len : BQ) * (q_heads / kv_heads);
  const int key_pitch = pitch_of(dim), rows = rows_of_block / WARPS;
  if (rows_of_block % WARPS || (rows != 1 && rows != (vdim <= 256 ? 4 : 2))) return LB_ERR_SIZE;
#define LB_SIMT(T)                                                                                                           \
  do {                                                                                                                       \
    Attention<T> a{(const T*)q, (const T*)k_pool, (const T*)v_pool, (T*)out, block_table, cu_q, ctx_len, tile_seq, tile_q0,   \
                   sinks, gates, splits > 1 ? partials : nullptr, chunk_room, table_width, q_heads, kv_heads, dim, key_pitch, \
                   vdim, page_tokens, window, mask_chunk, keep_first, 0, 0, (uintptr_t)q % (4 * sizeof(T)) == 0, scale, softcap, out_scale,  \
                   out_stride};                                                                                               \
    return launch_attention<T>(a, n_tiles, max_rows, rows, splits, stream);                                                      \
  } while (0)
  if (dtype == LB_F32) LB_SIMT(float);
  if (dtype == LB_BF16) LB_SIMT(bf16);
#undef LB_SIMT
  return LB_ERR_DTYPE;
}
