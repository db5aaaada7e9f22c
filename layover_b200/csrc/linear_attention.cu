// Linear attention with a constant decay per head, as a recurrence over a state of fixed size
// per request, and the gated RMSNorm that follows it.
//
// Per sequence and head, with q_t, k_t of size dim and v_t of size vdim (read from a stacked
// projection row and passed through an activation on the way in):
//
//   S_t = decay_h * S_(t-1) + k_t v_t^T        S is [dim, vdim], 32-bit, kept in the request's state slot
//   o_t = S_t^T q_t                            o_t[e] = sum_d S_t[d, e] q_t[d]
//
// One kernel serves a whole prompt, a portion of one and a single decoded token: a sequence's
// tokens of the step are walked in order from the state the step before left, and the new state
// is written back. Every state element follows the same sequence of operations whatever the cut
// (s = fma(k, v, decay * s); the sum over d is taken in a fixed order), so the result does not
// depend on how the tokens were cut into steps or on what else is in the batch, bit for bit.
// State, decay, products and sums are 32-bit; only q, k, v arrive in the run's type T.
//
// Grid (ceil(vdim / 32), heads, sequences), RANGES warps: warp r owns rows [r * DPT, (r + 1) * DPT) of
// S, lane j column blockIdx.x * 32 + j, so a thread keeps DPT state elements in registers and never
// synchronises inside a token. Tokens are taken CHUNK (8) at a time through two buffers in shared
// memory: while a chunk is computed (k and q are read as 16-byte broadcasts, each warp leaves its
// partial sums of o per token), the next chunk's q, k, v are already on their way from global
// memory into registers; the warps' partial sums are added in warp order at the end of the chunk.
// RANGES and DPT depend on the head size only, never on the batch.
//
// A long portion of one sequence is a long chain for few blocks. Steps that hold one (the host decides from the step's
// longest portion) run in three launches instead: every sequence's portion is cut into segments of `seg_tokens`. `products`:
// what a segment of n tokens does is written as products of matrices, S_in the state that comes in:
//
//   E     = sum_j decay^(n-1-j) k_j v_j^T                                      `segment_state_kernel`
//   S_in of the next segment = decay^n S_in + E, in order, the last one to the slot          `scan_combine_kernel`
//   o_i   = decay^(i+1) S_in^T q_i + sum_(j<=i) decay^(i-j) (q_i . k_j) v_j     `segment_output_kernel`
//
// Else MODE 1 scans every segment at once, a sequence's first segment from the slot's state and the others
// from zero, and leaves each segment's end state in `seg_state`; the combine kernel leaves S_in(s) where segment s finds
// it (in the place of the segment before); MODE 2 adds decay^(t+1) S_in^T q_t. Either way everything is 32-bit on the FFMA
// pipes and the sums are the same numbers in another order: results agree with the single pass within rounding, not bit
// for bit.
#include <math.h>

#include <type_traits>

#include "common.cuh"

namespace {
constexpr int COLS = 32;      // value columns per block (one per lane)
constexpr int CHUNK = 8;      // tokens per trip through shared memory (a thread stages at most one value of v: CHUNK * 32 <= threads)

template <int ACT> __device__ __forceinline__ float activate(float z) {
  return ACT == 1 ? z / (1.0f + __expf(-z)) : z;      // 1: silu, 0: none
}

// decay^n; 1 for n = 0 also where the decay is 0 (its logarithm is -inf)
__device__ __forceinline__ float decay_power(float log2_lam, int n) { return n == 0 ? 1.f : exp2f((float)n * log2_lam); }

// the sequence and the segment of it that global segment `g` is; a sequence has at least one segment
__device__ __forceinline__ void find_segment(const int* __restrict__ cu_q, int n_seqs, int seg_tokens, int g, int& seq,
                                             int& segment, int& first_segment) {
  seq = 0;
  first_segment = 0;
  for (; seq < n_seqs - 1; ++seq) {
    const int len = cu_q[seq + 1] - cu_q[seq], ns = max(1, (len + seg_tokens - 1) / seg_tokens);
    if (g < first_segment + ns) break;
    first_segment += ns;
  }
  segment = g - first_segment;
}

template <typename T, int RANGES, int DPT, int ACT, int MODE = 0>
__global__ void __launch_bounds__(RANGES * COLS)
decay_scan_kernel(const T* __restrict__ proj, long row_stride, int q_off, int k_off, int v_off,
                  float* __restrict__ out, float* __restrict__ state, const int* __restrict__ cu_q,
                  const int* __restrict__ state_slots, const float* __restrict__ decay, int heads, int dim, int vdim,
                  float* __restrict__ seg_state, int seg_tokens, int n_seqs) {
  static_assert(DPT % 4 == 0, "16-byte broadcasts");
  static_assert(CHUNK * COLS <= RANGES * COLS, "one value of v per staging thread");
  constexpr int DPAD = RANGES * DPT, THREADS = RANGES * COLS;
  constexpr int QK_EACH = (CHUNK * DPAD + THREADS - 1) / THREADS;     // q (and k) elements a thread stages per chunk
  extern __shared__ __align__(16) float scan_smem[];
  float (*q_s)[CHUNK][DPAD] = reinterpret_cast<float (*)[CHUNK][DPAD]>(scan_smem);                       // [2][CHUNK][DPAD]
  float (*k_s)[CHUNK][DPAD] = reinterpret_cast<float (*)[CHUNK][DPAD]>(scan_smem + 2 * CHUNK * DPAD);    // [2][CHUNK][DPAD]
  float (*v_s)[CHUNK][COLS] = reinterpret_cast<float (*)[CHUNK][COLS]>(scan_smem + 4 * CHUNK * DPAD);    // [2][CHUNK][COLS]
  float (*part_s)[RANGES][COLS] = reinterpret_cast<float (*)[RANGES][COLS]>(scan_smem + 4 * CHUNK * DPAD + 2 * CHUNK * COLS);
  pdl_launch_dependents();
  pdl_wait();
  const int head = blockIdx.y, e0 = blockIdx.x * COLS;
  const int r = threadIdx.x >> 5, j = threadIdx.x & 31, e = e0 + j;
  int seq = blockIdx.z, segment = 0, first_segment = 0;
  if (MODE != 0) find_segment(cu_q, n_seqs, seg_tokens, blockIdx.z, seq, segment, first_segment);
  if (MODE == 2 && segment == 0) return;          // a first segment started from the true state: nothing to add
  const int first = cu_q[seq] + (MODE != 0 ? segment * seg_tokens : 0);
  const int count = MODE != 0 ? min(seg_tokens, cu_q[seq + 1] - first) : cu_q[seq + 1] - first;
  const float lam = decay[head];
  const float log2_lam = log2f(lam);                // -inf for a decay of 0: exp2f gives 0
  // MODE 0: from and to the slot; 1: a first segment from the slot, the others from zero, the end to seg_state;
  // 2: the state that came into this segment (left by the combine kernel in the segment before's place), frozen
  float* mine = state + ((size_t)state_slots[seq] * heads + head) * dim * vdim;
  float* kept = MODE != 0 ? seg_state + ((size_t)(blockIdx.z - (MODE == 2 ? 1 : 0)) * heads + head) * dim * vdim : nullptr;
  const float* from = MODE == 2 ? kept : ((MODE == 1 && segment > 0) ? nullptr : mine);
  float s[DPT];
#pragma unroll
  for (int x = 0; x < DPT; ++x) {
    const int d = r * DPT + x;
    s[x] = (from && d < dim && e < vdim) ? from[(size_t)d * vdim + e] : 0.f;
  }
  // what this thread fetches of a chunk: QK_EACH elements of q and of k, and (the first CHUNK * 32 threads) one of v
  float q_reg[QK_EACH], k_reg[QK_EACH], v_reg = 0.f;
  auto fetch = [&](int t0, int n) {
#pragma unroll
    for (int u = 0; u < QK_EACH; ++u) {
      const int i = threadIdx.x + u * THREADS, t = i / DPAD, d = i - t * DPAD;
      q_reg[u] = k_reg[u] = 0.f;
      if (t < n && d < dim) {
        const T* row = proj + (size_t)(first + t0 + t) * row_stride + head * dim + d;
        q_reg[u] = Elem<T>::load(row + q_off);
        if (MODE != 2) k_reg[u] = Elem<T>::load(row + k_off);
      }
    }
    if (MODE != 2 && threadIdx.x < CHUNK * COLS) {
      const int t = threadIdx.x / COLS, c = threadIdx.x - t * COLS;
      v_reg = (t < n && e0 + c < vdim)
                  ? Elem<T>::load(proj + (size_t)(first + t0 + t) * row_stride + v_off + head * vdim + e0 + c) : 0.f;
    }
  };
  auto stage = [&](int buf) {
#pragma unroll
    for (int u = 0; u < QK_EACH; ++u) {
      const int i = threadIdx.x + u * THREADS, t = i / DPAD, d = i - t * DPAD;
      if (t < CHUNK) {
        q_s[buf][t][d] = activate<ACT>(q_reg[u]);
        k_s[buf][t][d] = activate<ACT>(k_reg[u]);
      }
    }
    if (threadIdx.x < CHUNK * COLS) v_s[buf][threadIdx.x / COLS][threadIdx.x % COLS] = activate<ACT>(v_reg);
  };
  fetch(0, min(CHUNK, count));
  stage(0);
  __syncthreads();
  int buf = 0;
  for (int t0 = 0; t0 < count; t0 += CHUNK, buf ^= 1) {
    const int n = min(CHUNK, count - t0);
    const bool more = t0 + CHUNK < count;
    if (more) fetch(t0 + CHUNK, min(CHUNK, count - t0 - CHUNK));     // in flight while this chunk is computed
#pragma unroll 2
    for (int t = 0; t < n; ++t) {
      const float v = v_s[buf][t][j];
      const float4* kr = reinterpret_cast<const float4*>(&k_s[buf][t][r * DPT]);
      const float4* qr = reinterpret_cast<const float4*>(&q_s[buf][t][r * DPT]);
      float partial[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int x4 = 0; x4 < DPT / 4; ++x4) {
        const float4 k4 = kr[x4], q4 = qr[x4];
        if (MODE != 2) {
          s[4 * x4 + 0] = fmaf(k4.x, v, lam * s[4 * x4 + 0]);
          s[4 * x4 + 1] = fmaf(k4.y, v, lam * s[4 * x4 + 1]);
          s[4 * x4 + 2] = fmaf(k4.z, v, lam * s[4 * x4 + 2]);
          s[4 * x4 + 3] = fmaf(k4.w, v, lam * s[4 * x4 + 3]);
        }
        partial[0] = fmaf(s[4 * x4 + 0], q4.x, partial[0]);
        partial[1] = fmaf(s[4 * x4 + 1], q4.y, partial[1]);
        partial[2] = fmaf(s[4 * x4 + 2], q4.z, partial[2]);
        partial[3] = fmaf(s[4 * x4 + 3], q4.w, partial[3]);
      }
      part_s[t][r][j] = (partial[0] + partial[1]) + (partial[2] + partial[3]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n * COLS; i += THREADS) {
      const int t = i / COLS, c = i - t * COLS;
      if (e0 + c >= vdim) continue;
      float total = 0.f;
#pragma unroll
      for (int w = 0; w < RANGES; ++w) total += part_s[t][w][c];
      float* at = out + ((size_t)(first + t0 + t) * heads + head) * vdim + e0 + c;
      if (MODE == 2) *at += exp2f((float)(t0 + t + 1) * log2_lam) * total;
      else *at = total;
    }
    if (more) stage(buf ^ 1);
    __syncthreads();      // the partial sums have been read, the next chunk is in place
  }
  if (MODE == 2) return;
  float* to = MODE == 1 ? kept : mine;
#pragma unroll
  for (int x = 0; x < DPT; ++x) {
    const int d = r * DPT + x;
    if (d < dim && e < vdim) to[(size_t)d * vdim + e] = s[x];
  }
}

// Per sequence, head and state element: the segments' end states become the states that come INTO the segments, and the
// state after the last segment goes to the slot. FROM_ZERO: all segments started from zero, and what comes into segment s
// is left in its own place; else the first one started from the slot, and it is left in the place of the segment before.
// WIDTH 4: four elements a thread, where all rows begin on 16 bytes and a head's size is a multiple of 4. What bounds it is the
// memory system, with eight segments' loads on their way at once (one B200, 24 segments of 32 heads of 128 x 128, 100 MB:
// 47 -> 20 us inside a step; one element a thread and four segments before).
// The walk over the segments starts when the joining has ended: its blocks, had they come early, would be placed around the
// joining's and share SMs (4 heads of 128 x 128, 600 tokens, the whole layer: 84 us, 61 so; 16 heads, 300 tokens 88 and 74).
template <bool FROM_ZERO, int WIDTH>
__global__ void __launch_bounds__(256)
scan_combine_kernel(float* __restrict__ seg_state, float* __restrict__ state, const int* __restrict__ cu_q,
                    const int* __restrict__ state_slots, const float* __restrict__ decay, int heads,
                    int per_head, int seg_tokens) {
  struct __align__(4 * WIDTH) Part { float v[WIDTH]; };
  if (FROM_ZERO) pdl_launch_dependents();
  pdl_wait();
  const int seq = blockIdx.y;
  const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * WIDTH, per_segment = (size_t)heads * per_head;
  if (i >= per_segment) return;
  int first_segment = 0;
  for (int q = 0; q < seq; ++q) first_segment += max(1, (cu_q[q + 1] - cu_q[q] + seg_tokens - 1) / seg_tokens);
  const int len = cu_q[seq + 1] - cu_q[seq], ns = max(1, (len + seg_tokens - 1) / seg_tokens);
  const float log2_lam = log2f(decay[i / per_head]);
  float* e = seg_state + (size_t)first_segment * per_segment + i;
  auto at = [&](int s) { return reinterpret_cast<Part*>(e + (size_t)s * per_segment); };
  Part* slot = reinterpret_cast<Part*>(state + (size_t)state_slots[seq] * per_segment + i);
  Part running = FROM_ZERO ? *slot : *at(0);         // what comes into segment 0, or the true state after it
  constexpr int AHEAD = 8;                           // segments whose own parts are on their way at once
  for (int s0 = FROM_ZERO ? 0 : 1; s0 < ns; s0 += AHEAD) {
    Part local[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (s0 + u < ns) local[u] = *at(s0 + u);
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int sg = s0 + u;
      if (sg >= ns) break;
      *at(FROM_ZERO ? sg : sg - 1) = running;
      const float w = decay_power(log2_lam, min(seg_tokens, len - sg * seg_tokens));
#pragma unroll
      for (int x = 0; x < WIDTH; ++x) running.v[x] = fmaf(w, running.v[x], local[u].v[x]);
    }
  }
  *slot = running;
}

template <bool FROM_ZERO>
void launch_combine(int n_seqs, float* seg_state, float* state, const int* cu_q, const int* state_slots, const float* decay, int heads,
                    int per_head, int seg_tokens, cudaStream_t stream) {
  const bool wide = per_head % 4 == 0 && (uintptr_t)seg_state % 16 == 0 && (uintptr_t)state % 16 == 0;
  const size_t threads = (size_t)heads * per_head / (wide ? 4 : 1);
  const dim3 grid((unsigned)((threads + 255) / 256), n_seqs);
  if (wide)
    lb_launch(scan_combine_kernel<FROM_ZERO, 4>, grid, 256, 0, stream, seg_state, state, cu_q, state_slots, decay, heads, per_head, seg_tokens);
  else
    lb_launch(scan_combine_kernel<FROM_ZERO, 1>, grid, 256, 0, stream, seg_state, state, cu_q, state_slots, decay, heads, per_head, seg_tokens);
}

// ------------------------------------------------------------------ segments as matrix products (head sizes up to 128)
constexpr int SEG_THREADS = 256, SEG_ROWS = 64, SEG_PITCH = 132, SEG_STEP = 16;

// Which tokens a block of the grid's z belongs to.
struct Tokens { int seq, first, count; };
__device__ __forceinline__ Tokens segment_tokens(const int* __restrict__ cu_q, int n_seqs, int seg_tokens, int g) {
  Tokens k;
  int segment, first_segment;
  find_segment(cu_q, n_seqs, seg_tokens, g, k.seq, segment, first_segment);
  k.first = cu_q[k.seq] + segment * seg_tokens;
  k.count = max(0, min(seg_tokens, cu_q[k.seq + 1] - k.first));
  return k;
}

// Four neighbouring activated channels c .. c + 3 of a token's head (zeros past `dim` and for a token that is not there).
template <typename T, int ACT>
__device__ __forceinline__ float4 load_quad(const T* __restrict__ head, int c, int dim, bool there, bool vec) {
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (there && vec && c + 4 <= dim) {
    if (sizeof(T) == 2) {
      const uint2 r = *reinterpret_cast<const uint2*>(head + c);
      const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&r.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&r.y);
      v[0] = __low2float(lo); v[1] = __high2float(lo); v[2] = __low2float(hi); v[3] = __high2float(hi);
    } else {
      const float4 r = *reinterpret_cast<const float4*>(head + c);
      v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
    }
  } else if (there) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (c + e < dim) v[e] = Elem<T>::load(head + c + e);
  }
  return make_float4(activate<ACT>(v[0]), activate<ACT>(v[1]), activate<ACT>(v[2]), activate<ACT>(v[3]));
}

// Two neighbouring sums at once: c = (x, x) * r + c, each the fused multiply-add that fmaf is.
__device__ __forceinline__ void multiply_add_pair(float2& c, float x, float2 r) {
  unsigned long long xx, rr = *reinterpret_cast<const unsigned long long*>(&r), cc = *reinterpret_cast<const unsigned long long*>(&c);
  asm("mov.b64 %0, {%1, %1};" : "=l"(xx) : "f"(x));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(cc) : "l"(xx), "l"(rr));
  c = *reinterpret_cast<float2*>(&cc);
}

// E of one segment and head, 128 value columns a block: a 128 x 128 tile, 8 x 8 sums a thread, 16 tokens a step through two
// buffers. What bounds it is the latency of its few warps: 128 registers a thread leave two blocks an SM, 22 % of its warps, which
// wait for the next step's rows and their stores (one prompt of 1,500 tokens, 32 heads of 128 x 128: FFMA pipes 33 % and issue slots
// 45 % busy, 27 % of the memory system's rate, with one sum an instruction: 84 us inside a step, 77 with two).
template <typename T, int ACT>
__global__ void __launch_bounds__(SEG_THREADS, 2)
segment_state_kernel(const T* __restrict__ proj, long row_stride, int k_off, int v_off, const int* __restrict__ cu_q,
                     const float* __restrict__ decay, int heads, int dim, int vdim, float* __restrict__ seg_state, int seg_tokens,
                     int n_seqs, bool vec) {
  __shared__ __align__(16) float k_s[2][SEG_STEP][128], v_s[2][SEG_STEP][128];
  pdl_launch_dependents();
  pdl_wait();
  const int head = blockIdx.y, e0 = blockIdx.x * 128, tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const Tokens seg = segment_tokens(cu_q, n_seqs, seg_tokens, blockIdx.z);
  const float log2_lam = log2f(decay[head]);
  float4 k_next[2], v_next[2];             // a thread stages two quads of k and of v a step
  auto fetch = [&](int t0) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = t0 + (threadIdx.x >> 5) + 8 * u, c = (threadIdx.x & 31) * 4;
      const T* row = proj + (size_t)(seg.first + t) * row_stride;
      k_next[u] = load_quad<T, ACT>(row + k_off + head * dim, c, dim, t < seg.count, vec);
      v_next[u] = load_quad<T, ACT>(row + v_off + head * vdim, e0 + c, vdim, t < seg.count, vec);
      const float w = t < seg.count ? decay_power(log2_lam, seg.count - 1 - t) : 0.f;
      k_next[u].x *= w; k_next[u].y *= w; k_next[u].z *= w; k_next[u].w *= w;
    }
  };
  auto stage = [&](int buf) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int t = (threadIdx.x >> 5) + 8 * u, c = (threadIdx.x & 31) * 4;
      *reinterpret_cast<float4*>(&k_s[buf][t][c]) = k_next[u];
      *reinterpret_cast<float4*>(&v_s[buf][t][c]) = v_next[u];
    }
  };
  float2 acc[8][4];                        // sums of columns 2 j, 2 j + 1
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
  fetch(0);
  stage(0);
  __syncthreads();
  for (int t0 = 0, buf = 0; t0 < seg.count; t0 += SEG_STEP, buf ^= 1) {
    const bool more = t0 + SEG_STEP < seg.count;
    if (more) fetch(t0 + SEG_STEP);
#pragma unroll 4
    for (int t = 0; t < SEG_STEP; ++t) {
      const float4 ka = *reinterpret_cast<const float4*>(&k_s[buf][t][4 * ty]), kb = *reinterpret_cast<const float4*>(&k_s[buf][t][64 + 4 * ty]);
      const float4 va = *reinterpret_cast<const float4*>(&v_s[buf][t][4 * tx]), vb = *reinterpret_cast<const float4*>(&v_s[buf][t][64 + 4 * tx]);
      const float k[8] = {ka.x, ka.y, ka.z, ka.w, kb.x, kb.y, kb.z, kb.w};
      const float2 v[4] = {make_float2(va.x, va.y), make_float2(va.z, va.w), make_float2(vb.x, vb.y), make_float2(vb.z, vb.w)};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) multiply_add_pair(acc[i][j], k[i], v[j]);
    }
    if (more) stage(buf ^ 1);
    __syncthreads();
  }
  float* to = seg_state + ((size_t)blockIdx.z * heads + head) * dim * vdim;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int d = 64 * (i >> 2) + 4 * ty + (i & 3);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int e = e0 + 64 * (j >> 2) + 4 * tx + (j & 3);
      if (d < dim && e < vdim) to[(size_t)d * vdim + e] = j & 1 ? acc[i][j >> 1].y : acc[i][j >> 1].x;
    }
  }
}

// The outputs of 64 tokens of one segment and head, 128 value columns a block. A thread has 4 tokens x 8 columns (8 x 8, half
// as many threads, took 282 us where this takes 194): first
// S_in^T q over slices of 64 rows of S_in, times decay^(i+1); then, for every block of 64 keys up to the tokens' own, the
// 64 x 64 weights decay^(i-j) (q_i . k_j) through shared memory, and their product with the values. Rows of 132 floats keep
// the 16-byte reads along a row free of bank conflicts. What bounds it is the latency of a block's chain, load, barrier,
// multiply, with two blocks an SM (registers and shared memory) to hide it: FFMA pipes 32 % and issue slots 45 % busy, shared-memory
// reads 43 %, with one sum an instruction: 150 us at the size below inside a step, 138 with two.
// Measured (one B200, one prompt of 1,500 tokens, 32 heads of 128 x 128, the three launches of a layer, states,
// joining, outputs): 129 + 10 + 310 us when the segments walked their tokens one by one, then 90 + 24 + 193 us with
// segments of 128, 283 in all with segments of 64, whose blocks have equal work, 237 with two sums an instruction and the joining
// in 20. The next block's rows on their way while one is
// multiplied changed nothing (305 against 306 us).
template <typename T, int ACT>
__global__ void __launch_bounds__(SEG_THREADS, 2)
segment_output_kernel(const T* __restrict__ proj, long row_stride, int q_off, int k_off, int v_off, float* __restrict__ out,
                      const int* __restrict__ cu_q, const float* __restrict__ decay, int heads, int dim, int vdim,
                      const float* __restrict__ seg_state, int seg_tokens, int n_seqs, int e_tiles, bool vec, bool vec_state) {
  extern __shared__ __align__(16) float scan_smem[];
  float* q_s = scan_smem;                                   // [64][SEG_PITCH]
  float* block_s = q_s + SEG_ROWS * SEG_PITCH;              // [64][SEG_PITCH]: a slice of S_in, keys, values
  float* a_s = block_s + SEG_ROWS * SEG_PITCH;              // [64][68]
  constexpr int A_PITCH = SEG_ROWS + 4;
  pdl_launch_dependents();
  pdl_wait();
  const int head = blockIdx.y, e0 = blockIdx.x % e_tiles * 128, i0 = blockIdx.x / e_tiles * SEG_ROWS;
  const Tokens seg = segment_tokens(cu_q, n_seqs, seg_tokens, blockIdx.z);
  if (i0 >= seg.count) return;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const float log2_lam = log2f(decay[head]);
  // 64 tokens from t0 on, 128 channels each from column `off` of their rows
  auto load_block = [&](float* dst, int t0, int off, int c0, int size) {
#pragma unroll
    for (int u = 0; u < SEG_ROWS * 32 / SEG_THREADS; ++u) {
      const int t = (threadIdx.x >> 5) + 8 * u, c = (threadIdx.x & 31) * 4;
      *reinterpret_cast<float4*>(dst + t * SEG_PITCH + c) =
          load_quad<T, ACT>(proj + (size_t)(seg.first + t0 + t) * row_stride + off, c0 + c, size, t0 + t < seg.count, vec);
    }
  };
  load_block(q_s, i0, q_off + head * dim, 0, dim);
  float2 acc[4][4];                                         // sums of columns 2 j, 2 j + 1
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = make_float2(0.f, 0.f);
  // acc += rows of `left` (4 ty ..; `columns` columns from c0 on) times the first `columns` rows of block_s; a CORNER leaves out
  // what lies above the diagonal of its four columns
  auto multiply_quad = [&](const float* left, int pitch, int c, auto corner) {
    constexpr bool CORNER = decltype(corner)::value;
    float4 l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) l[i] = *reinterpret_cast<const float4*>(left + (4 * ty + i) * pitch + c);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const float* row = block_s + (c % SEG_ROWS + s) * SEG_PITCH;
      const float4 ra = *reinterpret_cast<const float4*>(row + 4 * tx), rb = *reinterpret_cast<const float4*>(row + 64 + 4 * tx);
      const float2 r[4] = {make_float2(ra.x, ra.y), make_float2(ra.z, ra.w), make_float2(rb.x, rb.y), make_float2(rb.z, rb.w)};
#pragma unroll
      for (int i = CORNER ? s : 0; i < 4; ++i) {
        const float x = s == 0 ? l[i].x : s == 1 ? l[i].y : s == 2 ? l[i].z : l[i].w;
#pragma unroll
        for (int j = 0; j < 4; ++j) multiply_add_pair(acc[i][j], x, r[j]);
      }
    }
  };
  auto multiply = [&](const float* left, int pitch, int c0, int columns) {
#pragma unroll 2
    for (int c = 0; c < columns; c += 4) multiply_quad(left, pitch, c0 + c, std::false_type());
  };
  const float* from = seg_state + ((size_t)blockIdx.z * heads + head) * dim * vdim;
  for (int d0 = 0; d0 < dim; d0 += SEG_ROWS) {
    __syncthreads();                                        // the slice before is read
#pragma unroll
    for (int u = 0; u < SEG_ROWS * 32 / SEG_THREADS; ++u) {
      const int d = d0 + (threadIdx.x >> 5) + 8 * u, c = (threadIdx.x & 31) * 4;
      *reinterpret_cast<float4*>(block_s + (d - d0) * SEG_PITCH + c) =
          load_quad<float, 0>(from + (size_t)d * vdim, e0 + c, vdim, d < dim, vec_state);
    }
    __syncthreads();
    multiply(q_s, SEG_PITCH, d0, SEG_ROWS);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float w = decay_power(log2_lam, i0 + 4 * ty + i + 1);
#pragma unroll
    for (int j = 0; j < 4; ++j) { acc[i][j].x *= w; acc[i][j].y *= w; }
  }
  for (int j0 = 0; j0 <= i0; j0 += SEG_ROWS) {
    __syncthreads();                                        // block_s and a_s are read
    load_block(block_s, j0, k_off + head * dim, 0, dim);
    __syncthreads();
    float dot[4][4];                                        // tokens 4 ty + i, keys tx + 16 j
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) dot[i][j] = 0.f;
#pragma unroll 2
    for (int c = 0; c < dim; c += 4) {
      float4 qv[4], kv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const float4*>(q_s + (4 * ty + i) * SEG_PITCH + c);
#pragma unroll
      for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(block_s + (tx + 16 * j) * SEG_PITCH + c);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          dot[i][j] = fmaf(qv[i].x, kv[j].x, dot[i][j]);
          dot[i][j] = fmaf(qv[i].y, kv[j].y, dot[i][j]);
          dot[i][j] = fmaf(qv[i].z, kv[j].z, dot[i][j]);
          dot[i][j] = fmaf(qv[i].w, kv[j].w, dot[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int apart = i0 + 4 * ty + i - (j0 + tx + 16 * j);
        a_s[(4 * ty + i) * A_PITCH + tx + 16 * j] = apart >= 0 ? decay_power(log2_lam, apart) * dot[i][j] : 0.f;
      }
    __syncthreads();                                        // the keys are read, the weights are there
    load_block(block_s, j0, v_off + head * vdim, e0, vdim);
    __syncthreads();
    // a token takes the values of its own and of earlier tokens alone: a weight of 0 does not keep out a value that is not finite
    if (j0 < i0) {
      multiply(a_s, A_PITCH, 0, SEG_ROWS);
    } else {
      multiply(a_s, A_PITCH, 0, 4 * ty);
      multiply_quad(a_s, A_PITCH, 4 * ty, std::true_type());
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = i0 + 4 * ty + i;
    if (t >= seg.count) continue;
    float* o = out + ((size_t)(seg.first + t) * heads + head) * vdim + e0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int e = 64 * (j >> 2) + 4 * tx + (j & 3);
      if (e0 + e < vdim) o[e] = j & 1 ? acc[i][j >> 1].y : acc[i][j >> 1].x;
    }
  }
}

template <typename T, int ACT>
int launch_segments(int n_seqs, int total_segments, int seg_tokens, float* seg_state, cudaStream_t stream, const void* proj,
                    long row_stride, int q_off, int k_off, int v_off, float* out, float* state, const int* cu_q,
                    const int* state_slots, const float* decay, int heads, int dim, int vdim) {
  constexpr int smem = (2 * SEG_ROWS * SEG_PITCH + SEG_ROWS * (SEG_ROWS + 4)) * (int)sizeof(float);
  static LbPerDeviceOnce once;
  auto kernel = segment_output_kernel<T, ACT>;
  if (!once.run(LB_ALLOW_SMEM(kernel, smem))) return lb_last_error();
  const int e_tiles = (vdim + 127) / 128, row_blocks = (seg_tokens + SEG_ROWS - 1) / SEG_ROWS, per_head = dim * vdim;
  // four channels at a time where every head's rows start on four elements' boundaries
  const bool vec = (uintptr_t)proj % (4 * sizeof(T)) == 0 && row_stride % 4 == 0 && q_off % 4 == 0 && k_off % 4 == 0 && v_off % 4 == 0 &&
                   dim % 4 == 0 && vdim % 4 == 0;
  const bool vec_state = (uintptr_t)seg_state % 16 == 0 && vdim % 4 == 0;      // the caller's scratch may begin anywhere
  lb_launch(segment_state_kernel<T, ACT>, dim3(e_tiles, heads, total_segments), SEG_THREADS, 0, stream, (const T*)proj, row_stride, k_off,
            v_off, cu_q, decay, heads, dim, vdim, seg_state, seg_tokens, n_seqs, vec);
  launch_combine<true>(n_seqs, seg_state, state, cu_q, state_slots, decay, heads, per_head, seg_tokens, stream);
  lb_launch(segment_output_kernel<T, ACT>, dim3(row_blocks * e_tiles, heads, total_segments), SEG_THREADS, (size_t)smem, stream,
            (const T*)proj, row_stride, q_off, k_off, v_off, out, cu_q, decay, heads, dim, vdim, (const float*)seg_state, seg_tokens, n_seqs,
            e_tiles, vec, vec_state);
  return lb_last_error();
}

template <typename T, int RANGES, int DPT, int ACT, int MODE>
int launch_scan_mode(dim3 grid, cudaStream_t stream, const void* proj, long row_stride, int q_off, int k_off, int v_off,
                     float* out, float* state, const int* cu_q, const int* state_slots, const float* decay, int heads,
                     int dim, int vdim, float* seg_state, int seg_tokens, int n_seqs) {
  // q and k twice (two buffers), v twice, the warps' partial sums
  constexpr size_t smem = (size_t)(4 * CHUNK * RANGES * DPT + 2 * CHUNK * COLS + CHUNK * RANGES * COLS) * sizeof(float);
  static LbPerDeviceOnce once;
  auto kernel = decay_scan_kernel<T, RANGES, DPT, ACT, MODE>;
  if (smem > 48 * 1024 && !once.run(LB_ALLOW_SMEM(kernel, smem))) return lb_last_error();
  lb_launch(decay_scan_kernel<T, RANGES, DPT, ACT, MODE>, grid, RANGES * COLS, smem, stream, (const T*)proj, row_stride, q_off,
            k_off, v_off, out, state, cu_q, state_slots, decay, heads, dim, vdim, seg_state, seg_tokens, n_seqs);
  return lb_last_error();
}

template <typename T, int RANGES, int DPT, int ACT>
int launch_scan(int n_seqs, int total_segments, int seg_tokens, float* seg_state, cudaStream_t stream, const void* proj,
                long row_stride, int q_off, int k_off, int v_off, float* out, float* state, const int* cu_q,
                const int* state_slots, const float* decay, int heads, int dim, int vdim) {
  const unsigned cols = (vdim + COLS - 1) / COLS;
#define LB_MODE(M, Z) launch_scan_mode<T, RANGES, DPT, ACT, M>(dim3(cols, heads, Z), stream, proj, row_stride, q_off, k_off, \
                                                                v_off, out, state, cu_q, state_slots, decay, heads, dim, vdim, \
                                                                seg_state, seg_tokens, n_seqs)
  if (total_segments <= 0) return LB_MODE(0, n_seqs);
  int code = LB_MODE(1, total_segments);
  if (code) return code;
  const int per_head = dim * vdim;
  launch_combine<false>(n_seqs, seg_state, state, cu_q, state_slots, decay, heads, per_head, seg_tokens, stream);
  if ((code = lb_last_error())) return code;
  return LB_MODE(2, total_segments);
#undef LB_MODE
}

template <typename T>
int dispatch_scan(int act, int n_seqs, int total_segments, int seg_tokens, float* seg_state, cudaStream_t stream,
                  const void* proj, long row_stride, int q_off, int k_off, int v_off, float* out, float* state,
                  const int* cu_q, const int* state_slots, const float* decay, int heads, int dim, int vdim, bool products) {
#define LB_SCAN(R, D)                                                                                                        \
  (act == 1 ? launch_scan<T, R, D, 1>(n_seqs, total_segments, seg_tokens, seg_state, stream, proj, row_stride, q_off, k_off, \
                                      v_off, out, state, cu_q, state_slots, decay, heads, dim, vdim)                         \
            : launch_scan<T, R, D, 0>(n_seqs, total_segments, seg_tokens, seg_state, stream, proj, row_stride, q_off, k_off, \
                                      v_off, out, state, cu_q, state_slots, decay, heads, dim, vdim))
  if (total_segments > 0 && products) {
    if (act == 1)
      return launch_segments<T, 1>(n_seqs, total_segments, seg_tokens, seg_state, stream, proj, row_stride, q_off, k_off, v_off, out, state,
                                   cu_q, state_slots, decay, heads, dim, vdim);
    return launch_segments<T, 0>(n_seqs, total_segments, seg_tokens, seg_state, stream, proj, row_stride, q_off, k_off, v_off, out, state,
                                 cu_q, state_slots, decay, heads, dim, vdim);
  }
  if (dim <= 32) return LB_SCAN(8, 4);          // the split of S over warps is a function of the head size alone
  if (dim <= 64) return LB_SCAN(16, 4);
  if (dim <= 128) return LB_SCAN(16, 8);
  return LB_SCAN(8, 32);
#undef LB_SCAN
}

// out[t, i] = T(x[t, i] * rsqrt(mean_i x[t, i]^2 + eps) * weight[i] / (1 + exp(-gate[t, i])))
// x 32-bit [tokens, n]; gate logits in the run's type inside a wider row (gate_stride elements apart).
template <typename T, bool VEC>
__global__ void gated_rmsnorm_kernel(const float* __restrict__ x, const T* __restrict__ gate, long gate_stride,
                                     const float* __restrict__ weight, T* __restrict__ out, int n, float eps) {
  __shared__ float scratch[33];
  pdl_launch_dependents();
  pdl_wait();
  const float* xr = x + (size_t)blockIdx.x * n;
  const T* gr = gate + (size_t)blockIdx.x * gate_stride;
  T* o = out + (size_t)blockIdx.x * n;
  float ss = 0.f;
  if (VEC) {        // n a multiple of 4, rows on 16-byte (bf16: 8-byte) boundaries
    for (int i = threadIdx.x * 4; i < n; i += blockDim.x * 4) {
      const float4 v = *reinterpret_cast<const float4*>(xr + i);
      ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) ss += xr[i] * xr[i];
  }
  const float inv = 1.0f / sqrtf(block_sum(ss, scratch) / (float)n + eps);
  if (VEC) {
    for (int i = threadIdx.x * 4; i < n; i += blockDim.x * 4) {
      const float4 v = *reinterpret_cast<const float4*>(xr + i), w = *reinterpret_cast<const float4*>(weight + i);
      float g[4], y[4] = {v.x * inv * w.x, v.y * inv * w.y, v.z * inv * w.z, v.w * inv * w.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) g[u] = Elem<T>::load(gr + i + u);
#pragma unroll
      for (int u = 0; u < 4; ++u) Elem<T>::store(o + i + u, y[u] / (1.0f + expf(-g[u])));
    }
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x)
      Elem<T>::store(o + i, xr[i] * inv * weight[i] / (1.0f + expf(-Elem<T>::load(gr + i))));
  }
}
}  // namespace

// proj [tokens, row_stride] holds q at q_off (heads * dim), k at k_off (heads * dim), v at v_off (heads * vdim);
// out float [tokens, heads * vdim]; state float [slots, heads, dim, vdim]; decay float [heads]; act 0 none, 1 silu.
// total_segments > 0: the three-launch form for steps with long portions; seg_state float
// [total_segments, heads, dim, vdim], total_segments = sum over sequences of max(1, ceil(tokens / seg_tokens)). products: the
// segments as matrix products (head sizes up to 128), else they walk their tokens.
LB_EXPORT int lb_decay_scan(int dtype, const void* proj, long row_stride, int q_off, int k_off, int v_off, float* out,
                            float* state, const int* cu_q, const int* state_slots, const float* decay, int n_seqs,
                            int heads, int dim, int vdim, int act, float* seg_state, int seg_tokens, int total_segments,
                            int products, cudaStream_t stream) {
  if (n_seqs <= 0) return 0;
  if (products && dim > 128) return LB_ERR_SIZE;         // a block's shared memory holds 64 rows of 128 channels
  if (heads <= 0 || heads > 65535 || n_seqs > 65535 || dim <= 0 || dim > 256 || vdim <= 0 || act < 0 || act > 1)
    return LB_ERR_SIZE;
  if (total_segments > 0 && (!seg_state || seg_tokens <= 0 || total_segments < n_seqs || total_segments > 65535))
    return LB_ERR_SIZE;
  if (dtype == LB_F32)
    return dispatch_scan<float>(act, n_seqs, total_segments, seg_tokens, seg_state, stream, proj, row_stride, q_off, k_off,
                                v_off, out, state, cu_q, state_slots, decay, heads, dim, vdim, products != 0);
  if (dtype == LB_BF16)
    return dispatch_scan<bf16>(act, n_seqs, total_segments, seg_tokens, seg_state, stream, proj, row_stride, q_off, k_off,
                               v_off, out, state, cu_q, state_slots, decay, heads, dim, vdim, products != 0);
  return LB_ERR_DTYPE;
}

LB_EXPORT int lb_gated_rmsnorm(int dtype, const float* x, const void* gate, long gate_stride, const float* weight,
                               void* out, int tokens, int n, float eps, cudaStream_t stream) {
  if (tokens <= 0) return 0;
  if (n <= 0) return LB_ERR_SIZE;
  const int threads = n >= 1024 ? 256 : 128;
  const bool vec = n % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)weight % 16 == 0;
  if (dtype == LB_F32) {
    if (vec)
      lb_launch(gated_rmsnorm_kernel<float, true>, tokens, threads, 0, stream, x, (const float*)gate, gate_stride, weight, (float*)out, n, eps);
    else lb_launch(gated_rmsnorm_kernel<float, false>, tokens, threads, 0, stream, x, (const float*)gate, gate_stride, weight, (float*)out, n, eps);
  } else if (dtype == LB_BF16) {
    if (vec) lb_launch(gated_rmsnorm_kernel<bf16, true>, tokens, threads, 0, stream, x, (const bf16*)gate, gate_stride, weight, (bf16*)out, n, eps);
    else lb_launch(gated_rmsnorm_kernel<bf16, false>, tokens, threads, 0, stream, x, (const bf16*)gate, gate_stride, weight, (bf16*)out, n, eps);
  } else
    return LB_ERR_DTYPE;
  return lb_last_error();
}
