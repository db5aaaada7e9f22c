// C[M, N] = A[M, K] * W[N, K]^T with 32-bit FFMA accumulation: the matrix product of the true
// 32-bit path (no tensor cores, no TF32), also instantiated for bf16 operands as the slow
// oracle of the tensor-core kernel. Row strides are given in elements.
//
// Each output element is a sum in a fixed order, whatever M is and wherever the row sits in its tile, so a
// token's result does not depend on how a batch was cut. For 32-bit operands K is cut into the ranges of `Split`, which
// depend on K alone; a range is one sequential chain of fused multiply-adds from zero, the sums of four neighbouring ranges
// are added in order, and then the sums of those groups are. Ranges may therefore run one after the other, in the lanes
// of a warp or in different blocks, with the same bits. For bf16 operands there is one chain over the whole of K. Any
// M, N, K >= 1 is accepted: operands whose
// address and stride TMA can take go through the streaming kernels, others through the plain tiles, with the same bits.
#include "common.cuh"
#include "tcgen05.cuh"

namespace {
constexpr int TILE_M = 64, TILE_N = 64, TILE_K = 16, TM = 4, TN = 4, THREADS = 256;

template <typename T> struct Vec4;
template <> struct Vec4<float> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[4]) {
    const float4 r = *reinterpret_cast<const float4*>(p);
    v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
  }
};
template <> struct Vec4<bf16> {
  static __device__ __forceinline__ void load(const bf16* p, float (&v)[4]) {
    const uint2 r = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&r.x);
    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&r.y);
    v[0] = __low2float(a); v[1] = __high2float(a); v[2] = __low2float(b); v[3] = __high2float(b);
  }
};

// loads a [rows_in_tile=64, TILE_K] slab, K-contiguous in memory, into smem transposed [TILE_K][64+4]
template <typename T>
__device__ __forceinline__ void load_slab(const T* __restrict__ base, long ld, int row0, int n_rows, int k0, int K,
                                          bool vec_ok, float (*dst)[TILE_M + 4]) {
  const int r = threadIdx.x >> 2, kk = (threadIdx.x & 3) * 4;
  const int row = row0 + r;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  if (row < n_rows) {
    const T* p = base + (long)row * ld + k0 + kk;
    if (vec_ok && k0 + kk + 3 < K) {
      Vec4<T>::load(p, v);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (k0 + kk + j < K) v[j] = Elem<T>::load(p + j);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) dst[kk + j][r] = v[j];
}

// RANGES: sums over the ranges of `Split` (of `range_length` k each); what a thread keeps between them lies in shared memory, where
// it costs no registers: 261 tokens x 6,144 x 2,561 (rows that TMA does not take) 564 us, in registers 642, one chain of K 530.
template <typename TA, typename TC, bool RANGES = false>
__global__ void __launch_bounds__(THREADS, RANGES ? 5 : 0)
gemm_simt_kernel(const TA* __restrict__ A, const TA* __restrict__ W, TC* __restrict__ C, int M, int N, int K,
                 long lda, long ldw, long ldc, bool vec_a, bool vec_w, int range_length) {
  __shared__ float As[TILE_K][TILE_M + 4];
  __shared__ float Ws[TILE_K][TILE_N + 4];
  __shared__ float kept[RANGES ? 2 * TM * TN : 1][RANGES ? THREADS : 1];     // of the group's ranges before, of the groups before
  pdl_launch_dependents();
  pdl_wait();
  const int m0 = blockIdx.y * TILE_M, n0 = blockIdx.x * TILE_N;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[TM][TN];                      // of the current range of K
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

  int k0 = 0;
  for (int range = 0; k0 < K; ++range) {
    const int end = RANGES ? min(K, k0 + range_length) : K;
    for (; k0 < end; k0 += TILE_K) {
      load_slab<TA>(A, lda, m0, M, k0, K, vec_a, As);
      load_slab<TA>(W, ldw, n0, N, k0, K, vec_w, Ws);
      __syncthreads();
#pragma unroll
      for (int k = 0; k < TILE_K; ++k) {
        float a[TM], w[TN];
#pragma unroll
        for (int i = 0; i < TM; ++i) a[i] = As[k][ty * TM + i];
#pragma unroll
        for (int j = 0; j < TN; ++j) w[j] = Ws[k][tx * TN + j];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
      }
      __syncthreads();
    }
    if (!RANGES) break;
    const bool last = k0 >= K;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        float *group = &kept[i * TN + j][threadIdx.x], *total = &kept[TM * TN + i * TN + j][threadIdx.x];
        float sum = range % 4 ? *group + acc[i][j] : acc[i][j];
        if (range % 4 == 3 || last) {
          if (range >= 4) sum = *total + sum;
          *total = sum;
        } else {
          *group = sum;
        }
        acc[i][j] = last ? sum : 0.f;
      }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int row = m0 + ty * TM + i;
    if (row >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int col = n0 + tx * TN + j;
      if (col < N) Elem<TC>::store(C + (long)row * ldc + col, acc[i][j]);
    }
  }
}

// The same product of bf16 operands for steps of at most 16 tokens: tiles of 16 tokens x 16 weight rows, so that a
// weight matrix of a few thousand rows still gives every SM a block (the 64 x 64 tiles above leave
// most of the GPU idle then and spend 7/8 of their arithmetic on rows that are not there). A thread
// owns one weight row and two tokens; the next slab of 32 k is fetched into registers while the
// current one is used. Every output element is still ONE sequential fused-multiply-add chain over
// k = 0..K-1 starting from zero, so it has the bits the large-tile kernel gives the same token.
constexpr int FT_M = 16, FT_N = 16, FT_K = 32, FT_THREADS = 128;

template <typename T>
__device__ __forceinline__ void fetch_quad(const T* __restrict__ base, long ld, int row, int n_rows, int k, int K, bool vec,
                                           float (&v)[4]) {
  v[0] = v[1] = v[2] = v[3] = 0.f;
  if (row >= n_rows) return;
  const T* p = base + (long)row * ld + k;
  if (vec && k + 3 < K) {
    Vec4<T>::load(p, v);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (k + j < K) v[j] = Elem<T>::load(p + j);
  }
}

template <typename TA, typename TC>
__global__ void __launch_bounds__(FT_THREADS)
gemm_simt_fewtoken_kernel(const TA* __restrict__ A, const TA* __restrict__ W, TC* __restrict__ C, int M, int N, int K,
                          long lda, long ldw, long ldc, bool vec_a, bool vec_w) {
  __shared__ float As[FT_K][FT_M + 1];
  __shared__ float Ws[FT_K][FT_N + 1];
  pdl_launch_dependents();
  pdl_wait();
  const int n0 = blockIdx.x * FT_N, m0 = blockIdx.y * FT_M;
  const int lr = threadIdx.x >> 3, lk = (threadIdx.x & 7) * 4;      // the row and the four k this thread fetches of a slab
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;           // weight row of the tile, pair of tokens
  float acc[2] = {0.f, 0.f};
  float next_a[4], next_w[4];
  fetch_quad<TA>(A, lda, m0 + lr, M, lk, K, vec_a, next_a);
  fetch_quad<TA>(W, ldw, n0 + lr, N, lk, K, vec_w, next_w);
  for (int k0 = 0; k0 < K; k0 += FT_K) {
#pragma unroll
    for (int j = 0; j < 4; ++j) { As[lk + j][lr] = next_a[j]; Ws[lk + j][lr] = next_w[j]; }
    __syncthreads();
    if (k0 + FT_K < K) {
      fetch_quad<TA>(A, lda, m0 + lr, M, k0 + FT_K + lk, K, vec_a, next_a);
      fetch_quad<TA>(W, ldw, n0 + lr, N, k0 + FT_K + lk, K, vec_w, next_w);
    }
    const int steps = min(FT_K, K - k0);
    if (steps == FT_K) {
#pragma unroll
      for (int k = 0; k < FT_K; ++k) {
        const float w = Ws[k][tx];
        acc[0] = fmaf(As[k][2 * ty], w, acc[0]);
        acc[1] = fmaf(As[k][2 * ty + 1], w, acc[1]);
      }
    } else {
      for (int k = 0; k < steps; ++k) {      // the k beyond K would add exact zeros; they are left out all the same
        const float w = Ws[k][tx];
        acc[0] = fmaf(As[k][2 * ty], w, acc[0]);
        acc[1] = fmaf(As[k][2 * ty + 1], w, acc[1]);
      }
    }
    __syncthreads();
  }
  const int col = n0 + tx;
  if (col < N) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = m0 + 2 * ty + i;
      if (row < M) Elem<TC>::store(C + (long)row * ldc + col, acc[i]);
    }
  }
}

template <typename T> bool vec_ok(const void* p, long ld) {
  return ((uintptr_t)p % (4 * sizeof(T)) == 0) && (ld % 4 == 0);
}

// ------------------------------------------------------------------ 32-bit operands
__device__ int g_gemm_simt_error = 0;   // 0 = ok; a wait for a copy ran out in 1 the few-token kernel, 2 the many-token kernel

// The ranges of K: up to 32 of them, whole stages long. Four ranges are a group: the sums of a group's ranges are added in
// order, and then the groups' sums are.
constexpr int STAGE_K = 32;             // 128 bytes of a row
constexpr int GROUP = 4;
struct Split {
  int count, length;
  __host__ __device__ explicit Split(int K) {
    const int blocks = (K + 1023) / 1024, wanted = GROUP * (blocks < 8 ? blocks : 8);
    length = ((K + wanted - 1) / wanted + STAGE_K - 1) / STAGE_K * STAGE_K;
    count = (K + length - 1) / length;
  }
  __host__ __device__ int groups() const { return (count + GROUP - 1) / GROUP; }
};

// The 16 bytes of k .. k + 3 in row `row` of a tile of 128-byte rows as TMA's 128-byte swizzle leaves them.
__device__ __forceinline__ float4 swizzled(const float* tile, int row, int k) {
  return *reinterpret_cast<const float4*>(tile + row * STAGE_K + (((k >> 2) ^ (row & 7)) << 2));
}

// Up to 16 tokens without TMA (rows or addresses that it does not take) and for short K, where the few-token kernel's cluster and
// rings cost more than they bring: tiles of 16 tokens x 16 weight rows, a thread owns one weight row and two tokens. Slabs of 32 k
// come by 4-byte asynchronous copies, PLAIN_STAGES - 1 of them on their way; what bounds it are the reads of shared memory, three for
// two multiply-adds.
// Measured (one B200, 8 tokens, K 2,561, which TMA does not take): 1,024 rows 35 us, 2,560 50, 6,144 88; one slab in registers ahead of
// the other 47, 55 and 85, the 64 x 64 tiles 192, 193 and 226.
constexpr int PLAIN_STAGES = 4;
__device__ __forceinline__ void copy_float(float* dst, const float* src, bool there) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(there ? 4 : 0) : "memory");
}

__global__ void __launch_bounds__(FT_THREADS)
gemm_f32_plain_few_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K, long lda,
                          long ldw, long ldc) {
  __shared__ float As[PLAIN_STAGES][FT_K][FT_M + 1];
  __shared__ float Ws[PLAIN_STAGES][FT_K][FT_N + 1];
  pdl_launch_dependents();
  pdl_wait();
  const int n0 = blockIdx.x * FT_N, slabs = (K + FT_K - 1) / FT_K, range_slabs = Split(K).length / FT_K;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;        // a warp copies four rows of a slab, a lane one k of each
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;           // weight row of the tile, pair of tokens
  auto copy_slab = [&](int i) {                                     // what lies beyond K or the rows becomes zeros
    if (i < slabs) {
      const int buf = i % PLAIN_STAGES, k = i * FT_K + lane, k_at = min(k, K - 1);
#pragma unroll
      for (int j = 0; j < FT_M / 4; ++j) {
        const int r = warp * (FT_M / 4) + j;
        copy_float(&As[buf][lane][r], A + min(r, M - 1) * lda + k_at, r < M && k < K);
        copy_float(&Ws[buf][lane][r], W + min(n0 + r, N - 1) * ldw + k_at, n0 + r < N && k < K);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < PLAIN_STAGES - 1; ++i) copy_slab(i);
  float acc[2] = {0.f, 0.f}, group[2] = {0.f, 0.f}, total[2] = {0.f, 0.f};
  int range = 0, left = range_slabs;
  for (int i = 0; i < slabs; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(PLAIN_STAGES - 2) : "memory");
    __syncthreads();                                                // the slab is there, and the one before is read
    copy_slab(i + PLAIN_STAGES - 1);
    const int buf = i % PLAIN_STAGES;
#pragma unroll
    for (int k = 0; k < FT_K; ++k) {
      const float w = Ws[buf][k][tx];
      acc[0] = fmaf(As[buf][k][2 * ty], w, acc[0]);
      acc[1] = fmaf(As[buf][k][2 * ty + 1], w, acc[1]);
    }
    if (--left == 0 || i + 1 == slabs) {
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        group[t] = range % GROUP ? group[t] + acc[t] : acc[t];
        if (range % GROUP == GROUP - 1 || i + 1 == slabs) total[t] = range < GROUP ? group[t] : total[t] + group[t];
        acc[t] = 0.f;
      }
      left = range_slabs;
      ++range;
    }
  }
  const int col = n0 + tx;
  if (col < N) {
#pragma unroll
    for (int t = 0; t < 2; ++t)
      if (2 * ty + t < M) C[(2 * ty + t) * ldc + col] = total[t];
  }
}

// After a wait that ran out: copies still in flight get time to land before the block's memory goes away.
__device__ __forceinline__ void let_copies_land() {
  for (int i = 0; i < 2000; ++i) __nanosleep(1000);
}

// At most 16 tokens: a stream of the weight matrix. A block owns 32 weight rows and four ranges of K, the blocks of a row
// tile are a thread-block cluster. A warp fills a ring of stages of its own with TMA (32 k of its rows and of the
// tokens, for each of its ranges: one lane issues the copies) and waits for nobody else. Its lanes are 8 row lanes x
// ranges (x 2 halves of the tokens beyond 8), and a lane holds the sums of 4 rows x its tokens, so that a
// 16-byte read of shared memory feeds 16 multiply-adds or more (with one row a lane the reads were the bound). Every block
// adds up its group, receives its share of the rows' group sums from the others and adds those. What bounds it is the
// latency of its few warps: two stages of 16 KB a warp, five blocks an SM (three stages and three blocks: 121 us where
// these take 93). `partials` (clusters switched off): a group's sums go there, for `sum_groups_kernel`.
// Measured (one B200, the four products of a layer of 2,560 x 9,728 together, 402 MB of weights): 82 us for one token, 96 for 4
// (4.2 TB/s; 1,350 with one chain of K per thread and 128-thread blocks), 131 for 8, 202 for 16.
constexpr int FEW_ROWS = 32, FEW_STAGES = 2, FEW_LANE_ROWS = FEW_ROWS / 8;
template <int TOKENS> struct Few {
  static constexpr int WARPS = TOKENS > 8 ? 2 : 1, HALVES = WARPS, RANGES = GROUP / WARPS;      // ranges of a warp
  static constexpr int PER_LANE = TOKENS / HALVES;
  static constexpr int W_FLOATS = FEW_ROWS * STAGE_K, A_FLOATS = TOKENS * STAGE_K;                   // of one range
  static constexpr int STAGE_FLOATS = RANGES * (W_FLOATS + A_FLOATS);
  static constexpr int RING_BYTES = WARPS * FEW_STAGES * STAGE_FLOATS * 4, RECEIVED_FLOATS = TOKENS * (FEW_ROWS + 8);
  static constexpr int SMEM = 1024 /* alignment */ + RING_BYTES + RECEIVED_FLOATS * 4 + WARPS * FEW_STAGES * 8;
};

template <int TOKENS>
__global__ void __launch_bounds__(32 * Few<TOKENS>::WARPS)
gemm_f32_few_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, float* __restrict__ C,
                    float* __restrict__ partials, int M, int N, int K, long ldc, bool early_weights) {
  using F = Few<TOKENS>;
  extern __shared__ uint8_t raw_smem[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw_smem) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row_lane = lane & 7, lane_range = (lane >> 3) % F::RANGES, half = (lane >> 3) / F::RANGES;
  const int n0 = blockIdx.x * FEW_ROWS;
  const Split split(K);
  const int range0 = blockIdx.z * GROUP + warp * F::RANGES;             // the warp's first range
  const int stages = split.length / STAGE_K;
  // a warp's weight tiles [stage][range], then its tokens' [stage][range]
  float* w_ring = reinterpret_cast<float*>(smem) + warp * FEW_STAGES * F::RANGES * F::W_FLOATS;
  float* a_ring = reinterpret_cast<float*>(smem) + F::WARPS * FEW_STAGES * F::RANGES * F::W_FLOATS + warp * FEW_STAGES * F::RANGES * F::A_FLOATS;
  float* sums = reinterpret_cast<float*>(smem + F::RING_BYTES);              // [group][token][row of the block's share]
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + F::RING_BYTES + F::RECEIVED_FLOATS * 4) + warp * FEW_STAGES;

  if (lane == 0) {
    for (int s = 0; s < FEW_STAGES; ++s) mbar_init(&full[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncwarp();
  // one lane: what lies beyond K or the rows is filled with zeros
  auto copy_weights = [&](int i) {
    const int s = i % FEW_STAGES;
    mbar_expect_tx(&full[s], F::STAGE_FLOATS * 4);
    for (int r = 0; r < F::RANGES; ++r)
      tma_load_2d(w_ring + (s * F::RANGES + r) * F::W_FLOATS, &map_w, &full[s], (range0 + r) * split.length + i * STAGE_K, n0);
  };
  auto copy_tokens = [&](int i) {
    const int s = i % FEW_STAGES;
    for (int r = 0; r < F::RANGES; ++r)
      tma_load_2d(a_ring + (s * F::RANGES + r) * F::A_FLOATS, &map_a, &full[s], (range0 + r) * split.length + i * STAGE_K, 0);
  };
  if (!partials) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  pdl_launch_dependents();
  // before the wait only what no kernel that may still run writes: the caller says whether the weights are that
  auto first_weights = [&] {
    if (lane == 0)
      for (int i = 0; i < FEW_STAGES && i < stages; ++i) copy_weights(i);
  };
  if (early_weights) first_weights();
  pdl_wait();
  if (!early_weights) first_weights();
  if (lane == 0)
    for (int i = 0; i < FEW_STAGES && i < stages; ++i) copy_tokens(i);

  float acc[FEW_LANE_ROWS][F::PER_LANE];
#pragma unroll
  for (int j = 0; j < FEW_LANE_ROWS; ++j)
#pragma unroll
    for (int t = 0; t < F::PER_LANE; ++t) acc[j][t] = 0.f;
  bool ok = true;
  for (int i = 0; i < stages; ++i) {
    const int s = i % FEW_STAGES;
    ok = mbar_wait(&full[s], (i / FEW_STAGES) & 1);
    if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
    const float* w_tile = w_ring + (s * F::RANGES + lane_range) * F::W_FLOATS;
    const float* a_tile = a_ring + (s * F::RANGES + lane_range) * F::A_FLOATS + half * F::PER_LANE * STAGE_K;
#pragma unroll 4
    for (int k = 0; k < STAGE_K; k += 4) {
      float4 w[FEW_LANE_ROWS], a[F::PER_LANE];
#pragma unroll
      for (int j = 0; j < FEW_LANE_ROWS; ++j) w[j] = swizzled(w_tile, row_lane + 8 * j, k);
#pragma unroll
      for (int t = 0; t < F::PER_LANE; ++t) a[t] = *reinterpret_cast<const float4*>(a_tile + t * STAGE_K + k);
#pragma unroll
      for (int t = 0; t < F::PER_LANE; ++t)
#pragma unroll
        for (int j = 0; j < FEW_LANE_ROWS; ++j) acc[j][t] = fmaf(a[t].x, w[j].x, acc[j][t]);
#pragma unroll
      for (int t = 0; t < F::PER_LANE; ++t)
#pragma unroll
        for (int j = 0; j < FEW_LANE_ROWS; ++j) acc[j][t] = fmaf(a[t].y, w[j].y, acc[j][t]);
#pragma unroll
      for (int t = 0; t < F::PER_LANE; ++t)
#pragma unroll
        for (int j = 0; j < FEW_LANE_ROWS; ++j) acc[j][t] = fmaf(a[t].z, w[j].z, acc[j][t]);
#pragma unroll
      for (int t = 0; t < F::PER_LANE; ++t)
#pragma unroll
        for (int j = 0; j < FEW_LANE_ROWS; ++j) acc[j][t] = fmaf(a[t].w, w[j].w, acc[j][t]);
    }
    __syncwarp();                                        // every lane has read the stage
    if (lane == 0 && i + FEW_STAGES < stages) { copy_weights(i + FEW_STAGES); copy_tokens(i + FEW_STAGES); }
  }
  if (!ok) {
    if (lane == 0) atomicCAS(&g_gemm_simt_error, 0, 1);
    let_copies_land();
  }
  // the group's sum: its ranges' sums meet in this block's shared memory [range][token][row] (the rings are read through)
  float* own = reinterpret_cast<float*>(smem);
  __syncthreads();
#pragma unroll
  for (int j = 0; j < FEW_LANE_ROWS; ++j)
#pragma unroll
    for (int t = 0; t < F::PER_LANE; ++t)
      own[((warp * F::RANGES + lane_range) * TOKENS + half * F::PER_LANE + t) * FEW_ROWS + row_lane + 8 * j] = acc[j][t];
  __syncthreads();
  const int groups = gridDim.z, ranges = min(GROUP, split.count - (int)blockIdx.z * GROUP);
  const int rows_per = (FEW_ROWS + groups - 1) / groups;         // block g adds up rows g * rows_per .. of all groups
  if (!partials) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");      // all blocks run
  for (int i = threadIdx.x; i < M * FEW_ROWS; i += 32 * F::WARPS) {
    const int token = i / FEW_ROWS, row = i % FEW_ROWS;
    float total = own[i];
    for (int r = 1; r < ranges; ++r) total += own[r * TOKENS * FEW_ROWS + i];
    if (partials) {
      if (n0 + row < N) partials[((size_t)blockIdx.z * M + token) * N + n0 + row] = total;
    } else {
      const int owner = row / rows_per;
      lb_store_remote(lb_map_to_rank(smem_u32(sums + (blockIdx.z * TOKENS + token) * rows_per + row - owner * rows_per), owner), total);
    }
  }
  if (partials) return;
  lb_cluster_barrier();
  const int first = blockIdx.z * rows_per, rows = min(rows_per, FEW_ROWS - first);
  for (int i = threadIdx.x; i < M * rows; i += 32 * F::WARPS) {
    const int token = i / rows, r = i % rows, col = n0 + first + r;
    if (col >= N) continue;
    float total = sums[token * rows_per + r];
    for (int g = 1; g < groups; ++g) total += sums[(g * TOKENS + token) * rows_per + r];
    C[(long)token * ldc + col] = total;
  }
}

// More tokens: tiles of 8 TM tokens x 64 weight rows, 128 threads with TM x 4 sums each, a ring of stages of 32 k filled with
// TMA by one thread. A thread reads four k of TM + 4 rows and does 16 TM fused multiply-adds with them. What bounds it is
// the way from shared memory and the register file to the FFMA pipes: 73 % of the shared-memory rate, 49 % of the pipes' cycles, a
// dispatch stall for every instruction issued (261 tokens x 19,456 x 2,560; a loop of nothing but three-register FFMAs reaches
// 55 TFLOP/s);
// three blocks an SM of 32 sums a thread run at the rate of two of 64, and leave fewer rows and SMs idle. `partials` null: a block
// walks all groups of ranges and adds each group's sums to its elements of C, which nobody else touches. Else the grid's z deals
// the groups out, and each group's sums go to partials[group] for `sum_groups_kernel`: for products whose tiles are too few to keep
// every SM at work to the end.
// Measured (one B200, the four products of the same layer together): 1.98 ms for 261 tokens (26 TFLOP/s; 3.54 ms with 64 x 64
// tiles filled by plain loads), 5.99 ms for 1,024 (34 TFLOP/s). cuBLAS in 32-bit, without TF32: 1.38 and 4.01 ms.
constexpr int MANY_COLS = 64, MANY_TN = 4, MANY_STAGES = 3, MANY_THREADS = 128;
template <int TM> struct Many {
  static constexpr int ROWS = 8 * TM, STAGE_FLOATS = (ROWS + MANY_COLS) * STAGE_K;
  static constexpr int SMEM = 1024 /* alignment */ + MANY_STAGES * (STAGE_FLOATS * 4 + 8);
};

template <int TM>
__global__ void __launch_bounds__(MANY_THREADS, 3)
gemm_f32_many_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, float* __restrict__ C,
                     float* __restrict__ partials, int M, int N, int K, long ldc) {
  using T = Many<TM>;
  extern __shared__ uint8_t raw_smem[];
  float* ring = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(raw_smem) + 1023) & ~(uintptr_t)1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + MANY_STAGES * T::STAGE_FLOATS);
  const unsigned tiles_m = (M + T::ROWS - 1) / T::ROWS;        // the tiles of the same weight rows are neighbours
  const int m0 = (int)(blockIdx.x % tiles_m) * T::ROWS, n0 = (int)(blockIdx.x / tiles_m) * MANY_COLS;
  const int tn = threadIdx.x & 15, tm = threadIdx.x >> 4;      // weight rows tn + 16 j, tokens tm + 8 i
  const Split split(K);
  const int first_group = (int)(split.groups() * blockIdx.z / gridDim.z), end_group = (int)(split.groups() * (blockIdx.z + 1) / gridDim.z);
  const int k_begin = first_group * GROUP * split.length, k_end = min(K, end_group * GROUP * split.length);
  const int stages = (k_end - k_begin + STAGE_K - 1) / STAGE_K, per_range = split.length / STAGE_K;

  if (threadIdx.x == 0) {
    for (int s = 0; s < MANY_STAGES; ++s) mbar_init(&full[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  auto copy_stage = [&](int i) {                               // one thread
    const int s = i % MANY_STAGES, k = k_begin + i * STAGE_K;
    mbar_expect_tx(&full[s], T::STAGE_FLOATS * 4);
    tma_load_2d(ring + s * T::STAGE_FLOATS, &map_a, &full[s], k, m0);
    tma_load_2d(ring + s * T::STAGE_FLOATS + T::ROWS * STAGE_K, &map_w, &full[s], k, n0);
  };
  __syncthreads();
  pdl_launch_dependents();
  pdl_wait();
  if (threadIdx.x == 0)
    for (int i = 0; i < MANY_STAGES - 1 && i < stages; ++i) copy_stage(i);
  float acc[TM][MANY_TN], group[TM][MANY_TN];                  // of the current range, and of the group's ranges before it
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < MANY_TN; ++j) acc[i][j] = group[i][j] = 0.f;
  bool ok = true;
  for (int s = 0; s < stages; ++s) {
    const bool landed = mbar_wait(&full[s % MANY_STAGES], (s / MANY_STAGES) & 1);
    if (!__syncthreads_and(landed)) { ok = false; break; }     // and everybody has read the stage before
    if (threadIdx.x == 0 && s + MANY_STAGES - 1 < stages) copy_stage(s + MANY_STAGES - 1);
    const float* a_s = ring + (s % MANY_STAGES) * T::STAGE_FLOATS;
    const float* w_s = a_s + T::ROWS * STAGE_K;
#pragma unroll 4
    for (int k = 0; k < STAGE_K; k += 4) {
      float4 w[MANY_TN];
#pragma unroll
      for (int j = 0; j < MANY_TN; ++j) w[j] = swizzled(w_s, tn + 16 * j, k);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float4 a = swizzled(a_s, tm + 8 * i, k);
#pragma unroll
        for (int j = 0; j < MANY_TN; ++j) acc[i][j] = fmaf(a.x, w[j].x, acc[i][j]);
#pragma unroll
        for (int j = 0; j < MANY_TN; ++j) acc[i][j] = fmaf(a.y, w[j].y, acc[i][j]);
#pragma unroll
        for (int j = 0; j < MANY_TN; ++j) acc[i][j] = fmaf(a.z, w[j].z, acc[i][j]);
#pragma unroll
        for (int j = 0; j < MANY_TN; ++j) acc[i][j] = fmaf(a.w, w[j].w, acc[i][j]);
      }
    }
    const bool last = s + 1 == stages;
    if ((s + 1) % per_range == 0 || last) {                    // a range of K ends
      const int range = first_group * GROUP + s / per_range;
      const bool first = range % GROUP == 0, ends = range % GROUP == GROUP - 1 || last, add = !partials && range >= GROUP;
      float* out = partials ? partials + (size_t)(range / GROUP) * M * N : C;
      const long ld = partials ? N : ldc;
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const int row = m0 + tm + 8 * i;
#pragma unroll
        for (int j = 0; j < MANY_TN; ++j) {
          group[i][j] = first ? acc[i][j] : group[i][j] + acc[i][j];
          acc[i][j] = 0.f;
          const int col = n0 + tn + 16 * j;
          if (ends && row < M && col < N) {
            float* at = out + (long)row * ld + col;
            *at = add ? *at + group[i][j] : group[i][j];
          }
        }
      }
    }
  }
  if (!ok) {
    if (threadIdx.x == 0) atomicCAS(&g_gemm_simt_error, 0, 2);
    let_copies_land();
  }
}

// C = the groups' sums, added in their order.
__global__ void __launch_bounds__(256)
sum_groups_kernel(const float* __restrict__ partials, float* __restrict__ C, int groups, int M, int N, long ldc) {
  pdl_launch_dependents();
  pdl_wait();
  const long size = (long)M * N;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < size; i += (long)gridDim.x * blockDim.x) {
    float part[8];
#pragma unroll
    for (int g = 0; g < 8; ++g) part[g] = g < groups ? partials[g * size + i] : 0.f;
    float total = part[0];
#pragma unroll
    for (int g = 1; g < 8; ++g)
      if (g < groups) total += part[g];
    C[i / N * ldc + i % N] = total;
  }
}

// rows x K floats with row stride `ld`; box = 32 (K) x box_rows, zero fill beyond the matrix.
bool make_map_f32(CUtensorMap* map, const void* base, long rows, long K, long ld, int box_rows, bool swizzle) {
  auto encode = encode_fn();
  if (!encode) return false;
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t box[2] = {(cuuint32_t)STAGE_K, (cuuint32_t)box_rows};
  cuuint32_t elem[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A product of 32-bit operands; `partials` as the kernels take it.
struct Product {
  const void *A, *W;
  float *C, *partials;
  int M, N, K;
  long lda, ldw, ldc;
  int sm_count;
  bool early_weights;
  cudaStream_t stream;
  bool tma() const {      // 16-byte aligned addresses and row strides
    return (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0 && lda % 4 == 0 && ldw % 4 == 0 && lda >= K && ldw >= K;
  }
  bool streams() const;   // whether the streaming kernels take it
  long scratch() const;   // floats for the ranges' sums in their form of it
};

int sum_groups(const Product& p) {
  const long blocks = ((long)p.M * p.N + 255) / 256;
  lb_launch(sum_groups_kernel, dim3((unsigned)(blocks < 4096 ? blocks : 4096)), dim3(256), 0, p.stream, (const float*)p.partials, p.C,
            Split(p.K).groups(), p.M, p.N, p.ldc);
  return lb_last_error();
}

template <int TOKENS>
int launch_few(const Product& p) {
  using F = Few<TOKENS>;
  static LbPerDeviceOnce configured;
  auto kernel = gemm_f32_few_kernel<TOKENS>;
  if (!configured.run(LB_ALLOW_SMEM(kernel, F::SMEM))) return lb_last_error();
  CUtensorMap map_w, map_a;
  if (!make_map_f32(&map_w, p.W, p.N, p.K, p.ldw, FEW_ROWS, true) || !make_map_f32(&map_a, p.A, p.M, p.K, p.lda, TOKENS, false))
    return LB_ERR_ALIGN;
  const dim3 grid((p.N + FEW_ROWS - 1) / FEW_ROWS, 1, Split(p.K).groups()), block(32 * F::WARPS);
  if (!p.partials) {
    lb_launch_cluster(gemm_f32_few_kernel<TOKENS>, grid, block, (size_t)F::SMEM, p.stream, grid.z, map_w, map_a, p.C, p.partials, p.M,
                      p.N, p.K, p.ldc, p.early_weights);
    return lb_last_error();
  }
  lb_launch(gemm_f32_few_kernel<TOKENS>, grid, block, (size_t)F::SMEM, p.stream, map_w, map_a, p.C, p.partials, p.M, p.N, p.K, p.ldc,
            p.early_weights);
  return sum_groups(p);
}

// Tokens of a tile: 64 unless that leaves over a fifth more rows empty than tiles of 32 do, which reads the weights' tile
// twice as often.
bool wide_tiles(int M) { return (M + 63) / 64 * 64 * 5 <= (M + 31) / 32 * 32 * 6; }

// How many blocks share a tile's groups of ranges: as many as give every SM five rounds of its three blocks. With half of
// that 261 tokens take 2.08 ms a layer, with a quarter 2.29, with this 2.01; the groups' way through the L2 costs less
// than a last round that leaves SMs idle.
int many_parts(int M, int N, int K, int sm_count) {
  const int rows = wide_tiles(M) ? 64 : 32, groups = Split(K).groups();
  const long tiles = (long)((M + rows - 1) / rows) * ((N + MANY_COLS - 1) / MANY_COLS), wanted = 16L * sm_count;
  const long parts = (wanted + tiles - 1) / tiles;
  return parts < groups ? (int)parts : groups;
}

constexpr long SCRATCH_FLOATS = 64L << 20;       // the most that the ranges' sums may take (256 MiB); beyond, a block walks all of K

long Product::scratch() const {
  const long floats = (long)Split(K).groups() * M * N;
  if (M <= FT_M) return lb_cluster_reduce_enabled() ? 0 : floats;
  return many_parts(M, N, K, sm_count) > 1 && floats <= SCRATCH_FLOATS ? floats : 0;
}

// Short products are the plain tiles': the streaming kernels' rings and clusters take 2.8 us (2 tokens) to 5.6 us (16) before they
// bring anything, where the plain few-token kernel takes 1.6 us and as long again for every 2,560 x 64 weights. Where both take as
// long (us, plain and streaming): 2 tokens, 1,024 x 128 2.6 and 3.4, 2,560 x 96 3.2 and 3.4, 9,728 x 32 3.0 and 3.7; 4 tokens,
// 1,024 x 512 7.1 and 7.4, 2,560 x 256 5.9 and 5.4; 8 tokens, 1,024 x 1,024 13.1 and 16.9, 2,560 x 512 10.4 and 11.0, 9,728 x 128
// 8.4 and 7.4. Beyond 16 tokens the streaming kernel is ahead from one stage on (2,560 x 32, 32 tokens: 3.8 and 2.8).
bool Product::streams() const {
  if (!tma()) return false;
  if (M > FT_M) return K >= STAGE_K;
  const long limit = M <= 2 ? 1L << 17 : (M <= 4 ? 1L << 19 : 1L << 20);
  return (long)K * (N > 1024 ? N : 1024) > limit;
}

template <int TM>
int launch_many(const Product& p) {
  using T = Many<TM>;
  static LbPerDeviceOnce configured;
  auto kernel = gemm_f32_many_kernel<TM>;
  if (!configured.run(LB_ALLOW_SMEM(kernel, T::SMEM))) return lb_last_error();
  CUtensorMap map_w, map_a;
  if (!make_map_f32(&map_w, p.W, p.N, p.K, p.ldw, MANY_COLS, true) || !make_map_f32(&map_a, p.A, p.M, p.K, p.lda, T::ROWS, true))
    return LB_ERR_ALIGN;
  const long tiles = (long)((p.M + T::ROWS - 1) / T::ROWS) * ((p.N + MANY_COLS - 1) / MANY_COLS);
  if (tiles > 0x7fffffffL) return LB_ERR_SIZE;
  const dim3 grid((unsigned)tiles, 1, p.partials ? many_parts(p.M, p.N, p.K, p.sm_count) : 1);
  lb_launch(gemm_f32_many_kernel<TM>, grid, dim3(MANY_THREADS), (size_t)T::SMEM, p.stream, map_w, map_a, p.C, p.partials, p.M, p.N, p.K,
            p.ldc);
  return p.partials ? sum_groups(p) : lb_last_error();
}
}  // namespace

// Where this library's error word lies, its value (which is cleared), as the other libraries with bounded waits offer them.
LB_EXPORT void* lb_gemm_simt_status_address() {
  void* address = nullptr;
  if (cudaGetSymbolAddress(&address, g_gemm_simt_error) != cudaSuccess) { cudaGetLastError(); return nullptr; }
  return address;
}
LB_EXPORT int lb_gemm_simt_status() {
  int code = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&code, g_gemm_simt_error, sizeof(int)) != cudaSuccess) return -100;
  if (code) cudaMemcpyToSymbol(g_gemm_simt_error, &zero, sizeof(int));
  return code;
}

// Floats of scratch that a product of 32-bit operands wants for the ranges' sums in the form that it will take (0: none, one
// launch; else a second one adds them up).
LB_EXPORT long lb_gemm_simt_scratch(const void* A, const void* W, int M, int N, int K, long lda, long ldw, int sm_count) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  const Product p{A, W, nullptr, nullptr, M, N, K, lda, ldw, N, sm_count < 1 ? 1 : sm_count, false, nullptr};
  return p.streams() ? p.scratch() : 0;
}

// in_dtype: type of A and W; out_dtype: type of C (bf16 inputs may write 32-bit floats). `scratch`: null, or as many floats as
// `lb_gemm_simt_scratch` says, used by this call alone. `early_weights`: no kernel that may still run when this one is launched
// writes W, which is then read before that kernel has ended.
LB_EXPORT int lb_gemm_simt(int in_dtype, int out_dtype, const void* A, const void* W, void* C, int M, int N, int K,
                           long lda, long ldw, long ldc, float* scratch, int sm_count, int early_weights, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return LB_ERR_SIZE;
  if (in_dtype == LB_F32 && out_dtype == LB_F32) {
    const Product p{A, W, (float*)C, scratch, M, N, K, lda, ldw, ldc, sm_count < 1 ? 1 : sm_count, early_weights != 0, stream};
    if (p.streams() && (scratch || M > FT_M || !p.scratch())) {
      if (M <= 2) return launch_few<2>(p);
      if (M <= 4) return launch_few<4>(p);
      if (M <= 8) return launch_few<8>(p);
      if (M <= FT_M) return launch_few<16>(p);
      return wide_tiles(M) ? launch_many<8>(p) : launch_many<4>(p);
    }
  }
  if (M <= FT_M) {
    dim3 few((N + FT_N - 1) / FT_N, 1);
    if (in_dtype == LB_F32 && out_dtype == LB_F32)
      lb_launch(gemm_f32_plain_few_kernel, few, FT_THREADS, 0, stream, (const float*)A, (const float*)W, (float*)C, M, N, K, lda, ldw, ldc);
    else if (in_dtype == LB_BF16 && out_dtype == LB_BF16)
      lb_launch(gemm_simt_fewtoken_kernel<bf16, bf16>, few, FT_THREADS, 0, stream, (const bf16*)A, (const bf16*)W, (bf16*)C, M, N,
                K, lda, ldw, ldc, vec_ok<bf16>(A, lda), vec_ok<bf16>(W, ldw));
    else if (in_dtype == LB_BF16 && out_dtype == LB_F32)
      lb_launch(gemm_simt_fewtoken_kernel<bf16, float>, few, FT_THREADS, 0, stream, (const bf16*)A, (const bf16*)W, (float*)C, M,
                N, K, lda, ldw, ldc, vec_ok<bf16>(A, lda), vec_ok<bf16>(W, ldw));
    else
      return LB_ERR_DTYPE;
    return lb_last_error();
  }
  dim3 grid((N + TILE_N - 1) / TILE_N, (M + TILE_M - 1) / TILE_M);
  if (grid.y > 65535) return LB_ERR_SIZE;
  if (in_dtype == LB_F32 && out_dtype == LB_F32)
    lb_launch(gemm_simt_kernel<float, float, true>, grid, THREADS, 0, stream, (const float*)A, (const float*)W, (float*)C, M, N, K,
                                                                 lda, ldw, ldc, vec_ok<float>(A, lda),
                                                                 vec_ok<float>(W, ldw), Split(K).length);
  else if (in_dtype == LB_BF16 && out_dtype == LB_BF16)
    lb_launch(gemm_simt_kernel<bf16, bf16>, grid, THREADS, 0, stream, (const bf16*)A, (const bf16*)W, (bf16*)C, M, N, K, lda,
                                                               ldw, ldc, vec_ok<bf16>(A, lda), vec_ok<bf16>(W, ldw), 0);
  else if (in_dtype == LB_BF16 && out_dtype == LB_F32)
    lb_launch(gemm_simt_kernel<bf16, float>, grid, THREADS, 0, stream, (const bf16*)A, (const bf16*)W, (float*)C, M, N, K,
                                                                lda, ldw, ldc, vec_ok<bf16>(A, lda),
                                                                vec_ok<bf16>(W, ldw), 0);
  else
    return LB_ERR_DTYPE;
  return lb_last_error();
}
