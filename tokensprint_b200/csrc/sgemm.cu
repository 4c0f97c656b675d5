// True float32 matrix product on CUDA cores: C[M, N] = A[M, K] * W[N, K]^T.
//
// This is the float32 path's GEMM: FFMA only, no tensor cores and no reduced-precision
// mode.  Each output element is the sum of eight chains of fused multiply-adds: chain i of four takes the runs of 16 along k
// whose number is i modulo 4, in increasing order, its even and its odd k apart (the packed instruction multiplies two
// neighbours along k at once, as they lie in memory), and the element is (s0 + s1) + (s2 + s3) with s_i = even + odd.
// All kernels below and all their tiles do exactly that, so a row's result does not depend on which other rows
// share the launch, nor on the size of the step.
// W is row-major [out, in] as the reference's Linear weights are (engine/nn/attention.py:
// 122-135).
//
// Three kernels.  The wide one, where its tiles fill the chip: 32 x 128 outputs, see there; it multiplies in packed pairs, since scalar FFMA with
// three different registers issues 2.6 times a cycle and SM on B200, the packed one 1.9 times with twice the work (83 against
// 124 products a cycle).  The small tiles: four groups of warps, one per chain, work on the same 32 x 32 outputs, each on its own
// run of 16 of every 64 along k; the runs come by 16-byte cp.async into two buffers in the layout they have in memory, rows 20 floats apart, so that the
// eight rows a warp reads at once meet no bank twice; a thread holds 4 x 4 pairs of sums.  The third kernel is for steps of up to 16 rows, which are
// bound by reading W once: 16 or 32 rows of W and all of A pass through a ring of four slices of 64 along k, a thread owns
// one row of W and a few of A.  These two are bound by the latency of their chains, not by issue: packed pairs, in the same order, made them
// slower (100 rows of 2,048 x 2,048 45 us, scalar 40; 1 row of 6,144 x 1,024 27 and 12, of 151,936 x 1,024 259 and 105).
// Measured (B200, us; before: four chains, 64 x 64 scalar tiles): 333 rows, N x K = 4,096 x 1,024 104 -> 93, 6,144 x 1,024 134 -> 124, 1,024 x 2,048
// 86 -> 63, 1,024 x 3,072 127 -> 90; 512 rows of 8,192 x 2,048 450 -> 407 (42 TFLOP/s); 64 rows of 6,144 x 1,024 45 -> 34; 1 / 8 / 16 rows of
// 6,144 x 1,024 19 / 21 / 24 -> 12 / 20 / 25, of 151,936 x 1,024 189 / 217 / 254 -> 105 / 202 / 266.
#include "common.cuh"

namespace {

struct Product {
  const float* A;
  const float* W;
  float* C;
  int M, N, K;
  long long lda, ldw, ldc, batch_a, batch_w, batch_c;
};

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool real) {
  const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = real ? 16 : 0;  // 0: the piece is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(bytes));
}

__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool real) {
  const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = real ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to), "l"(src), "r"(bytes));
}

// Two products at once: (x, y) += (a.x b.x, a.y b.y), each rounded as fmaf rounds it.
typedef unsigned long long Pair;
__device__ __forceinline__ void fma_pair(Pair& acc, Pair a, Pair b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ float pair_sum(Pair v) { return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32)); }

constexpr int CHAINS = 4, RUN = 16, RSTRIDE = RUN + 4;

template <int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__(CHAINS * (BM / TM) * (BN / TN), 2) sgemm_tile_kernel(const Product p) {
  ts_pdl_prologue();
  constexpr int TX = BN / TN, TY = BM / TM, GROUP = TX * TY, THREADS = CHAINS * GROUP, ROWS = BM + BN, STAGE = CHAINS * ROWS * RSTRIDE;
  static_assert(GROUP % 32 == 0 && 2 * STAGE >= CHAINS * BM * (BN + 1), "a chain is whole warps; the sums fit where the runs were");
  extern __shared__ __align__(16) float sm[];  // [2][CHAINS][ROWS][RSTRIDE]
  const float* __restrict__ A = p.A + (size_t)blockIdx.z * p.batch_a;  // product blockIdx.z of a batch of equal shapes
  const float* __restrict__ W = p.W + (size_t)blockIdx.z * p.batch_w;
  float* __restrict__ C = p.C + (size_t)blockIdx.z * p.batch_c;
  const int chain = threadIdx.x / GROUP, tid = threadIdx.x % GROUP, tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  // piece j of a thread: 16 bytes of row tid / 4 + j * (GROUP / 4) of the tile's rows (A's first, then W's)
  auto fetch = [&](int run, int s) {
    float* to = sm + s * STAGE + chain * ROWS * RSTRIDE;
    const int c = run * RUN + (tid & 3) * 4;
#pragma unroll
    for (int j = 0; j < ROWS / (GROUP / 4); ++j) {
      const int r = (tid >> 2) + j * (GROUP / 4);
      const bool of_a = r < BM;
      const int row = of_a ? m0 + r : n0 + r - BM;
      const bool there = row < (of_a ? p.M : p.N);
      const float* src = of_a ? A + (size_t)row * p.lda + c : W + (size_t)row * p.ldw + c;
      float* dst = to + r * RSTRIDE + (tid & 3) * 4;
      if (VEC) {  // K is a multiple of 4: a piece lies inside the row or behind it
        const bool real = there && c < p.K;
        cp_async16(dst, real ? src : p.W, real);
      } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[i] = there && c + i < p.K ? src[i] : 0.f;
      }
    }
    if (VEC) asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float2 acc[TM][TN];  // the sums over the even and over the odd k of the chain
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
  const int rounds = (p.K + CHAINS * RUN - 1) / (CHAINS * RUN);
  fetch(chain, 0);
  for (int it = 0; it < rounds; ++it) {
    if (VEC) asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // the round's runs are here, and the round before has been read
    if (it + 1 < rounds) fetch((it + 1) * CHAINS + chain, (it + 1) & 1);
    const float* as = sm + (it & 1) * STAGE + chain * ROWS * RSTRIDE + ty * RSTRIDE;
    const float* ws = sm + (it & 1) * STAGE + chain * ROWS * RSTRIDE + (BM + tx) * RSTRIDE;
#pragma unroll
    for (int k = 0; k < RUN; k += 2) {
      float2 a[TM], b[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float2*>(as + i * TY * RSTRIDE + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float2*>(ws + j * TX * RSTRIDE + k);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j].x = fmaf(a[i].x, b[j].x, acc[i][j].x);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j].y = fmaf(a[i].y, b[j].y, acc[i][j].y);
    }
  }
  __syncthreads();
  float* sums = sm + chain * BM * (BN + 1);
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sums[(ty + i * TY) * (BN + 1) + tx + j * TX] = acc[i][j].x + acc[i][j].y;
  __syncthreads();
  for (int i = threadIdx.x; i < BM * BN; i += THREADS) {
    const int r = i / BN, c = i % BN;
    if (m0 + r >= p.M || n0 + c >= p.N) continue;
    const float* s = sm + r * (BN + 1) + c;
    C[(size_t)(m0 + r) * p.ldc + n0 + c] = (s[0] + s[BM * (BN + 1)]) + (s[2 * BM * (BN + 1)] + s[3 * BM * (BN + 1)]);
  }
}

// ---- many tiles: 32 x 128 outputs, a warp 16 rows x 128 columns ----

constexpr int WM = 32, WN = 128, WROWS = WM + WN, WCHAIN = WROWS * RSTRIDE, WSTAGE = CHAINS * WCHAIN, WSTAGES = 3, W_RM = 16, W_RN = 4;

// Two warps a chain, 16 of the tile's rows each; a lane has the columns lane, lane + 32, .. + 96.  The 16 values of A that a warp
// multiplies are the same for all its lanes, and 16 bytes of them cost a third of what 16 different bytes a lane cost (1.4 against 0.46
// such reads a cycle).  The chains wait for their own copies only (a named barrier of two warps).  What is left is latency at two
// warps a scheduler; four warps a chain with 8 rows each: 64 -> 65 us, the loop over k unrolled: 64 -> 67.
template <bool VEC>
__global__ void __launch_bounds__(CHAINS * 32 * (WM / W_RM), 1) sgemm_wide_kernel(const Product p) {
  constexpr int GROUP = 32 * (WM / W_RM), STEP = GROUP / 4;  // threads of a chain; rows they copy at once
  ts_pdl_prologue();
  extern __shared__ __align__(16) float sm[];  // [WSTAGES][CHAINS][WROWS][RSTRIDE], then the sums [CHAINS][WM][WN + 1]
  const float* __restrict__ A = p.A + (size_t)blockIdx.z * p.batch_a;
  const float* __restrict__ W = p.W + (size_t)blockIdx.z * p.batch_w;
  float* __restrict__ C = p.C + (size_t)blockIdx.z * p.batch_c;
  const int chain = threadIdx.x / GROUP, tid = threadIdx.x % GROUP, part = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * WM, n0 = blockIdx.x * WN;
  // a thread copies 16 bytes of every 16th row: two of A, eight of W
  const int row = tid >> 2, col = (tid & 3) * 4;
  const float* a_src = A + (size_t)(m0 + row) * p.lda + col;
  const float* w_src = W + (size_t)(n0 + row) * p.ldw + col;
  float* dst = sm + chain * WCHAIN + row * RSTRIDE + col;
  auto fetch_w = [&](int round) {
    const int k = (round * CHAINS + chain) * RUN;
    const bool in = k + col < p.K;  // K is a multiple of 4: a piece lies inside the row or behind it
#pragma unroll
    for (int j = 0; j < WN / STEP; ++j) {
      const bool real = in && n0 + row + j * STEP < p.N;
      cp_async16(dst + round % WSTAGES * WSTAGE + (WM + j * STEP) * RSTRIDE, real ? w_src + (size_t)j * STEP * p.ldw + k : p.W, real);
    }
  };
  auto fetch_a = [&](int round) {
    const int k = (round * CHAINS + chain) * RUN;
#pragma unroll
    for (int j = 0; j < WM / STEP; ++j) {
      const bool real = k + col < p.K && m0 + row + j * STEP < p.M;
      cp_async16(dst + round % WSTAGES * WSTAGE + j * STEP * RSTRIDE, real ? a_src + (size_t)j * STEP * p.lda + k : p.A, real);
    }
  };
  // rows of any address and length: a word at a time (512 rows of 6,144 x 1,025: 257 us, with words through registers in small tiles 369)
  auto fetch_words = [&](int round) {
    const int k = (round * CHAINS + chain) * RUN;
    float* to = dst + round % WSTAGES * WSTAGE;
    auto piece = [&](int r, const float* src, bool there) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const bool real = there && k + col + i < p.K;
        cp_async4(to + r * RSTRIDE + i, real ? src + k + i : p.W, real);
      }
    };
#pragma unroll
    for (int j = 0; j < WN / STEP; ++j) piece(WM + j * STEP, w_src + (size_t)j * STEP * p.ldw, n0 + row + j * STEP < p.N);
#pragma unroll
    for (int j = 0; j < WM / STEP; ++j) piece(j * STEP, a_src + (size_t)j * STEP * p.lda, m0 + row + j * STEP < p.M);
  };
  auto fetch = [&](int round) {
    if constexpr (VEC) {
      fetch_w(round);
      fetch_a(round);
    } else {
      fetch_words(round);
    }
  };
  Pair acc[W_RM][W_RN];
#pragma unroll
  for (int i = 0; i < W_RM; ++i)
#pragma unroll
    for (int j = 0; j < W_RN; ++j) acc[i][j] = 0;
  const int rounds = (p.K + CHAINS * RUN - 1) / (CHAINS * RUN);
#pragma unroll
  for (int r = 0; r < WSTAGES - 1; ++r) {
    if (r < rounds) fetch(r);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int it = 0; it < rounds; ++it) {
    asm volatile("cp.async.wait_group %0;" ::"n"(WSTAGES - 2) : "memory");
    asm volatile("bar.sync %0, %1;" ::"r"(1 + chain), "n"(GROUP) : "memory");  // the chain's run is here, and the one before has been read
    if (it + WSTAGES - 1 < rounds) fetch(it + WSTAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* as = sm + it % WSTAGES * WSTAGE + chain * WCHAIN + part * W_RM * RSTRIDE;
    const float* ws = sm + it % WSTAGES * WSTAGE + chain * WCHAIN + (WM + lane) * RSTRIDE;
#pragma unroll 1
    for (int k = 0; k < RUN; k += 4) {
      ulonglong2 b[W_RN];
#pragma unroll
      for (int j = 0; j < W_RN; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(ws + j * 32 * RSTRIDE + k);
#pragma unroll
      for (int i = 0; i < W_RM; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(as + i * RSTRIDE + k);
#pragma unroll
        for (int j = 0; j < W_RN; ++j) fma_pair(acc[i][j], a.x, b[j].x);
#pragma unroll
        for (int j = 0; j < W_RN; ++j) fma_pair(acc[i][j], a.y, b[j].y);
      }
    }
  }
  __syncthreads();
  constexpr int PLANE = WM * (WN + 1);
  static_assert(CHAINS * PLANE <= WSTAGES * WSTAGE, "the sums fit where the runs were");
#pragma unroll
  for (int i = 0; i < W_RM; ++i)
#pragma unroll
    for (int j = 0; j < W_RN; ++j) sm[chain * PLANE + (part * W_RM + i) * (WN + 1) + lane + j * 32] = pair_sum(acc[i][j]);
  __syncthreads();
  for (int i = threadIdx.x; i < WM * WN; i += CHAINS * GROUP) {
    const int r = i / WN, c = i % WN;
    if (m0 + r >= p.M || n0 + c >= p.N) continue;
    const float* q = sm + r * (WN + 1) + c;
    C[(size_t)(m0 + r) * p.ldc + n0 + c] = (q[0] + q[PLANE]) + (q[2 * PLANE] + q[3 * PLANE]);
  }
}

// ---- up to 16 rows ----

constexpr int FEW_ROWS = 16, FK = 64, FSTAGES = 4, FSTRIDE = FK + 4;  // rows of FK + 4 floats: 16-byte reads of 8 neighbour rows meet no bank twice

template <int R>
struct Rows {
  static constexpr int N = R;
};

// 128 threads; BN rows of W; thread (n, g) has the output row n and the rows g, g + G, ... of A (G = 128 / BN).
template <int BN, bool ALL_ROWS>
__global__ void __launch_bounds__(128, ALL_ROWS ? 1 : 4) sgemm_few_rows_kernel(const Product p) {
  constexpr int G = 128 / BN, RM = FEW_ROWS / G;
  extern __shared__ __align__(16) float sm[];  // FSTAGES x [BN + FEW_ROWS][FSTRIDE]
  constexpr int STAGE = (BN + FEW_ROWS) * FSTRIDE;
  const float* __restrict__ A = p.A + (size_t)blockIdx.z * p.batch_a;
  const float* __restrict__ W = p.W + (size_t)blockIdx.z * p.batch_w;
  float* __restrict__ C = p.C + (size_t)blockIdx.z * p.batch_c;
  const int n0 = blockIdx.x * BN, slices = (p.K + FK - 1) / FK;
  auto fetch_w = [&](int slice) {  // K is a multiple of 4 here: a piece lies inside the row or behind it
    float* to = sm + (slice % FSTAGES) * STAGE;
    for (int i = threadIdx.x; i < BN * (FK / 4); i += 128) {
      const int r = i / (FK / 4), c = slice * FK + (i % (FK / 4)) * 4;
      const bool real = n0 + r < p.N && c < p.K;
      cp_async16(to + r * FSTRIDE + (i % (FK / 4)) * 4, real ? W + (size_t)(n0 + r) * p.ldw + c : W, real);
    }
  };
  auto fetch_a = [&](int slice) {
    float* to = sm + (slice % FSTAGES) * STAGE + BN * FSTRIDE;
    for (int i = threadIdx.x; i < p.M * (FK / 4); i += 128) {
      const int r = i / (FK / 4), c = slice * FK + (i % (FK / 4)) * 4;
      const bool real = c < p.K;
      cp_async16(to + r * FSTRIDE + (i % (FK / 4)) * 4, real ? A + (size_t)r * p.lda + c : A, real);
    }
  };
  ts_pdl_prologue();
  for (int s = 0; s < FSTAGES - 1; ++s) {
    if (s < slices) fetch_w(s), fetch_a(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const int n = threadIdx.x % BN, g = threadIdx.x / BN;
  static_assert(FK == CHAINS * RUN, "a slice holds one run of every chain");
  float2 acc[CHAINS][RM];  // the sums over the even and over the odd k of each chain
#pragma unroll
  for (int c = 0; c < CHAINS; ++c)
#pragma unroll
    for (int i = 0; i < RM; ++i) acc[c][i] = make_float2(0.f, 0.f);
  // A slice's products with `count` of this thread's rows, from number `first` on.  A row at a time, its runs unrolled, unless the warp has all of its
  // rows: then a value of W is read once for them.  (All rows together behind a condition each: 30 against 22 us at 4 rows of 1,024 x 3,072.)
  auto multiply = [&](const float* ws, const float* as, int first, auto count) {
#pragma unroll
    for (int k = 0; k < RUN; k += 4) {
#pragma unroll
      for (int c = 0; c < CHAINS; ++c) {
        const float4 w = *reinterpret_cast<const float4*>(ws + c * RUN + k);
#pragma unroll
        for (int j = 0; j < decltype(count)::N; ++j) {
          const float4 a = *reinterpret_cast<const float4*>(as + (g + (first + j) * G) * FSTRIDE + c * RUN + k);
          float2& sum = acc[c][first + j];
          sum.x = fmaf(a.x, w.x, sum.x);
          sum.y = fmaf(a.y, w.y, sum.y);
          sum.x = fmaf(a.z, w.z, sum.x);
          sum.y = fmaf(a.w, w.w, sum.y);
        }
      }
    }
  };
  const int g0 = threadIdx.x / 32 * 32 / BN;  // the lowest g of this warp
  for (int s = 0; s < slices; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(FSTAGES - 2) : "memory");
    __syncthreads();  // slice s is here for everybody, and slice s - 1 has been read
    if (s + FSTAGES - 1 < slices) fetch_w(s + FSTAGES - 1), fetch_a(s + FSTAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* ws = sm + (s % FSTAGES) * STAGE + n * FSTRIDE;
    const float* as = sm + (s % FSTAGES) * STAGE + BN * FSTRIDE;
    if (ALL_ROWS || g0 + (RM - 1) * G < p.M) {
      multiply(ws, as, 0, Rows<RM>());
    } else {
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        if (g0 + i * G >= p.M) break;
        multiply(ws, as, i, Rows<1>());
      }
    }
  }
  if (n0 + n < p.N) {
#pragma unroll
    for (int i = 0; i < RM; ++i)
      if (g + i * G < p.M) {
        float v[CHAINS];
#pragma unroll
        for (int c = 0; c < CHAINS; ++c) v[c] = acc[c][i].x + acc[c][i].y;
        C[(size_t)(g + i * G) * p.ldc + n0 + n] = (v[0] + v[1]) + (v[2] + v[3]);
      }
  }
}

template <int BM, int BN, int TM, int TN, bool VEC>
int launch_tiles(const Product& p, int batch, cudaStream_t s) {
  const dim3 grid((p.N + BN - 1) / BN, (p.M + BM - 1) / BM, batch);
  if (grid.y > 65535 || batch > 65535) return TS_ERR_UNSUPPORTED_SIZE;
  constexpr size_t smem = (size_t)2 * CHAINS * (BM + BN) * RSTRIDE * sizeof(float);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(sgemm_tile_kernel<BM, BN, TM, TN, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  return ts_launch(sgemm_tile_kernel<BM, BN, TM, TN, VEC>, grid, dim3(CHAINS * (BM / TM) * (BN / TN)), smem, s, p);
}

template <bool VEC>
int launch_wide(const Product& p, int batch, cudaStream_t s) {
  const dim3 grid((p.N + WN - 1) / WN, (p.M + WM - 1) / WM, batch);
  if (grid.y > 65535 || batch > 65535) return TS_ERR_UNSUPPORTED_SIZE;
  constexpr size_t smem = (size_t)WSTAGES * WSTAGE * sizeof(float);
  const cudaError_t e = cudaFuncSetAttribute(sgemm_wide_kernel<VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  return ts_launch(sgemm_wide_kernel<VEC>, grid, dim3(CHAINS * 32 * (WM / W_RM)), smem, s, p);
}

template <int BN, bool ALL_ROWS>
int launch_few_rows(const Product& p, int batch, cudaStream_t s) {
  constexpr size_t smem = (size_t)FSTAGES * (BN + FEW_ROWS) * FSTRIDE * sizeof(float);
  if (batch > 65535) return TS_ERR_UNSUPPORTED_SIZE;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(sgemm_few_rows_kernel<BN, ALL_ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  return ts_launch(sgemm_few_rows_kernel<BN, ALL_ROWS>, dim3((p.N + BN - 1) / BN, 1, batch), dim3(128), smem, s, p);
}

bool aligned16(const Product& p) {
  const long long strides = p.lda | p.ldw | p.batch_a | p.batch_w;
  return ((reinterpret_cast<size_t>(p.A) | reinterpret_cast<size_t>(p.W)) & 15) == 0 && (strides & 3) == 0;
}

constexpr int MOST_ROWS = 65535 * 32;

// Which kernel: the choice changes the time only, never a bit of the result.
int launch(const Product& p, int batch, cudaStream_t s) {
  if (p.M > MOST_ROWS) {
    // Tiles have 32 rows and a grid 65,535 of them in this direction; twice as many rows are taken, in two launches.
    if (p.M > 2 * MOST_ROWS) return TS_ERR_UNSUPPORTED_SIZE;
    Product first = p, rest = p;
    first.M = MOST_ROWS;
    rest.M = p.M - MOST_ROWS;
    rest.A += (long long)MOST_ROWS * p.lda;
    rest.C += (long long)MOST_ROWS * p.ldc;
    const int status = launch(first, batch, s);
    return status != 0 ? status : launch(rest, batch, s);
  }
  const bool vec = aligned16(p) && p.K % 4 == 0;
  if (p.M <= FEW_ROWS && vec) {
    if ((long long)batch * ((p.N + 31) / 32) >= 148) return launch_few_rows<32, false>(p, batch, s);
    // above eight rows nearly every thread has both of its rows (13 rows of 2,048 x 8,192: 83 us, 90 with the conditions)
    return p.M > 8 ? launch_few_rows<16, true>(p, batch, s) : launch_few_rows<16, false>(p, batch, s);
  }
  // A round of wide tiles takes as long as 1.05 full rounds of small ones (two a SM), and more where it is one of several, since the
  // small tiles' last round is never as empty.  Small and wide tiles, us: 100 rows of 2,048 x 2,048 (256 small tiles, 64 wide) 40 : 65, 333 of
  // 1,024 x 2,048 (352, 88) 63 : 63, 128 of 4,096 x 1,024 (512, 128) 40 : 34; in two rounds of wide tiles, 333 of 2,048 x 2,048 (704, 176) 100 :
  // 105, 700 of 1,024 x 1,024 (704, 176) 56 : 56; in three, 333 of 4,096 x 1,024 (1,408, 352) 98 : 93.
  const long long wide = (long long)batch * ((p.M + WM - 1) / WM) * ((p.N + WN - 1) / WN);
  const long long small = (long long)batch * ((p.M + 31) / 32) * ((p.N + 31) / 32), rounds = (wide + 147) / 148;
  // Rows that the 16-byte copies do not take are read through registers by the small tiles, which costs them more: 333 rows of 2,048 x 2,050 208 :
  // 163, 128 of 6,144 x 1,025 (768, 192) 104 : 88.
  if (small * 100 >= 296 * rounds * (rounds == 1 || !vec ? 105 : 145)) return vec ? launch_wide<true>(p, batch, s) : launch_wide<false>(p, batch, s);
  return vec ? launch_tiles<32, 32, 4, 4, true>(p, batch, s) : launch_tiles<32, 32, 4, 4, false>(p, batch, s);
}

}  // namespace

TS_EXPORT int ts_sgemm_nt(const float* A, const float* W, float* C, int M, int N, int K,
                          long long lda, long long ldw, long long ldc, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || lda < K || ldw < K || ldc < N) return TS_ERR_BAD_ARGUMENT;
  return launch(Product{A, W, C, M, N, K, lda, ldw, ldc, 0LL, 0LL, 0LL}, 1, (cudaStream_t)stream);
}

// `batch` products of one shape: product b reads A + b * batch_a and W + b * batch_w and writes
// C + b * batch_c (elements); the rows of each may be strided (lda, ldw, ldc).
TS_EXPORT int ts_sgemm_nt_batched(const float* A, const float* W, float* C, int M, int N, int K, long long lda, long long ldw,
                                  long long ldc, int batch, long long batch_a, long long batch_w, long long batch_c, void* stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return 0;
  if (K <= 0 || lda < K || ldw < K || ldc < N) return TS_ERR_BAD_ARGUMENT;
  return launch(Product{A, W, C, M, N, K, lda, ldw, ldc, batch_a, batch_w, batch_c}, batch, (cudaStream_t)stream);
}
