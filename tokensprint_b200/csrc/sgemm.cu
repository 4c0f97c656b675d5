// True float32 matrix product on CUDA cores: C[M, N] = A[M, K] * W[N, K]^T.
//
// This is the float32 path's GEMM: FFMA only, no tensor cores and no reduced-precision
// mode.  Each output element is the sum of four chains of fused multiply-adds, (s0 + s1) + (s2 + s3):
// chain i takes the runs of 16 along k whose number is i modulo 4, in increasing order.  Both kernels
// below and all their tiles do exactly that, so a row's result does not depend on which other rows
// share the launch, nor on the size of the step.
// W is row-major [out, in] as the reference's Linear weights are (engine/nn/attention.py:
// 122-135).
//
// Two kernels.  The tiled one: four groups of warps, one per chain, work on the same 64 x 64 (or
// 32 x 32) outputs, each on its own run of 16 of every 64 along k; the runs come by 16-byte cp.async
// into two buffers in the layout they have in memory, rows 20 floats apart, so that the eight rows a
// warp reads at once meet no bank twice; a thread holds 8 x 8 (4 x 4) sums.  The four groups are there
// because a layer's product of a few hundred rows has too few tiles to keep the schedulers busy: with one chain
// a tile (64 x 64, 64 threads) 1.3 warps stood on a scheduler and issued an instruction every 3.4 cycles.
// The other kernel is for steps of up to 16 rows, which are bound by reading W once: 16 or 32 rows of W
// and all of A pass through a ring of four slices of 64 along k, a thread owns one row of W and a few of A.
// Measured (B200, 333 rows; before: 64 x 64 tiles, 4 x 4 sums a thread, loads a word at a time and nothing in
// flight, 270 to 400 us a product of this size): N x K = 4,096 x 1,024 104 us (27 TFLOP/s), 6,144 x 1,024 134 us,
// 1,024 x 3,072 177 us (96 tiles); 512 rows of 8,192 x 2,048 450 us (38 TFLOP/s: one wavefront of shared memory
// per value and warp holds it at about half of the FFMA rate); 64 rows of 4,096 x 2,048 41 us.
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
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
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
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
    }
  }
  __syncthreads();
  float* sums = sm + chain * BM * (BN + 1);
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) sums[(ty + i * TY) * (BN + 1) + tx + j * TX] = acc[i][j];
  __syncthreads();
  for (int i = threadIdx.x; i < BM * BN; i += THREADS) {
    const int r = i / BN, c = i % BN;
    if (m0 + r >= p.M || n0 + c >= p.N) continue;
    const float* s = sm + r * (BN + 1) + c;
    C[(size_t)(m0 + r) * p.ldc + n0 + c] = (s[0] + s[BM * (BN + 1)]) + (s[2 * BM * (BN + 1)] + s[3 * BM * (BN + 1)]);
  }
}

// ---- up to 16 rows ----

constexpr int FEW_ROWS = 16, FK = 64, FSTAGES = 4, FSTRIDE = FK + 4;  // rows of FK + 4 floats: 16-byte reads of 8 neighbour rows meet no bank twice

// 128 threads; BN rows of W; thread (n, g) has the output row n and the rows g, g + G, ... of A (G = 128 / BN).
template <int BN>
__global__ void __launch_bounds__(128) sgemm_few_rows_kernel(const Product p) {
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
  float acc[CHAINS][RM];
#pragma unroll
  for (int c = 0; c < CHAINS; ++c)
#pragma unroll
    for (int i = 0; i < RM; ++i) acc[c][i] = 0.f;
  for (int s = 0; s < slices; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(FSTAGES - 2) : "memory");
    __syncthreads();  // slice s is here for everybody, and slice s - 1 has been read
    if (s + FSTAGES - 1 < slices) fetch_w(s + FSTAGES - 1), fetch_a(s + FSTAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* ws = sm + (s % FSTAGES) * STAGE + n * FSTRIDE;
    const float* as = sm + (s % FSTAGES) * STAGE + BN * FSTRIDE;
#pragma unroll
    for (int k = 0; k < RUN; k += 4) {
#pragma unroll
      for (int c = 0; c < CHAINS; ++c) {
        const float4 w = *reinterpret_cast<const float4*>(ws + c * RUN + k);
#pragma unroll
        for (int i = 0; i < RM; ++i) {
          if (g + i * G < p.M) {
            const float4 a = *reinterpret_cast<const float4*>(as + (g + i * G) * FSTRIDE + c * RUN + k);
            acc[c][i] = fmaf(a.x, w.x, acc[c][i]);
            acc[c][i] = fmaf(a.y, w.y, acc[c][i]);
            acc[c][i] = fmaf(a.z, w.z, acc[c][i]);
            acc[c][i] = fmaf(a.w, w.w, acc[c][i]);
          }
        }
      }
    }
  }
  if (n0 + n < p.N) {
#pragma unroll
    for (int i = 0; i < RM; ++i)
      if (g + i * G < p.M) C[(size_t)(g + i * G) * p.ldc + n0 + n] = (acc[0][i] + acc[1][i]) + (acc[2][i] + acc[3][i]);
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

template <int BN>
int launch_few_rows(const Product& p, int batch, cudaStream_t s) {
  constexpr size_t smem = (size_t)FSTAGES * (BN + FEW_ROWS) * FSTRIDE * sizeof(float);
  if (batch > 65535) return TS_ERR_UNSUPPORTED_SIZE;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(sgemm_few_rows_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  return ts_launch(sgemm_few_rows_kernel<BN>, dim3((p.N + BN - 1) / BN, 1, batch), dim3(128), smem, s, p);
}

bool aligned16(const Product& p) {
  const long long strides = p.lda | p.ldw | p.batch_a | p.batch_w;
  return ((reinterpret_cast<size_t>(p.A) | reinterpret_cast<size_t>(p.W)) & 15) == 0 && (strides & 3) == 0;
}

// Which kernel: the choice changes the time only, never a bit of the result.  Small tiles where the
// large ones would leave half of the SMs without one.
int launch(const Product& p, int batch, cudaStream_t s) {
  const bool vec = aligned16(p) && p.K % 4 == 0;
  if (p.M <= FEW_ROWS && vec)
    return (long long)batch * ((p.N + 31) / 32) >= 148 ? launch_few_rows<32>(p, batch, s) : launch_few_rows<16>(p, batch, s);
  const long long tiles = (long long)batch * ((p.M + 63) / 64) * ((p.N + 63) / 64);
  if (tiles >= 80) return vec ? launch_tiles<64, 64, 8, 8, true>(p, batch, s) : launch_tiles<64, 64, 8, 8, false>(p, batch, s);
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
