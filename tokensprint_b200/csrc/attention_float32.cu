// Paged causal attention of the float32 path in tiles, on CUDA cores: the same function as
// attention_simple.cu (scale, window, blocks of positions, sinks, score cap, distance penalty; see
// there), for steps whose sequences are known by their cu_seqlens.
//
// One CTA per (sequence, KV head, 32 rows), a row being one (token, query head of the group) pair of
// the sequence, the heads of a token side by side.  Keys are taken 32 at a time, at multiples of 32 of
// the sequence's positions: K and V of a block are fetched once for all rows (16-byte cp.async, two
// blocks in flight), the scores come from shared memory (a thread has 2 rows x 4 keys), the online
// softmax runs over the 8 lanes that share a row, and the same threads add P V (2 rows x d / 8
// values).  Blocks start at multiples of 32 whatever the tile, so the order of the sums for one query
// depends only on its own keys, never on the batch around it nor on where its portion was cut.
// One warp per (token, head), as attention_simple.cu has it, re-reads every key row per query, four bytes
// a lane and rows apart: a prompt of 333 tokens, 16 heads of 128 on 8 KV heads, takes 636 us there and 84 here.
#include "common.cuh"

namespace {

constexpr int ROWS = 32, KEYS = 32, THREADS = 128;

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool real) {
  const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
  const int bytes = real ? 16 : 0;  // 0: the piece is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(src), "r"(bytes));
}

struct Args {
  const float *q, *k, *v;
  float* out;
  const int *cu, *lens, *table;
  int max_blocks, page, B, T, tiles, nq, nkv, d;
  float scale;
  int window, chunk, has_sink;
  float sink, softcap;
  const float *head_sinks, *r1, *r2;
};

// DP: the head size in shared memory, d rounded up to a power of two from 32 on (entries behind d are zeros)
template <int DP>
__global__ void __launch_bounds__(THREADS) attention_float32_kernel(const Args a) {
  ts_pdl_prologue();
  constexpr int KS = DP + 4;  // rows 16 bytes apart modulo 128: the 8 keys a warp reads at a time meet no bank twice
  extern __shared__ __align__(16) float sm[];
  float* Qs = sm;                       // [ROWS][DP], scaled
  float* Ks = Qs + ROWS * DP;           // [2][KEYS][KS]
  float* Vs = Ks + 2 * KEYS * KS;       // [2][KEYS][KS]
  float* Ps = Vs + 2 * KEYS * KS;       // [ROWS][KEYS + 1]
  const int b = blockIdx.x / a.tiles, tile = a.tiles - 1 - blockIdx.x % a.tiles;  // the longest rows of a sequence first
  const int hk = blockIdx.y, group = a.nq / a.nkv, d = a.d;
  const int t_begin = a.cu[b], n = a.cu[b + 1] - t_begin;
  if (blockIdx.x == 0) {  // padded lanes of a fixed-size batch: no sequence behind them, zeros
    for (int t = a.cu[a.B]; t < a.T; ++t)
      for (int i = threadIdx.x; i < group * d; i += THREADS) a.out[((size_t)t * a.nq + hk * group) * d + i] = 0.f;
  }
  const int row0 = tile * ROWS;
  if (row0 >= n * group) return;
  const int rows = min(ROWS, n * group - row0);
  const int p_base = a.lens[b] - n;  // position of the portion's first token
  const int p_first = p_base + row0 / group, p_last = p_base + (row0 + rows - 1) / group;
  auto first_key = [&](int p) {
    int lo = (a.window > 0 && p - a.window + 1 > 0) ? p - a.window + 1 : 0;
    return a.chunk > 0 ? max(lo, p / a.chunk * a.chunk) : lo;
  };
  const int key_lo = first_key(p_first);  // no row of the tile sees an earlier key (its page may have been given back)
  const int* table = a.table + (size_t)b * a.max_blocks;

  for (int i = threadIdx.x; i < ROWS * (DP / 4); i += THREADS) {
    const int r = i / (DP / 4), c = (i % (DP / 4)) * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows && c < d) {
      const int f = row0 + r;
      x = *reinterpret_cast<const float4*>(a.q + ((size_t)(t_begin + f / group) * a.nq + hk * group + f % group) * d + c);
    }
    *reinterpret_cast<float4*>(Qs + r * DP + c) = make_float4(x.x * a.scale, x.y * a.scale, x.z * a.scale, x.w * a.scale);
  }
  auto fetch = [&](int base, int s) {  // keys base .. base + 31 of the sequence into buffer s
    for (int i = threadIdx.x; i < KEYS * (DP / 4); i += THREADS) {
      const int r = i / (DP / 4), c = (i % (DP / 4)) * 4, j = base + r;
      const bool real = j >= key_lo && j <= p_last && c < d;
      const size_t at = real ? (((size_t)table[j / a.page] * a.page + j % a.page) * a.nkv + hk) * d + c : 0;
      cp_async16(Ks + (s * KEYS + r) * KS + c, a.k + at, real);
      cp_async16(Vs + (s * KEYS + r) * KS + c, a.v + at, real);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;  // rows 2 ty, 2 ty + 1; keys tx + 8 j; values 4 tx + 32 j
  int pos[2], lo[2], head[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int f = min(row0 + 2 * ty + i, row0 + rows - 1);
    pos[i] = p_base + f / group;
    lo[i] = first_key(pos[i]);
    head[i] = hk * group + f % group;
  }
  constexpr int NV = DP / 32;
  float4 acc[2][NV];
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NV; ++j) acc[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);

  int s = 0;
  const int base0 = key_lo / KEYS * KEYS;
  fetch(base0, 0);
  for (int base = base0; base <= p_last; base += KEYS, s ^= 1) {
    const bool more = base + KEYS <= p_last;
    if (more) fetch(base + KEYS, s ^ 1);
    if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const float* K = Ks + s * KEYS * KS;
    const float* V = Vs + s * KEYS * KS;
    float sc[2][4] = {};
#pragma unroll 4
    for (int c = 0; c < DP; c += 4) {
      const float4 q0 = *reinterpret_cast<const float4*>(Qs + (2 * ty) * DP + c), q1 = *reinterpret_cast<const float4*>(Qs + (2 * ty + 1) * DP + c);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 k = *reinterpret_cast<const float4*>(K + (tx + 8 * j) * KS + c);
        sc[0][j] = fmaf(q0.x, k.x, sc[0][j]), sc[1][j] = fmaf(q1.x, k.x, sc[1][j]);
        sc[0][j] = fmaf(q0.y, k.y, sc[0][j]), sc[1][j] = fmaf(q1.y, k.y, sc[1][j]);
        sc[0][j] = fmaf(q0.z, k.z, sc[0][j]), sc[1][j] = fmaf(q1.z, k.z, sc[1][j]);
        sc[0][j] = fmaf(q0.w, k.w, sc[0][j]), sc[1][j] = fmaf(q1.w, k.w, sc[1][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float top = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int key = base + tx + 8 * j;
        float x = sc[i][j];
        if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
        if (a.r1 != nullptr) x -= a.r1[head[i]] * log1pf(a.r2[head[i]] * (float)max(pos[i] - key, 0));
        sc[i][j] = key >= lo[i] && key <= pos[i] ? x : -INFINITY;
        top = fmaxf(top, sc[i][j]);
      }
      for (int o = 1; o < 8; o <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
      const float m_new = fmaxf(m[i], top), m_ref = m_new == -INFINITY ? 0.f : m_new;  // no key of the row so far: all weights are zero
      const float corr = expf(m[i] - m_ref);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float e = expf(sc[i][j] - m_ref);
        Ps[(2 * ty + i) * (KEYS + 1) + tx + 8 * j] = e;
        sum += e;
      }
      for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      l[i] = l[i] * corr + sum;
      m[i] = m_new;
#pragma unroll
      for (int j = 0; j < NV; ++j) acc[i][j].x *= corr, acc[i][j].y *= corr, acc[i][j].z *= corr, acc[i][j].w *= corr;
    }
    __syncwarp();  // the 8 lanes of a row sit in one warp
    const float* P0 = Ps + (2 * ty) * (KEYS + 1);
    const float* P1 = P0 + KEYS + 1;
    auto add = [&](int key, bool guard) {
      const float p0 = P0[key], p1 = P1[key];
#pragma unroll
      for (int j = 0; j < NV; ++j) {
        const float4 v = *reinterpret_cast<const float4*>(V + key * KS + 4 * tx + 32 * j);
        if (!guard || p0 != 0.f) {
          acc[0][j].x = fmaf(p0, v.x, acc[0][j].x), acc[0][j].y = fmaf(p0, v.y, acc[0][j].y);
          acc[0][j].z = fmaf(p0, v.z, acc[0][j].z), acc[0][j].w = fmaf(p0, v.w, acc[0][j].w);
        }
        if (!guard || p1 != 0.f) {
          acc[1][j].x = fmaf(p1, v.x, acc[1][j].x), acc[1][j].y = fmaf(p1, v.y, acc[1][j].y);
          acc[1][j].z = fmaf(p1, v.z, acc[1][j].z), acc[1][j].w = fmaf(p1, v.w, acc[1][j].w);
        }
      }
    };
    // where a row does not see the whole block, a value it does not see stays out whatever it is (an infinity, say)
    const bool whole = base + KEYS - 1 <= p_first && base >= first_key(p_last);
    if (whole) {
#pragma unroll 4
      for (int key = 0; key < KEYS; ++key) add(key, false);
    } else {
#pragma unroll 2
      for (int key = 0; key < KEYS; ++key) add(key, true);
    }
    __syncthreads();  // the block has been read
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = 2 * ty + i;
    if (r >= rows) continue;
    float corr = 1.f, denom = l[i];
    if (a.has_sink || a.head_sinks != nullptr) {  // the sink joins the denominator only
      const float sink = a.head_sinks != nullptr ? a.head_sinks[head[i]] : a.sink;
      const float m_new = fmaxf(m[i], sink);
      corr = expf(m[i] - m_new);
      denom = l[i] * corr + expf(sink - m_new);
    }
    const float inv = corr / denom;
    float* o = a.out + ((size_t)(t_begin + (row0 + r) / group) * a.nq + head[i]) * d;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int c = 4 * tx + 32 * j;
      if (c < d) *reinterpret_cast<float4*>(o + c) = make_float4(acc[i][j].x * inv, acc[i][j].y * inv, acc[i][j].z * inv, acc[i][j].w * inv);
    }
  }
}

template <int DP>
int launch(const Args& a, cudaStream_t s) {
  constexpr size_t smem = ((size_t)ROWS * DP + 4 * KEYS * (DP + 4) + ROWS * (KEYS + 1)) * sizeof(float);
  const cudaError_t e = cudaFuncSetAttribute(attention_float32_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  return ts_launch(attention_float32_kernel<DP>, dim3((unsigned)a.B * a.tiles, a.nkv), dim3(THREADS), smem, s, a);
}

}  // namespace

// Heads of 4 to 256 entries, a multiple of 4; q, k, v and out 16-byte aligned.
TS_EXPORT int ts_attention_paged_float32(const float* q, const float* k, const float* v, float* out, const int* cu_seqlens,
                                         const int* context_lens, const int* block_table, int max_blocks, int page, int B, int T, int max_q,
                                         int nq, int nkv, int d, float scale, int window, int chunk, int has_sink, float sink, float softcap,
                                         const float* head_sinks, const float* r1, const float* r2, void* stream) {
  if (B <= 0 || T <= 0 || max_q <= 0) return 0;
  if (nq <= 0 || nkv <= 0 || nq % nkv != 0 || d <= 0 || page <= 0 || max_blocks <= 0) return TS_ERR_BAD_ARGUMENT;
  if ((r1 == nullptr) != (r2 == nullptr)) return TS_ERR_BAD_ARGUMENT;
  if (d % 4 != 0 || d > 256 || nkv > 65535) return TS_ERR_UNSUPPORTED_SIZE;
  if ((reinterpret_cast<size_t>(q) | reinterpret_cast<size_t>(k) | reinterpret_cast<size_t>(v) | reinterpret_cast<size_t>(out)) & 15)
    return TS_ERR_BAD_ARGUMENT;
  const long long tiles = ((long long)max_q * (nq / nkv) + ROWS - 1) / ROWS;
  if (tiles * B > 0x7fffffffLL) return TS_ERR_UNSUPPORTED_SIZE;
  const Args a = {q, k, v, out, cu_seqlens, context_lens, block_table, max_blocks, page, B, T, (int)tiles, nq, nkv, d, scale,
                  window, chunk, has_sink, sink, softcap, head_sinks, r1, r2};
  cudaStream_t s = (cudaStream_t)stream;
  if (d <= 32) return launch<32>(a, s);
  if (d <= 64) return launch<64>(a, s);
  if (d <= 128) return launch<128>(a, s);
  return launch<256>(a, s);
}
