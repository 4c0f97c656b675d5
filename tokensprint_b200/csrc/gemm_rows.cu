// Products of at most 16 rows, out[M, N] = X[M, K] * W[N, K]^T in bfloat16 with float32 sums, for steps of few tokens.
//
// What bounds such a product is the weights' way from device memory and, for the smaller ones, the seam to the
// product before it: nothing of its input exists until that one has stored its last row.  The kernel is built
// so that as little as possible is left to do after that moment:
//   * every warp has a ring of its own in shared memory that its lanes fill by 16-byte cp.async, each lane with the very
//     bytes it will multiply, so that nobody waits for anybody: a lane waits for its own copies, in order.  128 KB
//     an SM are asked for before `griddepcontrol.wait` (no kernel writes weights), so a product whose weights fit
//     the rings of the chip finds them there when its input is ready.  (Loads into registers instead were as fast alone, and
//     10 to 16 us slower a product inside a step of 8 rows, 24,576 x 4,096: under way they stand in the L1, and an SM
//     keeps the small L1 of the kernel before while any of its CTAs runs.);
//   * no tile is shared between CTAs: a CTA takes 8 RU rows of W over the whole of K, its 16 warps 64 columns each in turn,
//     and the warps' sums meet in shared memory.  No partial sums in device memory, no tickets;
//   * the products are mma.sync m16n8k16 with the tokens as the 16 rows and 8 rows of W as columns: a lane's 2 x 16
//     bytes of a row of W are its part of four such products as they arrive.  (The columns that product i
//     takes as its k = 2t, 2t+1, 2t+8, 2t+9 are 32 (i / 2) + 8 t + 4 (i % 2) .. + 3 of the chunk, in X as in W: a sum over k has no order.)
//     The tensor cores are idle nine tenths of the time either way; what tcgen05 needs (tiles of 128 rows in
//     shared memory, accumulators in tensor memory) is what makes a product's end long when the tile is small.
// The epilogues are those of gemm_tcgen05.cu: row scale, gated activation, residual sum with the next norm's input and
// row sums of squares (per 16 columns), q/k norm with rotation and cache store (a head's 128 rows are shared by
// a cluster of four CTAs with 16 pairs (j, j + 64) each, which exchange their sums of squares through distributed shared memory).
// A row's sums are added up in one order whatever the rows beside it, the number of warps included.
//
// Measured (B200; a whole decode step, us, with gemm_tcgen05.cu's products and with these, about 60 of a small step's gain being its
// attention's): 0.6B of 1 request 1,124 -> 670, of 8 1,226 -> 802, of 14 1,312 -> 1,109; 8B of 1 3,278 -> 2,856, of 4 3,422 -> 3,132, of 8
// 3,467 -> 3,336; four small products of a layer (0.6B, 1 row) 27.8 -> 14.6, floor 4.9; gate and up of 24,576 x 4,096, 8 rows, alone 33.7: 6.0 TB/s.
//
// The reference runs these products through nn.Linear (engine/nn/attention.py:122-135, engine/nn/layers.py:61-66).
#include "common.cuh"

namespace {

constexpr int CHUNK = 64;       // columns of K a warp takes at a time: 128 bytes of every row
constexpr int MAX_ROWS = 16;
constexpr int CLUSTER = 4;      // CTAs that share a head
constexpr int HEAD = 128;
constexpr int X_PAD = 64;       // bytes
constexpr int MODE_PLAIN = 0, MODE_GLU = 1, MODE_RESIDUAL_NORM = 2, MODE_QK_ROPE = 3;

struct RowsArgs {
  const __nv_bfloat16* x;
  const char* w;
  long long ldx;
  unsigned int ldw_bytes;
  int M, N, K, tasks, mode;
  void* out;
  long long ldo;
  int out_f32, glu_act;
  const float* scale_ssq;  // [scale_tiles, M] or null
  int scale_tiles;
  float scale_width, scale_eps;
  float* hidden;           // MODE_RESIDUAL_NORM
  const float* norm_w;
  __nv_bfloat16* xprime;
  float* ssq_out;          // [tasks, M]
  long long ldh;
  float branch_scale;
  __nv_bfloat16* q_out;    // MODE_QK_ROPE
  __nv_bfloat16* k_cache;
  __nv_bfloat16* v_cache;
  const int* slot_mapping;
  const int* positions;
  const float* q_norm_w;
  const float* k_norm_w;
  const float* inv_freq;
  const float2* rope_cs;
  float qk_eps;
  int nq, nkv;
  const char* prefetch;
  unsigned long long prefetch_bytes;
};

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// The same place of this variable in the shared memory of CTA `cta` of the cluster.
__device__ __forceinline__ uint32_t remote_addr(const void* p, uint32_t cta) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr(p)), "r"(cta));
  return remote;
}
__device__ __forceinline__ void store_remote(const float* p, uint32_t cta, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote_addr(p, cta)), "f"(v) : "memory");
}
// 16 bytes of weights into this CTA's memory: they pass once, so they go first from the L2.
__device__ __forceinline__ void copy_weights(uint32_t dst, const char* src, uint64_t policy) {
  asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy) : "memory");
}
__device__ __forceinline__ uint4 read_16(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}

// RU groups of 8 rows of W per task, MH halves of 8 tokens; a warp's ring holds 8 KB, 8 / RU chunks of the RU groups.
template <int RU, int MH, int WARPS, bool QK>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 2 : 1) gemm_rows_kernel(const __grid_constant__ RowsArgs a) {
  constexpr int ROWS = 8 * MH, THREADS = WARPS * 32, CHAINS = 4 / RU, COLS = 8 * RU, SLOTS = 8 / RU;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ float rstd_s[MAX_ROWS];
  __shared__ float ssq_s[CLUSTER][MAX_ROWS];  // row sums of squares of a head, by the CTAs that share it
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int M = a.M, K = a.K;
  ts_pdl_launch_dependents();
  unsigned int rank = 0;
  if (QK) asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  // x rows 64 bytes longer than K: the eight lanes of a 16-byte read phase (half a line of two rows) hit different banks
  const int x_stride = K * 2 + X_PAD;
  unsigned char* x_s = smem + WARPS * SLOTS * RU * 1024;          // behind the rings
  float* red = reinterpret_cast<float*>(x_s + (size_t)M * x_stride);  // [QK ? 1 : 2][WARPS][ROWS][COLS]
  const int nc = (K / CHUNK - warp + WARPS - 1) / WARPS;                // chunks of this warp, at least 1
  const int n_tasks = QK ? 1 : (a.tasks - 1 - (int)blockIdx.x) / (int)gridDim.x + 1;

  // ---- the copies run ahead of the sums, chunk by chunk and task by task; one group of copies a chunk, also where it is empty
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  const uint32_t ring = smem_addr(smem) + warp * (SLOTS * RU * 1024) + lane * 16;
  unsigned int off[RU];
  int load_task = blockIdx.x, load_c = 0, tasks_to_load = n_tasks, load_slot = 0;
  auto row_offsets = [&]() {
#pragma unroll
    for (int u = 0; u < RU; ++u) {
      int row;
      if (QK) {
        // the CTA has 16 pairs (j, j + 64) of a head: 16 rank .. + 15 below 64, and the same above
        row = load_task / CLUSTER * HEAD + (u >= 2 ? 64 : 0) + rank * 16 + (u & 1) * 8 + g;
      } else if (a.mode == MODE_GLU) {  // four gate rows and the up rows of the same outputs
        const int o = (load_task * RU + u) * 4 + (g & 3);
        row = (o >> 6) * 128 + (o & 63) + (g >= 4 ? 64 : 0);
      } else {
        row = (load_task * RU + u) * 8 + g;
      }
      row = min(row, a.N - 1);
      off[u] = (unsigned int)row * a.ldw_bytes + (unsigned int)(warp * CHUNK * 2 + t * 16);
    }
  };
  auto load_next = [&]() {
    if (tasks_to_load > 0) {
      const uint32_t dst = ring + load_slot * (RU * 1024);
#pragma unroll
      for (int u = 0; u < RU; ++u) {
        const char* src = a.w + off[u];
        copy_weights(dst + u * 1024, src, policy);
        copy_weights(dst + u * 1024 + 512, src + 64, policy);
        off[u] += WARPS * CHUNK * 2;
      }
      load_slot = load_slot + 1 == SLOTS ? 0 : load_slot + 1;
      if (++load_c == nc) {
        load_c = 0;
        load_task += gridDim.x;
        tasks_to_load -= 1;
        if (tasks_to_load > 0) row_offsets();
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  row_offsets();
#pragma unroll
  for (int j = 0; j < SLOTS; ++j) load_next();

  if (QK) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // waited for before the first write to another CTA's memory
  // 16-byte pieces of x: this thread's first, and how far its next is
  const int row_pieces = K / 8, step_m = THREADS / row_pieces, step_col = THREADS % row_pieces;
  int x_m = tid / row_pieces, x_col = tid % row_pieces;
  ts_pdl_wait();
  // x through registers (as asynchronous copies it would be waited for behind the weights), eight pieces of a thread under way at once
  while (x_m < M) {
    uint4 v[8];
    unsigned char* to[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      to[j] = nullptr;
      if (x_m < M) {
        v[j] = __ldcg(reinterpret_cast<const uint4*>(a.x + (size_t)x_m * a.ldx + x_col * 8));
        to[j] = x_s + (size_t)x_m * x_stride + x_col * 16;
      }
      x_m += step_m;
      x_col += step_col;
      if (x_col >= row_pieces) {
        x_col -= row_pieces;
        x_m += 1;
      }
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (to[j] != nullptr) *reinterpret_cast<uint4*>(to[j]) = v[j];
  }
  for (int m = warp; m < M; m += WARPS) {
    float sum = 0.f;
    if (a.scale_ssq != nullptr)
      for (int j = lane; j < a.scale_tiles; j += 32) sum += __ldcg(a.scale_ssq + (size_t)j * M + m);
    sum = ts_warp_sum(sum);
    if (lane == 0) rstd_s[m] = a.scale_ssq != nullptr ? rsqrtf(sum / a.scale_width + a.scale_eps) : 1.f;
  }
  __syncthreads();

  const uint32_t x_lo = smem_addr(x_s) + g * x_stride + warp * CHUNK * 2 + t * 16, x_hi = x_lo + 8 * x_stride;
  const bool has_lo = g < M, has_hi = MH == 2 && g + 8 < M;
  int slot = 0;
  int task = blockIdx.x;
  for (int it = 0; it < n_tasks; ++it, task += gridDim.x) {
    float hidden0 = 0.f, norm0 = 0.f;
    if (!QK && a.mode == MODE_RESIDUAL_NORM && tid < M * COLS) {
      // what the epilogue adds to: asked for now.  Nobody else writes these columns.
      const int col = task * COLS + tid % COLS;
      if (col < a.N) {
        hidden0 = __ldcg(a.hidden + (size_t)(tid / COLS) * a.ldh + col);
        norm0 = a.norm_w[col];
      }
    }
    // 4 / RU chains per group of rows: a product waits for the one before it in its chain.  Eight warps that share a head keep the sums of every
    // other chunk apart, which are those of 16 warps, so that a row's bits do not depend on the form.
    constexpr int SETS = QK && WARPS == 8 ? 2 : 1;
    float acc[SETS][4][4];
#pragma unroll
    for (int i = 0; i < SETS; ++i)
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[i][u][0] = acc[i][u][1] = acc[i][u][2] = acc[i][u][3] = 0.f;
    auto chunk = [&](int c, float (&sums)[4][4]) {
      asm volatile("cp.async.wait_group %0;" ::"n"(SLOTS - 1) : "memory");
      const int x_off = c * (WARPS * CHUNK * 2);
      uint4 lo[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)}, hi[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
      if (has_lo) {
        lo[0] = read_16(x_lo + x_off);
        lo[1] = read_16(x_lo + x_off + 64);
      }
      if (has_hi) {
        hi[0] = read_16(x_hi + x_off);
        hi[1] = read_16(x_hi + x_off + 64);
      }
      const uint32_t from = ring + slot * (RU * 1024);
      uint4 w[RU][2];
#pragma unroll
      for (int u = 0; u < RU; ++u) {
        w[u][0] = read_16(from + u * 1024);
        w[u][1] = read_16(from + u * 1024 + 512);
      }
#pragma unroll
      for (int u = 0; u < RU; ++u) {
        mma_16816(sums[u * CHAINS], lo[0].x, hi[0].x, lo[0].y, hi[0].y, w[u][0].x, w[u][0].y);
        mma_16816(sums[u * CHAINS + 1 % CHAINS], lo[0].z, hi[0].z, lo[0].w, hi[0].w, w[u][0].z, w[u][0].w);
        mma_16816(sums[u * CHAINS + 2 % CHAINS], lo[1].x, hi[1].x, lo[1].y, hi[1].y, w[u][1].x, w[u][1].y);
        mma_16816(sums[u * CHAINS + 3 % CHAINS], lo[1].z, hi[1].z, lo[1].w, hi[1].w, w[u][1].z, w[u][1].w);
      }
      load_next();  // into the slot just read
      slot = slot + 1 == SLOTS ? 0 : slot + 1;
    };
    for (int c = 0; c < nc; c += SETS) {
      chunk(c, acc[0]);
      if (SETS == 2 && c + 1 < nc) chunk(c + 1, acc[SETS - 1]);
    }
    // ---- the warps' sums meet in shared memory (two buffers in turn: one barrier a task)
    float* r = red + (size_t)(it & 1) * (WARPS * ROWS * COLS);
    // Rows of a head's sums are as long as the banks: permuted so that neither four rows written at once nor two read at once share any.
    auto place = [](int m, int n) { return m * COLS + (QK ? n ^ ((m & 1) << 4 | (m & 2) << 2) : n); };
#pragma unroll
    for (int u = 0; u < RU; ++u) {
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[i] = acc[0][u * CHAINS][i];
#pragma unroll
        for (int k = 1; k < CHAINS; ++k) v[i] += acc[0][u * CHAINS + k][i];
      }
      float* mine = r + warp * ROWS * COLS + place(g, u * 8 + 2 * t);
      *reinterpret_cast<float2*>(mine) = make_float2(v[0], v[1]);
      if (MH == 2) *reinterpret_cast<float2*>(mine + 8 * COLS) = make_float2(v[2], v[3]);
    }
    // The second set takes the place of the warp's ring, which is empty: a head's CTA has one task, and its last chunks were waited for and read
    // (by other lanes too, hence the warp's barrier).
    float* odd = reinterpret_cast<float*>(smem);
    constexpr int ODD_WARP = SLOTS * RU * 1024 / (int)sizeof(float);
    static_assert(SETS == 1 || (CHAINS == 1 && ROWS * COLS <= ODD_WARP), "a set fits a ring");
    if (SETS == 2) {
      __syncwarp();
#pragma unroll
      for (int u = 0; u < RU; ++u) {
        const float(&v)[4] = acc[SETS - 1][u];
        float* mine = odd + warp * ODD_WARP + place(g, u * 8 + 2 * t);
        *reinterpret_cast<float2*>(mine) = make_float2(v[0], v[1]);
        if (MH == 2) *reinterpret_cast<float2*>(mine + 8 * COLS) = make_float2(v[2], v[3]);
      }
    }
    __syncthreads();
    auto total = [&](int m, int n) {
      float sum = 0.f;
#pragma unroll
      for (int w = 0; w < WARPS; ++w) sum += r[w * ROWS * COLS + place(m, n)];
      if (SETS == 2) {  // the warps 8 to 15 of the form with 16
#pragma unroll
        for (int w = 0; w < WARPS; ++w) sum += odd[w * ODD_WARP + place(m, n)];
      }
      return sum * rstd_s[m];
    };
    if (QK) {
      const int head = task / CLUSTER;
      const bool is_q = head < a.nq, is_k = !is_q && head < a.nq + a.nkv;
      const float* w = is_q ? a.q_norm_w : (is_k ? a.k_norm_w : nullptr);
      const int m = tid >> 4, jj = tid & 15, j = rank * 16 + jj;
      const bool mine = m < M;  // THREADS >= 16 * MAX_ROWS
      float lo = 0.f, hi = 0.f;
      if (mine) {
        lo = total(m, jj);
        hi = total(m, 16 + jj);
      }
      asm volatile("barrier.cluster.wait.aligned;" ::: "memory");  // the others have started: their memory may be written
      if (w != nullptr) {  // the same for the whole cluster
        float ss = lo * lo + hi * hi;
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (mine && jj < CLUSTER) store_remote(&ssq_s[rank][m], jj, ss);  // lane jj writes to CTA jj of the cluster
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (mine) {
          const float s = ssq_s[0][m] + ssq_s[1][m] + ssq_s[2][m] + ssq_s[3][m];
          const float rn = rsqrtf(s / (float)HEAD + a.qk_eps);
          lo *= rn * w[j];
          hi *= rn * w[64 + j];
        }
      }
      if (mine) {
        if ((is_q || is_k) && a.inv_freq != nullptr) {
          float sn, cs;
          if (a.rope_cs != nullptr) {
            const float2 v = a.rope_cs[(size_t)m * 64 + j];
            cs = v.x;
            sn = v.y;
          } else {
            sincosf((float)a.positions[m] * a.inv_freq[j], &sn, &cs);
          }
          const float l = lo * cs - hi * sn, h = hi * cs + lo * sn;
          lo = l;
          hi = h;
        }
        const int slot = is_q ? 0 : a.slot_mapping[m];
        if (slot >= 0) {
          __nv_bfloat16* dst = is_q ? a.q_out + ((size_t)m * a.nq + head) * HEAD
                                    : (is_k ? a.k_cache + ((size_t)slot * a.nkv + (head - a.nq)) * HEAD
                                            : a.v_cache + ((size_t)slot * a.nkv + (head - a.nq - a.nkv)) * HEAD);
          dst[j] = __float2bfloat16_rn(lo);
          dst[64 + j] = __float2bfloat16_rn(hi);
        }
      }
    } else if (a.mode == MODE_GLU) {
      constexpr int OUTS = COLS / 2;
      for (int idx = tid; idx < M * OUTS; idx += THREADS) {
        const int m = idx / OUTS, n = idx % OUTS, col = task * OUTS + n;
        const int at = (n >> 2) * 8 + (n & 3);
        const float gate = total(m, at), up = total(m, at + 4);
        if (col < (a.N >> 1))
          reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)m * a.ldo + col] = __float2bfloat16_rn(ts_glu_gate_fast(gate, a.glu_act) * up);
      }
    } else if (a.mode == MODE_RESIDUAL_NORM) {
      static_assert(QK || THREADS >= MAX_ROWS * COLS, "a thread finishes at most one element");
      if ((tid & ~31) < M * COLS) {  // whole warps: COLS divides 32
        const int m = tid / COLS, n = tid % COLS, col = task * COLS + n;
        float ss = 0.f;
        if (m < M && col < a.N) {
          const size_t at = (size_t)m * a.ldh + col;
          const float h = fmaf(a.branch_scale, total(m, n), hidden0);
          a.hidden[at] = h;
          a.xprime[at] = __float2bfloat16_rn(h * norm0);
          ss = h * h;
        }
#pragma unroll
        for (int o = COLS / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (m < M && n == 0) a.ssq_out[(size_t)task * M + m] = ss;
      }
    } else {
      for (int idx = tid; idx < M * COLS; idx += THREADS) {
        const int m = idx / COLS, n = idx % COLS, col = task * COLS + n;
        const float v = total(m, n);
        if (col < a.N) {
          if (a.out_f32)
            reinterpret_cast<float*>(a.out)[(size_t)m * a.ldo + col] = v;
          else
            reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)m * a.ldo + col] = __float2bfloat16_rn(v);
        }
      }
    }
  }
  if (a.prefetch != nullptr && tid == THREADS - 1) {
    // its share of the next product's weights into the L2, while small kernels stand between the two
    constexpr unsigned long long PIECE = 16 * 1024;
    for (unsigned long long o = (unsigned long long)blockIdx.x * PIECE; o < a.prefetch_bytes; o += (unsigned long long)gridDim.x * PIECE) {
      const unsigned bytes = (unsigned)min(PIECE, a.prefetch_bytes - o) & ~15u;
      if (bytes) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.prefetch + o), "r"(bytes) : "memory");
    }
  }
}

int sm_count() {
  static int count = 0;
  if (count == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || count <= 0)
      count = 148;
  }
  return count;
}

struct Shape {
  int warps;
};

constexpr int RU_PLAIN = 2, RU_QK = 4;
constexpr size_t SMEM_TWO = 115 * 1000;  // two CTAs of an SM
constexpr size_t SMEM_ONE = 225 * 1024;  // one
constexpr int CLUSTER_SLOTS = 132;       // CTAs in clusters of four that stand on the chip at one CTA an SM

size_t smem_bytes(int M, int K, bool qk, int warps) {
  const int sums = qk ? RU_QK : 2 * RU_PLAIN;  // one buffer where a CTA has one task
  return (size_t)warps * 8 * 1024 + (size_t)M * (K * 2 + X_PAD) + (size_t)warps * (M > 8 ? 16 : 8) * 8 * sums * sizeof(float);
}

// Whether this kernel takes a product, and with how many warps a CTA.  Decode steps in us, the products of gemm_tcgen05.cu before:
// with two groups of rows and 16 warps (one CTA an SM, which reads the input once) 0.6B of 1 / 8 / 14 requests 1,133 / 1,240 /
// 1,379 -> 900 / 986 / 1,256, 8B of 1 / 4 / 8 requests 3,324 / 3,412 / 3,485 -> 3,192 / 3,206 / 3,311; with one group 960 .. 1,346
// and 3,387 .. 3,333; with four 909 .. 1,350 and 3,170 .. 3,362; with 8 warps and two CTAs an SM 947 .. 1,380 and 3,226 .. 3,486.
// K below 1,024 would leave warps without a chunk; an input that leaves no room for rings of 128 KB stays with the other kernel.
bool choose(int M, int N, int K, bool qk, Shape* s) {
  if (M < 1 || M > MAX_ROWS || K % CHUNK != 0 || K / CHUNK < 16) return false;
  s->warps = 16;
  // Tasks of few columns end often: above 8 rows their sums over the warps and the epilogue outlast the copies where a CTA has many of them.  us, here :
  // gemm_tcgen05.cu, K = 1,024: the logits' 151,936 columns at 9 / 16 rows 53 / 57 : 49 / 50, gate and up of 24,576 at 16 rows 15.3 : 13.6, of
  // 8,192 8.9 : 9.5; K = 1,536, gate and up of 32,768 at 16 rows 24 : 21; K = 2,048 25 : 26.  Up to 8 rows they are even (50.1 : 48.6 at 8).
  if (!qk && M > 8 && K < 2048 && N > 4 * 148 * 8 * RU_PLAIN) return false;
  if (!qk) return smem_bytes(M, K, false, 16) <= SMEM_ONE;
  // Four CTAs a head: two an SM (0.6B of 8 requests 986 -> 898, 8B of 4 3,206 -> 3,146), or, where all stand at once, one of 16
  // warps for a small input (0.6B of 1 request: 781 beside 813) or one too large for two an SM (of 14: 1,256 -> 1,218).
  // In two rounds either is slower than the other kernel (one an SM: 8B of 8 requests 3,545 against 3,311; two an SM: 80 heads over
  // 5,120 columns, 320 CTAs, 26 and 27 us at 1 and 4 rows against 24 and 21; 56 heads, 224 CTAs, 15 and 16 against 21 and 18).
  const bool two = smem_bytes(M, K, true, 8) <= SMEM_TWO && N / HEAD * CLUSTER <= 2 * CLUSTER_SLOTS;
  if (N / HEAD * CLUSTER <= CLUSTER_SLOTS && (M <= 2 || !two)) return smem_bytes(M, K, true, 16) <= SMEM_ONE;
  s->warps = 8;
  return two;
}

template <int MH, int WARPS, bool QK>
int launch(RowsArgs& a, cudaStream_t stream) {
  constexpr int RU = QK ? RU_QK : RU_PLAIN;
  static bool configured = false;
  auto kernel = gemm_rows_kernel<RU, MH, WARPS, QK>;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(WARPS == 8 ? SMEM_TWO : SMEM_ONE));
    // the L1 is of no use here, and an SM changes its share only when it stands empty
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  const size_t smem = smem_bytes(a.M, a.K, QK, WARPS);
  if (QK) {
    a.tasks = (a.nq + 2 * a.nkv) * CLUSTER;
    return ts_launch_cluster(kernel, dim3(a.tasks), dim3(WARPS * 32), smem, stream, CLUSTER, a);
  }
  a.tasks = (a.N + 8 * RU - 1) / (8 * RU);
  return ts_launch(kernel, dim3(a.tasks < sm_count() ? a.tasks : sm_count()), dim3(WARPS * 32), smem, stream, a);
}

template <int MH>
int dispatch(RowsArgs& a, const Shape& s, bool qk, cudaStream_t stream) {
  if (!qk) return launch<MH, 16, false>(a, stream);
  return s.warps == 16 ? launch<MH, 16, true>(a, stream) : launch<MH, 8, true>(a, stream);
}

int run_rows(RowsArgs& a, const void* x, const void* w, int M, int N, int K, long long ldx, long long ldw, bool qk, const void* prefetch,
             long long prefetch_bytes, void* stream_) {
  if (K <= 0 || ldx < K || ldw < K) return TS_ERR_BAD_ARGUMENT;
  Shape s;
  if (!choose(M, N, K, qk, &s)) return TS_ERR_UNSUPPORTED_SIZE;
  // rows of W on whole sectors of 32 bytes: the 64 bytes that four lanes ask for at a time would touch three of them otherwise, not two
  if ((ldx % 8) || (ldw % 16) || ((uintptr_t)x % 16) || ((uintptr_t)w % 32) || (long long)N * ldw * 2 >= (1ll << 32)) return TS_ERR_UNSUPPORTED_SIZE;
  if (a.scale_ssq != nullptr && (a.scale_tiles <= 0 || !(a.scale_width > 0.f))) return TS_ERR_BAD_ARGUMENT;
  a.x = (const __nv_bfloat16*)x;
  a.w = (const char*)w;
  a.ldx = ldx;
  a.ldw_bytes = (unsigned int)(ldw * 2);
  a.M = M;
  a.N = N;
  a.K = K;
  a.prefetch = (prefetch_bytes > 0 && ((uintptr_t)prefetch % 16) == 0) ? (const char*)prefetch : nullptr;
  a.prefetch_bytes = prefetch_bytes > 0 ? (unsigned long long)prefetch_bytes : 0ull;
  cudaStream_t stream = (cudaStream_t)stream_;
  return M > 8 ? dispatch<2>(a, s, qk, stream) : dispatch<1>(a, s, qk, stream);
}

}  // namespace

// Rows of sums of squares that mode 2 leaves for an [N, K] weight and M rows, or 0 where this kernel does not take the product.
TS_EXPORT int ts_gemm_rows_ssq_tiles(int M, int N, int K) {
  Shape s;
  if (!choose(M, N, K, false, &s)) return 0;
  return (N + 8 * RU_PLAIN - 1) / (8 * RU_PLAIN);
}

// With how many warps a CTA ts_gemm_rows_qk_rope takes the product of M rows with `heads` heads of W (0: not at all).
TS_EXPORT int ts_gemm_rows_takes_heads(int M, int heads, int K) {
  Shape s;
  return choose(M, heads * HEAD, K, true, &s) ? s.warps : 0;
}

// Arguments as for ts_gemm_skinny_fused (ssq_out: ts_gemm_rows_ssq_tiles(M, N, K) rows).
TS_EXPORT int ts_gemm_rows_fused(const void* x, const void* w, void* out, int M, int N, int K, long long ldx, long long ldw, long long ldo,
                                 int out_f32, int mode, const float* scale_ssq, int scale_tiles, float scale_width, float scale_eps,
                                 float* hidden, long long ldh, const float* norm_w, void* xprime, float* ssq_out, float branch_scale,
                                 int glu_act, const void* prefetch, long long prefetch_bytes, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (mode < MODE_PLAIN || mode > MODE_RESIDUAL_NORM || (glu_act != TS_GLU_SILU && glu_act != TS_GLU_GELU_TANH)) return TS_ERR_BAD_ARGUMENT;
  if (mode == MODE_GLU && ((N % 128) || out_f32 || ldo < N / 2)) return TS_ERR_BAD_ARGUMENT;
  if (mode == MODE_RESIDUAL_NORM && (hidden == nullptr || norm_w == nullptr || xprime == nullptr || ssq_out == nullptr || ldh < N))
    return TS_ERR_BAD_ARGUMENT;
  if (mode == MODE_PLAIN && ldo < N) return TS_ERR_BAD_ARGUMENT;
  RowsArgs a = {};
  a.mode = mode;
  a.out = out;
  a.ldo = ldo;
  a.out_f32 = out_f32;
  a.glu_act = glu_act;
  a.scale_ssq = scale_ssq;
  a.scale_tiles = scale_tiles;
  a.scale_width = scale_width;
  a.scale_eps = scale_eps;
  a.hidden = hidden;
  a.norm_w = norm_w;
  a.xprime = (__nv_bfloat16*)xprime;
  a.ssq_out = ssq_out;
  a.ldh = ldh;
  a.branch_scale = branch_scale;
  return run_rows(a, x, w, M, N, K, ldx, ldw, false, prefetch, prefetch_bytes, stream);
}

// Arguments as for ts_gemm_skinny_qk_rope.
TS_EXPORT int ts_gemm_rows_qk_rope(const void* x, const void* w, int M, int K, long long ldx, long long ldw, int nq, int nkv, void* q_out,
                                   void* k_cache, void* v_cache, const int* slot_mapping, const int* positions, const float* q_norm_w,
                                   const float* k_norm_w, float qk_eps, const float* inv_freq, const float* rope_cos_sin,
                                   const float* scale_ssq, int scale_tiles, float scale_width, float scale_eps, const void* prefetch,
                                   long long prefetch_bytes, void* stream) {
  if (M <= 0) return 0;
  if (nq <= 0 || nkv <= 0 || q_out == nullptr || k_cache == nullptr || v_cache == nullptr || slot_mapping == nullptr ||
      (inv_freq != nullptr && positions == nullptr))
    return TS_ERR_BAD_ARGUMENT;
  // what the tcgen05 kernel refuses; the table's (cos, sin) are read as pairs of 8 bytes
  if (((uintptr_t)q_out | (uintptr_t)k_cache | (uintptr_t)v_cache) % 8 || (uintptr_t)rope_cos_sin % 16) return TS_ERR_UNSUPPORTED_SIZE;
  RowsArgs a = {};
  a.mode = MODE_QK_ROPE;
  a.scale_ssq = scale_ssq;
  a.scale_tiles = scale_tiles;
  a.scale_width = scale_width;
  a.scale_eps = scale_eps;
  a.q_out = (__nv_bfloat16*)q_out;
  a.k_cache = (__nv_bfloat16*)k_cache;
  a.v_cache = (__nv_bfloat16*)v_cache;
  a.slot_mapping = slot_mapping;
  a.positions = positions;
  a.q_norm_w = q_norm_w;
  a.k_norm_w = k_norm_w;
  a.inv_freq = inv_freq;
  a.rope_cs = inv_freq != nullptr ? reinterpret_cast<const float2*>(rope_cos_sin) : nullptr;
  a.qk_eps = qk_eps;
  a.nq = nq;
  a.nkv = nkv;
  return run_rows(a, x, w, M, (nq + 2 * nkv) * HEAD, K, ldx, ldw, true, prefetch, prefetch_bytes, stream);
}
