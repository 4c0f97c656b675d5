// The two products of a routed feed-forward on the 5th-generation tensor cores (bfloat16, tcgen05.mma, float32
// sums in tensor memory, operands by TMA), over the plan that moe.cu makes: the (token, choice) pairs
// sorted by expert, in row tiles (of 128 places, or of 32 in steps of few tokens) that never straddle two experts.
//
// Two kernels, both of persistent CTAs, one per SM, that take items in turn, the columns of a row tile side by side, so
// that an expert's weights come from device memory once and from the L2 after that; operands pass through a ring of
// slices of 64 along k with a full and an empty mbarrier each, and two accumulators take turns, so that the epilogue of an
// item runs under the products of the next.  Rows of shared memory that no copy fills hold old values: a sum reads its own
// place's row and its own weight row only, and sums that belong to no pair are never stored.
//
// Many rows (moe_many_kernel): an item is a row tile of 128 places, the MMA's M, and 256 weight rows, its N: for the first
// product the gate rows and the up rows of the same 128 outputs (so the activation is the epilogue).
//   warp 4       TMA: per slice two boxes of weight rows and, for the second product, one box of consecutive places;
//   warps 6-9    (first product) the tokens' rows by 16-byte cp.async in the swizzled layout, only as many as the tile has
//                (tile::gather4 copies, 40 ns each, took 981 us where this takes 397: 16,384 pairs of 32 experts, 4,096 -> 2 x 1,536);
//   warp 5       one elected lane: every tcgen05.mma;
//   the others   epilogue: a thread has a place and half of its columns, reads its sums from tensor memory and writes them.
// 8,192 pairs of these experts 242 us, 0.85 PFLOP/s, and 122 us for down (mma.sync tiles of 128 x 128: 863 and 450): the tensor pipes are
// busy 62 % of the time that the SMs are, which ask the L2 for 48 KB a slice (42 % of its peak), and 768 items leave the last of six
// rounds of CTAs a fifth full; 32,768 pairs 748 us, 1.10 PFLOP/s.
//
// Few rows (moe_few_kernel; up to 12 pairs per expert on average): the step streams the chosen experts' weights and little
// else, at a rate that follows the bytes of weights in flight.  Row tiles of 32 places are the MMA's N and the weight rows
// its M, two tiles of 128 (or, without a gate, one: see `narrow`), so 192 KB of weights are in flight per SM, and the epilogue, which nothing
// hides where a CTA has one item, is spread over 128 threads that each have a weight row and only as many
// columns as the tile has places (with the places as M one warp did all of it, 5 to 8 us of the 35).  The tokens' rows come by
// tile::gather4, four rows a copy, only as many as the tile has.
// 32 experts, 4,096 -> 2 x 1,536, cold L2, gate/up and down: 32 pairs 84 and 46 us (6.3 and 5.7 TB/s), 256 pairs 132 and 66 (6.1 and 6.1 TB/s).
// 16 experts, 2,048 -> 2 x 1,024, six calls in a graph, gate/up and down: 2 pairs 15.5 and 8.1 us, 8 pairs 15.8 and 8.9, 66 pairs 26.3 and 10.6
// (the down matrices stay in the L2 in part); tiles of 16 rows on mma.sync, three CTAs an SM, took 22.2 and 11.8, 26.6 and 14.3, 33.1 and 17.6.
//
// The pair's routing weight multiplies the float32 sums, not the rounded input: (w x) . g = w (x . g) without
// a second rounding of x.  Every output element is one chain of sums over k in a fixed order.
// Every wait is on an mbarrier fed by this CTA's own copies, MMAs and warps, bounded; one that gives up raises the
// error word, and the CTA lets its copies land and its products end, frees its tensor memory and returns.
#include <cuda.h>
#include <math.h>

#include "common.cuh"
#include "moe_act.cuh"
#include "variants/kv_tensor_map.cuh"

namespace {

constexpr int BK = 64, SHARED_EXPERTS = 1024;  // up to this many experts the plan's offsets are kept in shared memory
constexpr int ROWS_MANY = 128, ROWS_FEW = 32;  // places per row tile
constexpr int GATHER_WARPS = 4, GATHER_THREADS = 32 * GATHER_WARPS;
constexpr uint32_t SPIN_LIMIT = 1u << 22;

struct Args {
  const float* pair_weight;
  const int *order, *offsets, *tile_offsets;
  __nv_bfloat16* out;
  int* error;
  int E, K, NOUT, top, cols;  // cols: items per row tile
  float limit, alpha;
  int act_mode;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  for (uint32_t i = 0; i < SPIN_LIMIT; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
// four rows of 64 entries, by row number (the map's box is one row)
__device__ __forceinline__ void tma_gather4(uint32_t dst, const CUtensorMap* map, uint32_t bar, int c0, const int (&r)[4]) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool real) {
  const int bytes = real ? 16 : 0;  // 0: the piece is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// K-major operand, 128-byte swizzle: 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t desc_k_major(uint32_t addr) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool elect_one() {  // one lane of a converged warp
  uint32_t chosen;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(chosen));
  return chosen != 0;
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
__device__ __forceinline__ uint32_t idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ float rounded(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// 16 results of a row, from column n on
__device__ __forceinline__ void store16(__nv_bfloat16* dst, int n, int n_end, const float (&y)[16]) {
  if (n + 16 <= n_end && ((reinterpret_cast<uintptr_t>(dst + n) & 15) == 0)) {
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __nv_bfloat162 two = __floats2bfloat162_rn(y[2 * i], y[2 * i + 1]);
      v[i] = *reinterpret_cast<const uint32_t*>(&two);
    }
    *reinterpret_cast<uint4*>(dst + n) = make_uint4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<uint4*>(dst + n + 8) = make_uint4(v[4], v[5], v[6], v[7]);
  } else {
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (n + i < n_end) dst[n + i] = __float2bfloat16_rn(y[i]);
  }
}

// An item: a row tile of expert e with `rows` places from row0 on, and COLS outputs from n0 on.
struct Item {
  int e, row0, rows, n0;
};
template <int COLS, int BM>
__device__ __forceinline__ Item item_at(const Args& a, const int* plan, int it) {
  const int* offsets = plan != nullptr ? plan : a.offsets;
  const int* tile_offsets = plan != nullptr ? plan + a.E + 1 : a.tile_offsets;
  const int tile = it / a.cols;
  int lo = 0, hi = a.E;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (tile_offsets[mid] <= tile) lo = mid; else hi = mid;
  }
  Item w;
  w.e = lo;
  w.row0 = offsets[lo] + (tile - tile_offsets[lo]) * BM;
  w.rows = min(BM, offsets[lo + 1] - w.row0);
  w.n0 = (it - tile * a.cols) * COLS;
  return w;
}

// What both kernels share: the ring's barriers, the plan in shared memory, tensor memory, and leaving.
template <int STAGES>
struct Common {
  uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2], all_done;
  uint32_t tmem_base;
  int abort;
};
template <int STAGES>
__device__ __forceinline__ void begin(Common<STAGES>& c, const Args& a, int* plan, int fills, int readers, uint32_t tmem_cols) {
  const int tid = threadIdx.x;
  if (tid == 0) {
    c.abort = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(smem_u32(&c.full[s]), fills);
      mbar_init(smem_u32(&c.empty[s]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&c.acc_full[i]), 1);
      mbar_init(smem_u32(&c.acc_empty[i]), readers);
    }
    mbar_init(smem_u32(&c.all_done), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  for (int i = tid; plan != nullptr && i <= a.E; i += blockDim.x) {
    plan[i] = a.offsets[i];
    plan[a.E + 1 + i] = a.tile_offsets[i];
  }
  if (tid < 32) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&c.tmem_base)), "r"(tmem_cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  ts_pdl_launch_dependents();
}
template <int STAGES>
__device__ __forceinline__ void leave(Common<STAGES>& c, const Args& a, uint32_t tmem_cols) {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (c.abort != 0 && threadIdx.x == 0) *a.error = 1;
  if (threadIdx.x < 32) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem_base), "r"(tmem_cols) : "memory");
  }
}
// the last copies of a CTA whose waits gave up: wait (bounded, on a count of its own) until they have landed
template <int STAGES>
__device__ __forceinline__ void let_land(Common<STAGES>& c, int asked) {
  int patience = 0;
  for (int i = max(0, asked - STAGES); i < asked; ++i) mbar_wait(smem_u32(&c.full[i % STAGES]), (uint32_t)(i / STAGES) & 1, &patience);
}

// Everything this CTA asked of the tensor core is done when the commit arrives.  The warp that asked waits for it, on a count
// of its own: leave()'s barrier then holds everybody until no product writes tensor memory and no commit has yet to
// arrive, also where a wait gave up before.
template <int STAGES>
__device__ __forceinline__ void let_finish(Common<STAGES>& c) {
  if (elect_one()) umma_commit(smem_u32(&c.all_done));
  __syncwarp();
  int patience = 0;
  mbar_wait(smem_u32(&c.all_done), 0, &patience);
  if (patience != 0) c.abort = 1;
}

// ---- many rows ----

constexpr int TN = 256;
constexpr uint32_t MANY_A = ROWS_MANY * 128, MANY_B = TN * 128, MANY_STAGE = MANY_A + MANY_B;
constexpr int MANY_STAGES = 4;
constexpr uint32_t MANY_SMEM = MANY_STAGES * MANY_STAGE, MANY_TMEM = 2 * TN;
__host__ __device__ constexpr int many_threads(int mode) { return 320 + (mode != 0 ? GATHER_THREADS : 0); }

// MODE 1: gate and up; MODE 2: the first product of experts without a gate; MODE 0: down.
template <int MODE>
__global__ void __launch_bounds__(many_threads(MODE), 1) moe_many_kernel(const __nv_bfloat16* __restrict__ x, const __grid_constant__ CUtensorMap map_a,
                                                                         const __grid_constant__ CUtensorMap map_b0,
                                                                         const __grid_constant__ CUtensorMap map_b1, const Args a) {
  constexpr bool BY_TOKEN = MODE != 0;
  constexpr int COLS = MODE == 1 ? TN / 2 : TN;  // outputs of an item
  ts_pdl_wait();  // tensor memory is never held while waiting for another kernel
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_unaligned + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) Common<MANY_STAGES> c;
  int* plan = a.E <= SHARED_EXPERTS ? reinterpret_cast<int*>(smem + MANY_SMEM) : nullptr;  // offsets and tile_offsets, looked up for every item
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  begin(c, a, plan, BY_TOKEN ? 1 + GATHER_WARPS : 1, 8, MANY_TMEM);
  volatile int* abort_flag = &c.abort;
  const uint32_t sm = smem_u32(smem);
  const int items = a.tile_offsets[a.E] * a.cols, slices = (a.K + BK - 1) / BK;

  if (warp == 4) {
    int n = 0;  // slices asked for
    bool ok = true;
    for (int it = blockIdx.x; ok && it < items; it += gridDim.x) {
      const Item w = item_at<COLS, ROWS_MANY>(a, plan, it);
      const int b_row = w.e * a.NOUT + w.n0;
      for (int k = 0; k < slices; ++k, ++n) {
        const int st = n % MANY_STAGES;
        if (n >= MANY_STAGES) ok = mbar_wait(smem_u32(&c.empty[st]), (uint32_t)(n / MANY_STAGES - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint32_t bar = smem_u32(&c.full[st]), a_dst = sm + st * MANY_STAGE, b_dst = a_dst + MANY_A;
        if (lane == 0) mbar_expect_tx(bar, (BY_TOKEN ? 0u : MANY_A) + MANY_B);
        __syncwarp();
        if (lane < 2) {
          if (MODE == 1)
            tma_load_2d(b_dst + lane * (MANY_B / 2), lane == 0 ? &map_b0 : &map_b1, bar, k * BK, b_row);
          else
            tma_load_2d(b_dst + lane * (MANY_B / 2), &map_b0, bar, k * BK, b_row + lane * (TN / 2));
        }
        if (!BY_TOKEN && lane == 2) tma_load_2d(a_dst, &map_a, bar, k * BK, w.row0);
      }
    }
    if (*abort_flag) let_land(c, n);
  } else if (BY_TOKEN && warp >= 6 && warp < 6 + GATHER_WARPS) {
    // thread g: piece g % 8 (16 bytes) of the rows g / 8, g / 8 + 16, ... of the tile
    const int g = tid - 192, piece = g & 7, first_row = g >> 3;
    const uint32_t to = (uint32_t)first_row * 128 + (uint32_t)((piece ^ (first_row & 7)) << 4);
    constexpr int ROW_STEP = GATHER_THREADS / 8, PER = ROWS_MANY / ROW_STEP, AHEAD = MANY_STAGES - 1;
    static_assert(ROW_STEP % 8 == 0, "a thread's rows swizzle alike");
    int n = 0;
    bool ok = true;
    auto hand_over = [&](int i) {  // slice i of this warp's rows has landed and the tensor core may read it
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&c.full[i % MANY_STAGES]));
    };
    int mine_next = 0, pairs_next[PER];  // of the item after this one: its trips to the plan run under this one's slices
    auto look_up = [&](int it) {
      mine_next = 0;
      if (it >= items) return;
      const Item w = item_at<COLS, ROWS_MANY>(a, plan, it);
      mine_next = w.rows > first_row ? (w.rows - first_row + ROW_STEP - 1) / ROW_STEP : 0;
#pragma unroll
      for (int j = 0; j < PER; ++j) pairs_next[j] = j < mine_next ? a.order[w.row0 + first_row + j * ROW_STEP] : 0;
    };
    look_up(blockIdx.x);
    for (int it = blockIdx.x; ok && it < items; it += gridDim.x) {
      const __nv_bfloat16* src[PER];
      const int mine = mine_next;
#pragma unroll
      for (int j = 0; j < PER; ++j) src[j] = x + (size_t)(j < mine ? pairs_next[j] / a.top : 0) * a.K + piece * 8;
      look_up(it + gridDim.x);
      for (int k = 0; k < slices; ++k, ++n) {
        const int st = n % MANY_STAGES;
        if (n >= MANY_STAGES) ok = mbar_wait(smem_u32(&c.empty[st]), (uint32_t)(n / MANY_STAGES - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const bool real = k * BK + piece * 8 < a.K;
        const uint32_t dst = sm + st * MANY_STAGE + to;
#pragma unroll
        for (int j = 0; j < PER; ++j)
          if (j < mine) cp_async16(dst + j * (ROW_STEP * 128), real ? src[j] + k * BK : x, real);
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (n >= AHEAD - 1) {
          asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD - 1) : "memory");
          hand_over(n - (AHEAD - 1));
        }
      }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (ok)
      for (int i = max(0, n - (AHEAD - 1)); i < n; ++i) hand_over(i);
  } else if (warp == 5) {
    const uint64_t a_desc = desc_k_major(sm), b_desc = desc_k_major(sm + MANY_A);
    int n = 0, turn = 0;
    bool ok = true;
    for (int it = blockIdx.x; ok && it < items; it += gridDim.x, ++turn) {
      const int acc = turn & 1;
      if (turn >= 2) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.acc_empty[acc]), (uint32_t)(turn / 2 - 1) & 1, abort_flag));
      for (int k = 0; ok && k < slices; ++k, ++n) {
        const int st = n % MANY_STAGES;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.full[st]), (uint32_t)(n / MANY_STAGES) & 1, abort_flag));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elect_one()) {
          const uint64_t off = (uint64_t)((st * MANY_STAGE) >> 4);
#pragma unroll
          for (int ks = 0; ks < BK / 16; ++ks)
            umma_bf16(c.tmem_base + acc * TN, a_desc + off + ks * 2, b_desc + off + ks * 2, idesc(TN), (k | ks) != 0 ? 1u : 0u);
          umma_commit(smem_u32(&c.empty[st]));
          if (k == slices - 1) umma_commit(smem_u32(&c.acc_full[acc]));
        }
        __syncwarp();
      }
    }
    let_finish(c);
  } else {
    // warps 0-3 have the first half of the columns, the last four the second; a warp reaches the 32 lanes of tensor memory
    // of its number modulo 4
    const int half = warp < 4 ? 0 : 1, quarter = warp & 3;
    const int r = quarter * 32 + lane;
    int turn = 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x, ++turn) {
      const Item w = item_at<COLS, ROWS_MANY>(a, plan, it);
      const int acc = turn & 1;
      const bool mine = r < w.rows;
      const int pair = mine ? a.order[w.row0 + r] : 0;
      const float weight = (BY_TOKEN && mine && a.pair_weight != nullptr) ? a.pair_weight[pair] : 1.f;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&c.acc_full[acc]), (uint32_t)(turn / 2) & 1, abort_flag))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (quarter * 32 < w.rows) {
        const uint32_t addr = c.tmem_base + ((uint32_t)(quarter * 32) << 16) + acc * TN;
        __nv_bfloat16* dst = a.out + (size_t)(BY_TOKEN ? w.row0 + r : pair) * a.NOUT;
#pragma unroll 1
        for (int col = half * (COLS / 2); col < (half + 1) * (COLS / 2); col += 16) {
          uint32_t v[16], u[16];
          tmem_ld16(addr + col, v);
          if (MODE == 1) tmem_ld16(addr + COLS + col, u);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (mine && w.n0 + col < a.NOUT) {
            float y[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float s = __uint_as_float(v[i]);
              // the sums are rounded to bfloat16 before the activation, as a product stored to memory would be
              if (MODE == 1) y[i] = moe_gated_activation(a.act_mode, rounded(weight * s), rounded(weight * __uint_as_float(u[i])), a.limit, a.alpha);
              else if (MODE == 2) y[i] = moe_gated_activation(a.act_mode, 0.f, rounded(weight * s), a.limit, a.alpha);
              else y[i] = s;
            }
            store16(dst, w.n0 + col, a.NOUT, y);
          }
          __syncwarp();  // the next load from tensor memory is the whole warp's
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&c.acc_empty[acc]));
    }
  }
  leave(c, a, MANY_TMEM);
}

// ---- few rows ----

// TILES: tiles of 128 weight rows per item; MODE 1 has two, the gate rows and the up rows of 128 outputs.
template <int TILES>
struct Few {
  static constexpr uint32_t W_BYTES = TILES * 128 * 128, STAGE = W_BYTES + ROWS_FEW * 128;
  static constexpr int STAGES = 216 * 1024 / STAGE;
  static constexpr uint32_t SMEM = STAGES * STAGE;
  static constexpr uint32_t ACC = TILES * ROWS_FEW, TMEM_COLS = 2 * ACC;  // columns of one accumulator, and of both
};

template <int MODE, int TILES>
__global__ void __launch_bounds__(224, 1) moe_few_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w0,
                                                         const __grid_constant__ CUtensorMap map_w1, const Args a) {
  using F = Few<TILES>;
  static_assert(MODE != 1 || TILES == 2, "gate rows and up rows");
  constexpr bool BY_TOKEN = MODE != 0;
  constexpr int COLS = MODE == 1 ? 128 : TILES * 128;
  ts_pdl_wait();  // tensor memory is never held while waiting for another kernel
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_unaligned + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) Common<F::STAGES> c;
  int* plan = a.E <= SHARED_EXPERTS ? reinterpret_cast<int*>(smem + F::SMEM) : nullptr;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  begin(c, a, plan, 2, 4, F::TMEM_COLS);
  volatile int* abort_flag = &c.abort;
  const uint32_t sm = smem_u32(smem);
  const int items = a.tile_offsets[a.E] * a.cols, slices = (a.K + BK - 1) / BK;

  if (warp == 4 || warp == 6) {  // the weight rows; the tokens' or places' rows
    int n = 0;  // slices asked for
    bool ok = true;
    for (int it = blockIdx.x; ok && it < items; it += gridDim.x) {
      const Item w = item_at<COLS, ROWS_FEW>(a, plan, it);
      const int quads = (w.rows + 3) >> 2;  // gathers of four rows; the last one repeats the tile's last row
      int rows[4] = {0, 0, 0, 0};
      if (BY_TOKEN && warp == 6 && lane < quads) {
#pragma unroll
        for (int i = 0; i < 4; ++i) rows[i] = a.order[w.row0 + min(4 * lane + i, w.rows - 1)] / a.top;
      }
      const uint32_t bytes = warp == 4 ? F::W_BYTES : BY_TOKEN ? (uint32_t)quads * 512u : ROWS_FEW * 128u;
      const int w_row = w.e * a.NOUT + w.n0;
      for (int k = 0; k < slices; ++k, ++n) {
        const int st = n % F::STAGES;
        if (n >= F::STAGES) ok = mbar_wait(smem_u32(&c.empty[st]), (uint32_t)(n / F::STAGES - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint32_t bar = smem_u32(&c.full[st]), w_dst = sm + st * F::STAGE, x_dst = w_dst + F::W_BYTES;
        if (lane == 0) mbar_expect_tx(bar, bytes);
        __syncwarp();
        if (warp == 4) {
          if (lane < TILES)
            tma_load_2d(w_dst + lane * 16384, MODE == 1 && lane == 1 ? &map_w1 : &map_w0, bar, k * BK, w_row + (MODE == 1 ? 0 : lane * 128));
        } else if (BY_TOKEN) {
          if (lane < quads) tma_gather4(x_dst + lane * 512, &map_x, bar, k * BK, rows);
        } else if (lane == 0) {
          tma_load_2d(x_dst, &map_x, bar, k * BK, w.row0);
        }
      }
    }
    if (*abort_flag) let_land(c, n);
  } else if (warp == 5) {
    const uint64_t w_desc = desc_k_major(sm), x_desc = desc_k_major(sm + F::W_BYTES);
    int n = 0, turn = 0;
    bool ok = true;
    for (int it = blockIdx.x; ok && it < items; it += gridDim.x, ++turn) {
      const int acc = turn & 1;
      if (turn >= 2) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.acc_empty[acc]), (uint32_t)(turn / 2 - 1) & 1, abort_flag));
      for (int k = 0; ok && k < slices; ++k, ++n) {
        const int st = n % F::STAGES;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&c.full[st]), (uint32_t)(n / F::STAGES) & 1, abort_flag));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elect_one()) {
          const uint64_t off = (uint64_t)((st * F::STAGE) >> 4);
#pragma unroll
          for (int ks = 0; ks < BK / 16; ++ks)
#pragma unroll
            for (int t = 0; t < TILES; ++t)
              umma_bf16(c.tmem_base + acc * F::ACC + t * ROWS_FEW, w_desc + off + t * 1024 + ks * 2, x_desc + off + ks * 2, idesc(ROWS_FEW),
                        (k | ks) != 0 ? 1u : 0u);
          umma_commit(smem_u32(&c.empty[st]));
          if (k == slices - 1) umma_commit(smem_u32(&c.acc_full[acc]));
        }
        __syncwarp();
      }
    }
    let_finish(c);
  } else if (warp < 4) {
    int turn = 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x, ++turn) {
      const Item w = item_at<COLS, ROWS_FEW>(a, plan, it);
      const int acc = turn & 1;
      // lane i looks place i's pair and weight up for everybody
      const int pair_of = lane < w.rows ? a.order[w.row0 + lane] : 0;
      const float weight_of = (BY_TOKEN && a.pair_weight != nullptr && lane < w.rows) ? a.pair_weight[pair_of] : 1.f;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&c.acc_full[acc]), (uint32_t)(turn / 2) & 1, abort_flag))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t addr = c.tmem_base + ((uint32_t)(warp * 32) << 16) + acc * F::ACC;
      const int n = w.n0 + tid;  // this thread's output (of tile 0)
      for (int p0 = 0; p0 < w.rows; p0 += 8) {
        __syncwarp();  // the load from tensor memory is the whole warp's
        uint32_t v[TILES][8];
#pragma unroll
        for (int t = 0; t < TILES; ++t) tmem_ld8(addr + t * ROWS_FEW + p0, v[t]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          if (p0 + i >= w.rows) break;  // the same for the whole warp
          const int pair = __shfl_sync(0xffffffffu, pair_of, p0 + i);
          const float weight = __shfl_sync(0xffffffffu, weight_of, p0 + i);
          __nv_bfloat16* dst = a.out + (size_t)(BY_TOKEN ? w.row0 + p0 + i : pair) * a.NOUT;
          const float s0 = __uint_as_float(v[0][i]), s1 = __uint_as_float(v[TILES - 1][i]);
          // the sums are rounded to bfloat16 before the activation, as a product stored to memory would be
          if (MODE == 1) {
            if (n < a.NOUT) dst[n] = __float2bfloat16_rn(moe_gated_activation(a.act_mode, rounded(weight * s0), rounded(weight * s1), a.limit, a.alpha));
          } else {
#pragma unroll
            for (int t = 0; t < TILES; ++t) {
              const float s = t == 0 ? s0 : s1;
              if (n + t * 128 < a.NOUT)
                dst[n + t * 128] = __float2bfloat16_rn(MODE == 2 ? moe_gated_activation(a.act_mode, 0.f, rounded(weight * s), a.limit, a.alpha) : s);
            }
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&c.acc_empty[acc]));
    }
  }
  leave(c, a, F::TMEM_COLS);
}

// A [rows, K] matrix, boxes of box_rows rows of 64 entries, 128-byte swizzle (box_rows 1: for gathers)
int rows_map(const void* ptr, long long rows, int K, int box_rows, CUtensorMap* out) {
  TsEncodeTiledFn fn = ts_encode_tiled();
  if (!fn) return TS_ERR_UNSUPPORTED_SIZE;
  const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)K * 2};
  const cuuint32_t box[2] = {BK, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  return fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
             ? 0
             : TS_ERR_BAD_ARGUMENT;
}

// Bytes of dynamic shared memory behind `tiles` of ring, and the attribute that allows the most of it.
size_t shared_bytes(uint32_t ring, int E) { return ring + 1024 + (E <= SHARED_EXPERTS ? 2 * (E + 1) * sizeof(int) : 0); }
template <typename Kernel>
int allow_shared(Kernel kernel, uint32_t ring) {
  return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shared_bytes(ring, SHARED_EXPERTS));
}
// How many CTAs: at most one per item, and every expert that got a pair may have one row tile that is not full.
long long most_items(int P, int rows, const Args& a) { return ((long long)P / rows + min(a.E, P)) * a.cols; }

template <int MODE>
int launch_many(const void* A, const void* W0, const void* W1, int P, Args a, int sms, cudaStream_t s) {
  constexpr int COLS = MODE == 1 ? TN / 2 : TN;
  a.cols = (a.NOUT + COLS - 1) / COLS;
  CUtensorMap ma, m0, m1;
  int st = rows_map(W0, (long long)a.E * a.NOUT, a.K, TN / 2, &m0);
  if (!st) st = W1 != nullptr ? rows_map(W1, (long long)a.E * a.NOUT, a.K, TN / 2, &m1) : (m1 = m0, 0);
  if (!st) st = MODE == 0 ? rows_map(A, P, a.K, ROWS_MANY, &ma) : (ma = m0, 0);
  if (st) return st;
  static bool configured = false;
  if (!configured) {
    if ((st = allow_shared(moe_many_kernel<MODE>, MANY_SMEM))) return st;
    configured = true;
  }
  const long long most = most_items(P, ROWS_MANY, a);
  if (most > 0x7fffffffLL) return TS_ERR_UNSUPPORTED_SIZE;
  return ts_launch(moe_many_kernel<MODE>, dim3((unsigned)min((long long)sms, most)), dim3(many_threads(MODE)), shared_bytes(MANY_SMEM, a.E), s,
                   (const __nv_bfloat16*)A, ma, m0, m1, a);
}

template <int MODE, int TILES>
int launch_few(const void* A, int rows, const void* W0, const void* W1, int P, Args a, int sms, cudaStream_t s) {
  using F = Few<TILES>;
  constexpr int COLS = MODE == 1 ? 128 : TILES * 128, BOX = 128;
  a.cols = (a.NOUT + COLS - 1) / COLS;
  CUtensorMap mx, m0, m1;
  int st = rows_map(W0, (long long)a.E * a.NOUT, a.K, BOX, &m0);
  if (!st) st = W1 != nullptr ? rows_map(W1, (long long)a.E * a.NOUT, a.K, BOX, &m1) : (m1 = m0, 0);
  if (!st) st = rows_map(A, rows, a.K, MODE == 0 ? ROWS_FEW : 1, &mx);
  if (st) return st;
  static bool configured = false;
  if (!configured) {
    if ((st = allow_shared(moe_few_kernel<MODE, TILES>, F::SMEM))) return st;
    configured = true;
  }
  const long long most = most_items(P, ROWS_FEW, a);
  if (most > 0x7fffffffLL) return TS_ERR_UNSUPPORTED_SIZE;
  return ts_launch(moe_few_kernel<MODE, TILES>, dim3((unsigned)min((long long)sms, most)), dim3(224), shared_bytes(F::SMEM, a.E), s, mx, m0, m1, a);
}

// One tile of 128 weight rows per item instead of two where the wide items would leave SMs idle: the width whose fullest CTA
// streams the fewest weight rows.  How many experts got a pair is known on the device only; on average P pairs meet
// E (1 - (1 - 1/E)^P) of them.  Down, one / two tiles, us: 2 pairs of 16 experts of 1,024 -> 2,048 8.2 / 9.5, 128 pairs 13.8 / 10.7; 2
// to 32 pairs of 8 experts of 3,584 -> 1,024 19 / 24.  Not for gate and up, whose narrow items would be 64 outputs in boxes of 16 rows: 4 to 384
// pairs of 32 experts, 4,096 -> 2 x 1,536, 33 / 28 to 180 / 130; 32 to 1,024 of 128, 2,048 -> 2 x 768, 48 / 38 to 170 / 126.
bool narrow(int P, int E, int wide_cols, int sms) {
  const double met = E * (1.0 - pow(1.0 - 1.0 / E, (double)P));
  return ceil(met * 2 * wide_cols / sms) < 2 * ceil(met * wide_cols / sms);
}

// A: `rows` rows (tokens of the first product, places of the second)
template <int MODE>
int launch_shape(int tile_rows, const void* A, int rows, const void* W0, const void* W1, int P, const Args& a, int sms, cudaStream_t s) {
  constexpr int COLS = MODE == 1 ? 128 : 256;
  if (tile_rows == ROWS_MANY) return launch_many<MODE>(A, W0, W1, P, a, sms, s);
  if constexpr (MODE != 1)
    if (narrow(P, a.E, (a.NOUT + COLS - 1) / COLS, sms)) return launch_few<MODE, 1>(A, rows, W0, W1, P, a, sms, s);
  return launch_few<MODE, 2>(A, rows, W0, W1, P, a, sms, s);
}

}  // namespace

// Places per row tile of the two shapes: what the plan's tile_offsets must be made for.
TS_EXPORT int ts_moe_tcgen05_row_tile(int few_rows) { return few_rows ? ROWS_FEW : ROWS_MANY; }

// bfloat16 only; pair_weight null: ones; K (the inner width) must be a multiple of 8 and every base address 16-byte aligned; x has
// `tokens` rows; tile_rows: the row tile the plan was made for (one of the two above); `sms`: how many CTAs run at once;
// `error`: one int the kernel sets to 1 if one of its waits gave up.
TS_EXPORT int ts_moe_gate_up_tcgen05(const void* x, int tokens, const float* pair_weight, const int* order, const int* offsets, const int* tile_offsets,
                                     const void* gate, const void* up, void* act, int P, int E, int K, int I, int top, float limit, float alpha,
                                     int act_mode, int tile_rows, int sms, int* error, void* stream) {
  if (P <= 0) return 0;
  if (E <= 0 || K <= 0 || I <= 0 || top <= 0 || tokens <= 0 || sms <= 0 || error == nullptr || (tile_rows != ROWS_MANY && tile_rows != ROWS_FEW))
    return TS_ERR_BAD_ARGUMENT;
  if ((gate == nullptr) != (act_mode == MOE_ACT_GELU)) return TS_ERR_BAD_ARGUMENT;
  if (K % 8 || (((uintptr_t)x | (uintptr_t)gate | (uintptr_t)up) & 15) || (long long)E * I > 0x7fffffffLL - 256) return TS_ERR_UNSUPPORTED_SIZE;
  const Args a = {pair_weight, order, offsets, tile_offsets, (__nv_bfloat16*)act, error, E, K, I, top, 0, limit, alpha, act_mode};
  if (gate == nullptr) return launch_shape<2>(tile_rows, x, tokens, up, nullptr, P, a, sms, (cudaStream_t)stream);
  return launch_shape<1>(tile_rows, x, tokens, gate, up, P, a, sms, (cudaStream_t)stream);
}

TS_EXPORT int ts_moe_down_tcgen05(const void* act, const int* order, const int* offsets, const int* tile_offsets, const void* down,
                                  void* pair_out, int P, int E, int I, int N, int tile_rows, int sms, int* error, void* stream) {
  if (P <= 0) return 0;
  if (E <= 0 || I <= 0 || N <= 0 || sms <= 0 || error == nullptr || (tile_rows != ROWS_MANY && tile_rows != ROWS_FEW)) return TS_ERR_BAD_ARGUMENT;
  if (I % 8 || (((uintptr_t)act | (uintptr_t)down) & 15) || (long long)E * N > 0x7fffffffLL - 256) return TS_ERR_UNSUPPORTED_SIZE;
  const Args a = {nullptr, order, offsets, tile_offsets, (__nv_bfloat16*)pair_out, error, E, I, N, 1, 0, 0.f, 0.f, 0};
  return launch_shape<0>(tile_rows, act, P, down, nullptr, P, a, sms, (cudaStream_t)stream);
}
