// The two products of a routed feed-forward on the 5th-generation tensor cores (bfloat16, tcgen05.mma, float32
// sums in tensor memory, operands by TMA), over the plan that moe.cu makes: the (token, choice) pairs
// sorted by expert, in row tiles (of 128 places, or of 32 in steps of few tokens) that never straddle two experts.
//
// A work item is one row tile and TN weight rows: for the first product the gate rows and the up rows of the same
// TN / 2 outputs (so the activation is the epilogue), for the second TN rows of the down matrix.  CTAs are
// persistent, one per SM, and take items in turn, the columns of a row tile side by side, so that an expert's
// weights come from device memory once and from the L2 after that.  Roles in a CTA:
//   warp 4      TMA: per slice of 64 along k two boxes of weight rows and, for the second product, one box of consecutive
//               places, for the first with short row tiles the tokens' rows (tile::gather4, four rows a copy, only as many
//               as the tile has), into a ring of slices with a full and an empty mbarrier each;
//   warps 6-9   (first product, long row tiles) the tokens' rows by 16-byte cp.async in the swizzled layout.
//               Each way where it is the faster one: the copy engine takes 40 ns per gather4, which a tile of 128 rows shows
//               (16,384 pairs of 32 experts, 4,096 -> 2 x 1,536: 397 us by warps, 981 by gather4); the proxy fence behind a slice
//               waits for the younger slices' copies too, so the slices of the warps follow one another at 0.45 us, which
//               a tile of few rows shows (it then streams weights and little else);
//   warp 5      one elected lane: every tcgen05.mma (M = 128 places, N = TN, K = 16; with row tiles of 32 the other 96 rows
//               are whatever lies behind them in shared memory);
//   warps 0-3   epilogue: thread r owns place r, reads its sums from tensor memory and writes its row.
// Two accumulators take turns, so the epilogue of an item runs under the products of the next.  Rows of shared memory that no
// copy fills hold old values: a place's sums read its own row only, and places without a pair are never stored.
// The pair's routing weight multiplies the float32 sums, not the rounded input: (w x) . g = w (x . g) without
// a second rounding of x.  Every output element is one chain of sums over k in a fixed order.
//
// Bounds.  Many rows: the L2, at 48 KB a slice and SM (13 TB/s in all; 8,192 pairs of 32 experts, 4,096 -> 2 x 1,536: 241 us, 0.86
// PFLOP/s, and 121 us for down; mma.sync tiles of 128 x 128 took 863 and 450).  Few rows: the weights, at a rate
// that follows the bytes of weights in flight, hence the short row tile (16 KB of a stage would hold A otherwise): 66 pairs
// of the same experts 138 and 72 us (5.9 and 5.6 TB/s; mma.sync 153 and 86).
// Every wait is on an mbarrier fed by this CTA's own copies, MMAs and warps, bounded; one that gives up raises the
// error word, and the CTA lets its copies land, frees its tensor memory and returns.
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
__host__ __device__ constexpr bool by_warps(int mode, int bm) { return mode != 0 && bm == ROWS_MANY; }
__host__ __device__ constexpr int threads(int mode, int bm) { return by_warps(mode, bm) ? 192 + GATHER_THREADS : 192; }

template <int TN, int BM>
struct Tile {
  static constexpr uint32_t A_BYTES = BM * 128, B_BYTES = TN * 128, STAGE = A_BYTES + B_BYTES;
  static constexpr int STAGES = 216 * 1024 / STAGE;
  static constexpr uint32_t SMEM = STAGES * STAGE;
  static constexpr uint32_t TMEM_COLS = 2 * TN;
};

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

// MODE 1: gate and up; MODE 2: the first product of experts without a gate; MODE 0: down.
template <int MODE, int TN, int BM>
__global__ void __launch_bounds__(threads(MODE, BM), 1) moe_tcgen05_kernel(const __nv_bfloat16* __restrict__ x, const __grid_constant__ CUtensorMap map_a,
                                                                           const __grid_constant__ CUtensorMap map_b0,
                                                                           const __grid_constant__ CUtensorMap map_b1, const Args a) {
  using T = Tile<TN, BM>;
  constexpr bool BY_TOKEN = MODE != 0, BY_WARPS = by_warps(MODE, BM);
  constexpr int COLS = MODE == 1 ? TN / 2 : TN;  // outputs of an item
  constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
  static_assert(T::A_BYTES + T::B_BYTES >= 128 * 128, "the 128 rows that an MMA reads lie inside the stage");
  ts_pdl_wait();  // tensor memory is never held while waiting for another kernel
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_unaligned + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[T::STAGES], empty[T::STAGES], acc_full[2], acc_empty[2], all_done;
  __shared__ uint32_t tmem_base_s;
  __shared__ int abort_s;
  int* plan = a.E <= SHARED_EXPERTS ? reinterpret_cast<int*>(smem + T::SMEM) : nullptr;  // offsets and tile_offsets, looked up for every item
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    abort_s = 0;
    for (int s = 0; s < T::STAGES; ++s) {
      mbar_init(smem_u32(&full[s]), BY_WARPS ? 1 + GATHER_WARPS : 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&acc_full[i]), 1);
      mbar_init(smem_u32(&acc_empty[i]), 4);
    }
    mbar_init(smem_u32(&all_done), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  for (int i = tid; plan != nullptr && i <= a.E; i += threads(MODE, BM)) {
    plan[i] = a.offsets[i];
    plan[a.E + 1 + i] = a.tile_offsets[i];
  }
  if (warp == 0) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "r"(T::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  ts_pdl_launch_dependents();
  const uint32_t tmem_base = tmem_base_s;
  volatile int* abort_flag = &abort_s;
  const uint32_t sm = smem_u32(smem);
  const int items = a.tile_offsets[a.E] * a.cols, slices = (a.K + BK - 1) / BK;

  if (warp == 4) {
    int n = 0;  // slices asked for
    bool ok = true;
    for (int it = blockIdx.x; ok && it < items; it += gridDim.x) {
      const Item w = item_at<COLS, BM>(a, plan, it);
      const int quads = (w.rows + 3) >> 2;  // gathers of four rows; the last one repeats the tile's last row
      int rows[4] = {0, 0, 0, 0};
      if (BY_TOKEN && !BY_WARPS && lane < quads) {
#pragma unroll
        for (int i = 0; i < 4; ++i) rows[i] = a.order[w.row0 + min(4 * lane + i, w.rows - 1)] / a.top;
      }
      const uint32_t a_bytes = BY_WARPS ? 0u : BY_TOKEN ? (uint32_t)quads * 512u : T::A_BYTES;
      const int b_row = w.e * a.NOUT + w.n0;
      for (int k = 0; k < slices; ++k, ++n) {
        const int st = n % T::STAGES;
        if (n >= T::STAGES) ok = mbar_wait(smem_u32(&empty[st]), (uint32_t)(n / T::STAGES - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint32_t bar = smem_u32(&full[st]), a_dst = sm + st * T::STAGE, b_dst = a_dst + T::A_BYTES;
        if (lane == 0) mbar_expect_tx(bar, a_bytes + T::B_BYTES);
        __syncwarp();
        if (lane < 2) {
          if (MODE == 1)
            tma_load_2d(b_dst + lane * (T::B_BYTES / 2), lane == 0 ? &map_b0 : &map_b1, bar, k * BK, b_row);
          else
            tma_load_2d(b_dst + lane * (T::B_BYTES / 2), &map_b0, bar, k * BK, b_row + lane * (TN / 2));
        }
        if (!BY_TOKEN && lane == 2) tma_load_2d(a_dst, &map_a, bar, k * BK, w.row0);
        if (BY_TOKEN && !BY_WARPS && lane < quads) tma_gather4(a_dst + lane * 512, &map_a, bar, k * BK, rows);
      }
    }
    if (*abort_flag) {  // leave nothing in flight: wait (bounded, on a count of its own) for the copies already asked for
      int patience = 0;
      volatile int* own = &patience;
      for (int i = max(0, n - T::STAGES); i < n; ++i) mbar_wait(smem_u32(&full[i % T::STAGES]), (uint32_t)(i / T::STAGES) & 1, own);
    }
  } else if (BY_WARPS && warp >= 6) {
    // thread g: piece g % 8 (16 bytes) of the rows g / 8, g / 8 + 16, ... of the tile
    const int g = tid - 192, piece = g & 7, first_row = g >> 3;
    const uint32_t to = (uint32_t)first_row * 128 + (uint32_t)((piece ^ (first_row & 7)) << 4);
    constexpr int ROW_STEP = GATHER_THREADS / 8, PER = BM / ROW_STEP, AHEAD = T::STAGES - 1;
    static_assert(ROW_STEP % 8 == 0, "a thread's rows swizzle alike");
    int n = 0;
    bool ok = true;
    auto hand_over = [&](int i) {  // slice i of this warp's rows has landed and the tensor core may read it
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&full[i % T::STAGES]));
    };
    int mine_next = 0, pairs_next[PER];  // of the item after this one: its trips to the plan run under this one's slices
    auto look_up = [&](int it) {
      mine_next = 0;
      if (it >= items) return;
      const Item w = item_at<COLS, BM>(a, plan, it);
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
        const int st = n % T::STAGES;
        if (n >= T::STAGES) ok = mbar_wait(smem_u32(&empty[st]), (uint32_t)(n / T::STAGES - 1) & 1, abort_flag);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const bool real = k * BK + piece * 8 < a.K;
        const uint32_t dst = sm + st * T::STAGE + to;
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
    const uint64_t a_desc = desc_k_major(sm), b_desc = desc_k_major(sm + T::A_BYTES);
    int n = 0, turn = 0;
    bool ok = true;
    for (int it = blockIdx.x; ok && it < items; it += gridDim.x, ++turn) {
      const int acc = turn & 1;
      if (turn >= 2) ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&acc_empty[acc]), (uint32_t)(turn / 2 - 1) & 1, abort_flag));
      for (int k = 0; ok && k < slices; ++k, ++n) {
        const int st = n % T::STAGES;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&full[st]), (uint32_t)(n / T::STAGES) & 1, abort_flag));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (elect_one()) {
          const uint64_t off = (uint64_t)((st * T::STAGE) >> 4);
#pragma unroll
          for (int ks = 0; ks < BK / 16; ++ks)
            umma_bf16(tmem_base + acc * TN, a_desc + off + ks * 2, b_desc + off + ks * 2, IDESC, (k | ks) != 0 ? 1u : 0u);
          umma_commit(smem_u32(&empty[st]));
          if (k == slices - 1) umma_commit(smem_u32(&acc_full[acc]));
        }
        __syncwarp();
      }
    }
    // everything this CTA asked of the tensor core is done when this arrives: nobody leaves before
    if (elect_one()) umma_commit(smem_u32(&all_done));
    __syncwarp();
  } else if (warp < 4) {
    int turn = 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x, ++turn) {
      const Item w = item_at<COLS, BM>(a, plan, it);
      const int acc = turn & 1;
      const int r = warp * 32 + lane;
      const bool mine = r < w.rows;
      const int pair = mine ? a.order[w.row0 + r] : 0;
      const float weight = (BY_TOKEN && mine && a.pair_weight != nullptr) ? a.pair_weight[pair] : 1.f;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&acc_full[acc]), (uint32_t)(turn / 2) & 1, abort_flag))) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (warp * 32 < w.rows) {
        const uint32_t addr = tmem_base + ((uint32_t)(warp * 32) << 16) + acc * TN;
        __nv_bfloat16* dst = a.out + (size_t)(BY_TOKEN ? w.row0 + r : pair) * a.NOUT;
#pragma unroll 1
        for (int c = 0; c < COLS; c += 16) {
          uint32_t v[16], u[16];
          tmem_ld16(addr + c, v);
          if (MODE == 1) tmem_ld16(addr + COLS + c, u);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (mine && w.n0 + c < a.NOUT) {
            float y[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float s = __uint_as_float(v[i]);
              // the sums are rounded to bfloat16 before the activation, as a product stored to memory would be
              if (MODE == 1) y[i] = moe_gated_activation(a.act_mode, rounded(weight * s), rounded(weight * __uint_as_float(u[i])), a.limit, a.alpha);
              else if (MODE == 2) y[i] = moe_gated_activation(a.act_mode, 0.f, rounded(weight * s), a.limit, a.alpha);
              else y[i] = s;
            }
            store16(dst, w.n0 + c, a.NOUT, y);
          }
          __syncwarp();  // the next load from tensor memory is the whole warp's
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&acc_empty[acc]));
    }
    mbar_wait(smem_u32(&all_done), 0, abort_flag);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (abort_s != 0 && tid == 0) *a.error = 1;
  if (warp == 0) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(T::TMEM_COLS) : "memory");
  }
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

template <int MODE, int TN, int BM>
int launch(const void* A, int tokens, const void* B0, const void* B1, int P, Args a, int sms, cudaStream_t s) {
  constexpr int COLS = MODE == 1 ? TN / 2 : TN;
  a.cols = (a.NOUT + COLS - 1) / COLS;
  CUtensorMap ma, m0, m1;
  int st = MODE == 0 ? rows_map(A, P, a.K, BM, &ma) : by_warps(MODE, BM) ? 0 : rows_map(A, tokens, a.K, 1, &ma);
  if (!st) st = rows_map(B0, (long long)a.E * a.NOUT, a.K, TN / 2, &m0);
  if (!st) st = rows_map(B1 != nullptr ? B1 : B0, (long long)a.E * a.NOUT, a.K, TN / 2, &m1);
  if (st) return st;
  if (by_warps(MODE, BM)) ma = m0;  // not used
  static bool configured = false;
  const size_t smem = Tile<TN, BM>::SMEM + 1024 + (a.E <= SHARED_EXPERTS ? 2 * (a.E + 1) * sizeof(int) : 0);
  if (!configured) {
    constexpr size_t most = Tile<TN, BM>::SMEM + 1024 + 2 * (SHARED_EXPERTS + 1) * sizeof(int);
    cudaError_t e = cudaFuncSetAttribute(moe_tcgen05_kernel<MODE, TN, BM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  // at most this many items: every expert that got a pair may have one row tile that is not full
  const long long most = ((long long)P / BM + min(a.E, P)) * a.cols;
  if (most > 0x7fffffffLL) return TS_ERR_UNSUPPORTED_SIZE;
  return ts_launch(moe_tcgen05_kernel<MODE, TN, BM>, dim3((unsigned)min((long long)sms, most)), dim3(threads(MODE, BM)), smem, s,
                   (const __nv_bfloat16*)A, ma, m0, m1, a);
}

// Items of 256 weight rows, or of 128 in steps of few pairs where the wide ones would leave SMs idle: the width whose
// fullest CTA streams the fewest weight rows.  How many experts got a pair is known on the device only; on average P pairs meet
// E (1 - (1 - 1/E)^P) of them.  (16 experts, 2,048 -> 2 x 1,024, one token's 2 pairs: 20.5 us with 128, 26.6 with 256 and nearly
// twice with the 64 that would balance 16 pairs: a slice costs what it costs however few its rows.)
bool narrow(int P, int E, int cols, int sms) {
  const double met = E * (1.0 - pow(1.0 - 1.0 / E, (double)P));
  return ceil(met * 2 * cols / sms) < 2 * ceil(met * cols / sms);
}

template <int MODE>
int launch_shape(int tile_rows, const void* A, int tokens, const void* B0, const void* B1, int P, const Args& a, int sms, cudaStream_t s) {
  constexpr int COLS = MODE == 1 ? 128 : 256;
  if (tile_rows == ROWS_MANY) return launch<MODE, 256, ROWS_MANY>(A, tokens, B0, B1, P, a, sms, s);
  if (narrow(P, a.E, (a.NOUT + COLS - 1) / COLS, sms)) return launch<MODE, 128, ROWS_FEW>(A, tokens, B0, B1, P, a, sms, s);
  return launch<MODE, 256, ROWS_FEW>(A, tokens, B0, B1, P, a, sms, s);
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
  return launch_shape<0>(tile_rows, act, 0, down, nullptr, P, a, sms, (cudaStream_t)stream);
}
