// Grouped product of a mixture of experts on the 5th-generation tensor cores: y[row] = W_e x[row] for rows ordered by
// expert, cut into tiles of at most kN rows of one expert each (the list b200dec_dispatch writes).
//
// Roles as in skinny_linear_tc5.cu: 128 WEIGHT rows are the M dimension of tcgen05.mma (bf16 -> fp32), the tokens of a tile
// its N dimension, which follows the tile's row count in steps of 16, so a short tile costs only its own products.  The same
// kernel so serves prompts (kN = 256: M128 N256 K16, the full rate of the tensor core) and decode steps (kN = 64, where it
// streams the weights of the experts in use and the ring is twice as deep).
//   grid: one persistent CTA per SM; work items (tile, block of 128 weight rows), weight blocks fastest
//   warp 0, one lane   per 64 channels one TMA box of weights (128 rows, 16 KB) and the tile's rows of x in boxes of 64 or 16
//                      rows, into a ring of slots counted in bytes on `full`
//   warp 1, one lane   4 x tcgen05.mma per slot, commit on the slot's `empty`; after an item commit on `done[buffer]`
//   warps 2-5          epilogue from one of two accumulators in tensor memory (lane = weight row, column = token) while the
//                      other is being filled.  With the gated unit, gate and up rows of an output channel are neighbouring
//                      lanes and meet in one shuffle per two tokens; the token's score multiplies both (the experts'
//                      input is scaled, and the products are linear in it).
// Both products of the experts can be one launch (kMode 2, two phases of items): a kernel's start, 4.3 us, and the last round of items, which few
// CTAs have, are there once.  The tiles' items of the second phase come in the order of the first, whose epilogues count the weight
// blocks done of each tile; the fetching lane waits for its tile's before it fetches what they wrote.  Items are then drawn from a counter,
// so that a CTA only ever waits for items that running CTAs hold and have in front of any wait: it does not matter how many are resident.
// The fetching lane hands its items to the other roles through a queue of kMgQueue.
// Every wait is bounded; when one runs out its role stops, the CTA stores nothing more and sets B200KV_S_TIMEOUT.
#include <type_traits>

#include "dec_tma.cuh"
#include "tmem_ldst.cuh"

namespace b200kv {

constexpr int kMgM = 128;       // weight rows per item
constexpr int kMgStep = 64;     // channels per slot
constexpr int kMgThreads = 192;
constexpr int kMgLost = -2;
constexpr int kMgQueue = 4;     // items on their way from the fetching lane to the other roles
constexpr uint32_t kMgWBytes = kMgM * kMgStep * 2;  // 16 KB

template <int kN>
struct MgShape {
  static constexpr int kBox = kN == 256 ? 64 : 16;          // token rows per TMA box
  static constexpr int kStages = kN == 256 ? 4 : 8;
  static constexpr uint32_t kSlot = kMgWBytes + kN * kMgStep * 2;
  static constexpr uint32_t kCols = 2 * kN;                 // tensor-memory columns, two accumulators
  static constexpr size_t kSmem = kStages * kSlot + 1024 + 256;
};

__device__ __forceinline__ void mg_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
// K-major operand in the 128-byte-swizzled layout a tensor-map copy writes: rows of 128 bytes, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t mg_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(16u >> 4) << 16) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) |
         (2ull << 61);
}
// kind::f16: fp32 accumulator, bf16 A and B (both K-major), M = 128, N = n
__device__ __forceinline__ uint32_t mg_idesc(uint32_t n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24); }
__device__ __forceinline__ void mg_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}

// Until `blocks` epilogue warps have counted a tile, and so written it; false when the limit ran out.
__device__ __forceinline__ bool mg_wait_done(const int32_t* count, int blocks) {
  for (uint32_t spin = 0; spin < kDtSpin; ++spin) {
    int got;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];\n" : "=r"(got) : "l"(count) : "memory");
    if (got >= blocks) {
      asm volatile("fence.proxy.async;\n" ::: "memory");
      return true;
    }
  }
  return false;
}

// Work item: a tile of one expert's rows and a block of its weight rows.  An entry of the list that does not fit (it would be
// the product of an inconsistent routing) is reported and passed over, alike by every role.
struct MgItem {
  int e, row0, rows, m0, t;
  bool ok, second;  // second: of the second product
};
template <int kN>
__device__ __forceinline__ MgItem mg_item(const int32_t* tiles, int it, int blocks, int first_items, int blocks2, int experts, int total_rows) {
  MgItem x;
  x.second = it >= first_items;
  if (x.second) {
    it -= first_items;
    blocks = blocks2;
  }
  const int t = it / blocks;
  x.t = t;
  x.m0 = (it - t * blocks) * kMgM;
  x.e = ld_fresh(tiles + 1 + 3 * t);
  x.row0 = ld_fresh(tiles + 2 + 3 * t);
  x.rows = ld_fresh(tiles + 3 + 3 * t);
  x.ok = x.e >= 0 && x.e < experts && x.rows >= 1 && x.rows <= kN && x.row0 >= 0 && x.row0 <= total_rows - x.rows;
  return x;
}

// What a product writes and how long it is.
struct MgProduct {
  uint16_t* y;
  int out_rows, steps;
};

// Tensor maps of the weights and rows of each product.
template <int kMode>
struct MgMaps {
  CUtensorMap w[kMode == 2 ? 2 : 1], x[kMode == 2 ? 2 : 1];
};

// kMode 0: a product; 1: one with the gated unit; 2: that, then the second product on what it wrote.
template <int kN, int kMode>
__global__ void __launch_bounds__(kMgThreads, 1)
grouped_linear_tc5_kernel(const __grid_constant__ MgMaps<kMode> maps, const int32_t* tiles, int max_tiles, int experts, int total_rows,
                          const MgProduct p1, const MgProduct p2, int32_t* done, const float* score_sorted, float limit, float slope,
                          int32_t* status) {
  using S = MgShape<kN>;
  extern __shared__ uint8_t mg_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t base = (dt_smem(mg_raw) + 1023u) & ~1023u;
  const uint32_t bars = base + S::kStages * S::kSlot;
  auto bar_full = [&](int s) { return bars + 8 * s; };
  auto bar_empty = [&](int s) { return bars + 8 * (S::kStages + s); };
  auto bar_done = [&](int b) { return bars + 16 * S::kStages + 8 * b; };        // accumulator b is complete
  auto bar_free = [&](int b) { return bars + 16 * S::kStages + 16 + 8 * b; };   // ... and read (4 epilogue warps)
  const uint32_t slot_word = bars + 16 * S::kStages + 32;
  const uint32_t queue = slot_word + 8;                                          // kMgQueue items
  auto bar_item = [&](int s) { return queue + 4 * kMgQueue + 8 * s; };           // an item is in its place
  auto bar_taken = [&](int s) { return bar_item(kMgQueue + s); };                // ... and read by the issuing lane and the epilogue warps
  if (tid == 0) {
    for (int s = 0; s < S::kStages; ++s) {
      dt_mbar_init(bar_full(s), 1);
      dt_mbar_init(bar_empty(s), 1);
    }
    for (int s = 0; kMode == 2 && s < kMgQueue; ++s) {
      dt_mbar_init(bar_item(s), 1);
      dt_mbar_init(bar_taken(s), 5);
    }
    for (int b = 0; b < 2; ++b) {
      dt_mbar_init(bar_done(b), 1);
      dt_mbar_init(bar_free(b), 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(slot_word), "r"(S::kCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  uint32_t tmem;
  asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(tmem) : "r"(slot_word) : "memory");
  pdl_wait();  // the tile list and the rows come from the kernels before this one
  const int blocks = (p1.out_rows + kMgM - 1) / kMgM, blocks2 = kMode == 2 ? (p2.out_rows + kMgM - 1) / kMgM : 0;
  const int num_tiles = min(max(ld_fresh(tiles), 0), max_tiles), first_items = num_tiles * blocks, items = num_tiles * (blocks + blocks2);

  auto take = [&](int n) {  // the n-th item of this CTA, -1 behind the last, kMgLost when the wait ran out
    if (!dt_mbar_wait(bar_item(n % kMgQueue), (n / kMgQueue) & 1)) return kMgLost;
    int it;
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(it) : "r"(queue + 4 * (n % kMgQueue)) : "memory");
    return it;
  };
  if (warp == 0) {
    if (lane == 0) {
      int i = 0, n = 0;
      bool live = true;
      auto hand_on = [&](int it) {
        const int s = n % kMgQueue;
        if (n >= kMgQueue && !dt_mbar_wait(bar_taken(s), (n / kMgQueue - 1) & 1)) { live = false; return; }
        asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(queue + 4 * s), "r"(it) : "memory");
        dt_mbar_arrive(bar_item(s));
        ++n;
      };
      int it = kMode == 2 ? atomicAdd(done + max_tiles, 1) : blockIdx.x;
      MgItem drawn = {};
      if (kMode == 2 && it < items) drawn = mg_item<kN>(tiles, it, blocks, first_items, blocks2, experts, total_rows);
      while (it < items) {
        const MgItem x = kMode == 2 ? drawn : mg_item<kN>(tiles, it, blocks, first_items, blocks2, experts, total_rows);
        // the next one and its tile are on their way while this one is fetched: nothing is in flight while the lane waits for them
        const int next = kMode == 2 ? atomicAdd(done + max_tiles, 1) : it + gridDim.x;
        if (!x.ok) {
          if (status) atomicOr(status, B200KV_S_BAD_POSITION);
          it = next;
          if (kMode == 2 && it < items) drawn = mg_item<kN>(tiles, it, blocks, first_items, blocks2, experts, total_rows);
          continue;
        }
        if (kMode == 2) hand_on(it);
        if (!live) break;
        const bool second = kMode == 2 && x.second;
        const int out_rows = second ? p2.out_rows : p1.out_rows, steps = second ? p2.steps : p1.steps;
        const CUtensorMap *map_w = maps.w + second, *map_x = maps.x + second;
        if (second && !mg_wait_done(done + x.t, 4 * blocks)) live = false;
        const int boxes = (x.rows + S::kBox - 1) / S::kBox;
        const uint32_t bytes = kMgWBytes + (uint32_t)boxes * S::kBox * 128;
        for (int k = 0; k < steps && live; ++k, ++i) {
          const int s = i % S::kStages;
          if (kMode == 2 && k == steps / 2 && next < items) drawn = mg_item<kN>(tiles, next, blocks, first_items, blocks2, experts, total_rows);
          if (i >= S::kStages && !dt_mbar_wait(bar_empty(s), (i / S::kStages - 1) & 1)) { live = false; break; }
          const uint32_t dst = base + s * S::kSlot;
          dt_expect_tx(bar_full(s), bytes);
          dt_tma_2d(dst, map_w, k * kMgStep, x.e * out_rows + x.m0, bar_full(s));
          for (int b = 0; b < boxes; ++b) dt_tma_2d(dst + kMgWBytes + b * S::kBox * 128, map_x, k * kMgStep, x.row0 + b * S::kBox, bar_full(s));
        }
        if (!live) break;
        it = next;
      }
      if (kMode == 2 && live) hand_on(-1);
      pdl_trigger();  // nothing left to fetch: the next kernel may be brought up
      if (!live) {    // the copies in flight land before the CTA may end
        if (status) atomicOr(status, B200KV_S_TIMEOUT);
        for (int k = i > S::kStages ? i - S::kStages : 0; k < i; ++k) dt_mbar_wait(bar_full(k % S::kStages), (k / S::kStages) & 1);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int i = 0, n = 0;
      bool live = true;
      for (int at = blockIdx.x; live; at += gridDim.x) {
        const int it = kMode == 2 ? take(n) : (at < items ? at : -1);
        if (it < 0) break;
        if (kMode == 2) dt_mbar_arrive(bar_taken(n % kMgQueue));
        const MgItem x = mg_item<kN>(tiles, it, blocks, first_items, blocks2, experts, total_rows);
        if (kMode < 2 && !x.ok) continue;
        const int buf = n & 1, steps = kMode == 2 && x.second ? p2.steps : p1.steps;
        const uint32_t idesc = mg_idesc((uint32_t)((x.rows + 15) & ~15));
        if (n >= 2 && !dt_mbar_wait(bar_free(buf), (n / 2 - 1) & 1)) break;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        for (int k = 0; k < steps; ++k, ++i) {
          const int s = i % S::kStages;
          if (!dt_mbar_wait(bar_full(s), (i / S::kStages) & 1)) { live = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
          const uint64_t da = mg_desc(base + s * S::kSlot), db = mg_desc(base + s * S::kSlot + kMgWBytes);
#pragma unroll
          for (int j = 0; j < kMgStep / 16; ++j)
            mg_mma(tmem + buf * kN, da + (uint64_t)((j * 32) >> 4), db + (uint64_t)((j * 32) >> 4), idesc, (k | j) != 0);
          mg_commit(bar_empty(s));
        }
        if (live) mg_commit(bar_done(buf));
        ++n;
      }
    }
  } else {
    int n = 0;
    const int wl = warp & 3;  // tensor-memory lanes 32 wl ..
    for (int at = blockIdx.x;; at += gridDim.x) {
      int it = kMode == 2 ? take(n) : (at < items ? at : -1);
      if (kMode == 2) {
        // each lane has a limit of its own: where one's ran out the warp stops as a whole, as its lanes vote and load tensor memory together
        if (__any_sync(0xffffffffu, it == kMgLost)) it = kMgLost;
        if (lane == 0 && it >= 0) dt_mbar_arrive(bar_taken(n % kMgQueue));
        if (it == kMgLost && lane == 0 && status) atomicOr(status, B200KV_S_TIMEOUT);
      }
      if (it < 0) break;
      const MgItem x = mg_item<kN>(tiles, it, blocks, first_items, blocks2, experts, total_rows);
      if (kMode < 2 && !x.ok) continue;
      const bool second = kMode == 2 && x.second, act = kMode > 0 && !second;
      const int buf = n & 1, row0 = x.row0, rows = x.rows, out_rows = second ? p2.out_rows : p1.out_rows;
      uint16_t* y = second ? p2.y : p1.y;
      const int o = x.m0 + 32 * wl + lane;  // this lane's weight row
      const bool ok = dt_mbar_wait(bar_done(buf), (n / 2) & 1);
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0 && status) atomicOr(status, B200KV_S_TIMEOUT);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      for (int c0 = 0; c0 < rows; c0 += 32) {
        uint32_t u[32];
        t5_ld32(tmem + buf * kN + c0 + ((uint32_t)(32 * wl) << 16), u);
        if (act) {
          const float sl = c0 + lane < rows ? ld_fresh(score_sorted + row0 + c0 + lane) : 0.f;
          const bool odd = lane & 1;
          uint16_t* dst = y + (long long)(row0 + c0 + odd) * (out_rows / 2) + o / 2;
#pragma unroll
          for (int c = 0; c < 32; c += 2) {
            const float a = __uint_as_float(u[c]) * __shfl_sync(0xffffffffu, sl, c);
            const float b = __uint_as_float(u[c + 1]) * __shfl_sync(0xffffffffu, sl, c + 1);
            const float got = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
            const float g = fminf(odd ? got : a, limit), up = fminf(fmaxf(odd ? b : got, -limit), limit);
            const float v = __fdividef(g, 1.0f + __expf(-slope * g)) * (up + 1.0f);
            if (c0 + c + odd < rows && o < out_rows) *dst = (uint16_t)float_to_bf16_bits(v);
            dst += out_rows;  // two tokens further: 2 * (out_rows / 2)
          }
        } else {
          uint16_t* dst = y + (long long)(row0 + c0) * out_rows + o;
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            if (c0 + c < rows && o < out_rows) *dst = (uint16_t)float_to_bf16_bits(__uint_as_float(u[c]));
            dst += out_rows;
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      if (kMode == 2 && !second) {  // what this lane wrote, before any copy that starts behind the count
        __threadfence();
        asm volatile("fence.proxy.async;\n" ::: "memory");
      }
      __syncwarp();
      if (lane == 0) {
        dt_mbar_arrive(bar_free(buf));
        if (kMode == 2 && !second) asm volatile("red.release.gpu.global.add.s32 [%0], 1;\n" ::"l"(done + x.t) : "memory");
      }
      ++n;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(S::kCols) : "memory");
}

static bool mg_maps(CUtensorMap* tm_w, CUtensorMap* tm_x, const void* w, const void* x, int experts, int out_rows, int width, int total_rows, int box) {
  const uint64_t wd[2] = {(uint64_t)width, (uint64_t)experts * out_rows}, xd[2] = {(uint64_t)width, (uint64_t)total_rows};
  const uint64_t st[1] = {(uint64_t)width};
  const uint32_t wb[2] = {kMgStep, kMgM}, xb[2] = {kMgStep, (uint32_t)box};
  return dt_make_map(tm_w, w, 2, wd, st, wb) && dt_make_map(tm_x, x, 2, xd, st, xb);
}
static MgProduct mg_product(void* y, int out_rows, int width) { return MgProduct{(uint16_t*)y, out_rows, (width + kMgStep - 1) / kMgStep}; }

template <int kMode>
static int mg_launch(const MgMaps<kMode>& maps, const int32_t* tiles, int max_tiles, int tile_rows, int experts, int total_rows,
                     const MgProduct& p1, const MgProduct& p2, int32_t* done, const float* score_sorted, float limit, float slope, int sms,
                     int32_t* status, cudaStream_t stream) {
  const long long blocks = (p1.out_rows + kMgM - 1) / kMgM + (kMode == 2 ? (p2.out_rows + kMgM - 1) / kMgM : 0), items = max_tiles * blocks;
  if (items > 0x7FFFFFFFll) return B200KV_E_RANGE;
  const int grid = (int)(items < sms ? items : sms);
  auto run = [&](auto* kernel, size_t smem) -> int {
    if (!allow_smem(kernel, smem)) return B200KV_E_LAUNCH;
    return launch_result(launch_chained(kernel, dim3(grid), dim3(kMgThreads), smem, stream, maps, tiles, max_tiles, experts,
                                        total_rows, p1, p2, done, score_sorted, limit, slope, status));
  };
  return tile_rows > 64 ? run(grouped_linear_tc5_kernel<256, kMode>, MgShape<256>::kSmem)
                        : run(grouped_linear_tc5_kernel<64, kMode>, MgShape<64>::kSmem);
}
static int mg_box(int tile_rows) { return tile_rows > 64 ? MgShape<256>::kBox : MgShape<64>::kBox; }

int launch_grouped_linear_tc5(const void* x, const void* w, const int32_t* tiles, int max_tiles, int tile_rows, int total_rows, int experts,
                              int out_rows, int width, const float* score_sorted, int act, float limit, float slope, void* y, int sms,
                              int32_t* status, cudaStream_t stream) {
  if (tile_rows > 256) return B200KV_E_SHAPE;
  if ((long long)experts * out_rows > 0x7FFFFFFFll) return B200KV_E_RANGE;
  const MgProduct p = mg_product(y, out_rows, width);
  auto run = [&](auto mode) -> int {
    MgMaps<decltype(mode)::value> m;
    if (!mg_maps(m.w, m.x, w, x, experts, out_rows, width, total_rows, mg_box(tile_rows))) return B200KV_E_LAUNCH;
    return mg_launch(m, tiles, max_tiles, tile_rows, experts, total_rows, p, p, nullptr, score_sorted, limit, slope, sms, status, stream);
  };
  return act ? run(std::integral_constant<int, 1>{}) : run(std::integral_constant<int, 0>{});
}

int launch_expert_products_tc5(const void* x, const void* gate_up, const void* down, const int32_t* tiles, int max_tiles, int tile_rows,
                               int total_rows, int experts, int ff, int width, const float* score_sorted, float limit, float slope, void* h,
                               void* y, int32_t* done, int sms, int32_t* status, cudaStream_t stream) {
  if (tile_rows > 256) return B200KV_E_SHAPE;
  if ((long long)experts * 2 * ff > 0x7FFFFFFFll || (long long)experts * width > 0x7FFFFFFFll) return B200KV_E_RANGE;
  MgMaps<2> m;
  const int box = mg_box(tile_rows);
  if (!mg_maps(m.w, m.x, gate_up, x, experts, 2 * ff, width, total_rows, box) || !mg_maps(m.w + 1, m.x + 1, down, h, experts, width, ff, total_rows, box))
    return B200KV_E_LAUNCH;
  return mg_launch(m, tiles, max_tiles, tile_rows, experts, total_rows, mg_product(h, 2 * ff, width), mg_product(y, width, ff), done,
                      score_sorted, limit, slope, sms, status, stream);
}

}  // namespace b200kv
