// Chunked-prefill attention on the 5th-generation tensor cores (tcgen05 + tensor memory).
// Same contract as prefill_attn_kernel (prefill_attn.cu): packed variable-length causal
// attention of the prefilling entries over [dequantized prefix | own chunk], replacing
// prefill_attention_kernel (qwen3-1.7b/kernels.py:987-1126).
//
// One CTA owns 128 query rows of one q head and runs twelve warps in three roles:
//   warps 0-3 and 4-7   two softmax warpgroups.  The keys of the tile are cut into blocks of 64 and dealt
//                       alternately to the two; each keeps its own running (offset, sum, O) and the two are
//                       merged at the end.  Thread t of a warpgroup owns query row t = lane t of tensor
//                       memory: every row-wise softmax quantity lives in one thread, no shuffles.
//   warps 8 and 9       one lane of each issues every tcgen05.mma of warpgroup 0 and 1.
//   warps 10 and 11     fetch the K and V tiles of warpgroup 0 and 1 (tensor-map copies started by one lane).
// Per key block h of a warpgroup:
//   S(h) = Q K^T   8 x tcgen05.mma (M128 N64 K16, bf16 -> fp32), Q and K from shared memory, into one of the
//                  warpgroup's two S buffers (64 tensor-memory columns each)
//   softmax        one tcgen05.ld of the thread's 64 scores, max, exp2, sum; P rounded to bf16 as the
//                  reference does (kernels.py:1068,1113) and stored over the first 32 columns of the same
//                  S buffer
//   O += P V       4 x tcgen05.mma (M128 N128 K16) with P read from tensor memory and V from shared memory
//                  (channel-contiguous: N-major B operand), accumulating in the warpgroup's 128 O columns
// The products are software-pipelined against the softmax: when P(h) is stored (128 arrivals on a `ready`
// barrier), the issuing lane queues P V(h) and then S(h+2) into the buffer P(h) occupies (the tensor core
// executes one thread's products in issue order), while S(h+1) is already complete or running in the other
// buffer; the warpgroup goes from one softmax straight into the next.  Completions come back through
// tcgen05.commit on mbarriers: `s_done` to the softmax threads, `kempty` / `vempty` to the fetching warp,
// which refills the ring slot (three K and three V tiles of 16 KB per warpgroup) and reports on `kfull` /
// `vfull`.  Measured on a B200 an M128 N64 K16 product from shared memory takes 49 cycles and an
// M128 N128 K16 one 65 (the latter is the nominal rate; the former is bound by the 128 B/clk the tensor
// core reads shared memory at), so one block pair costs the tensor core about 1300 cycles.
// O stays in tensor memory for the whole tile.  Its rescaling is lazy: the reference offset of the
// exponentials only moves when the row maximum has grown by more than 2^8 since it was set (then, after
// waiting for the one P V that may be in flight, O and the sum are multiplied by the correction, a
// tensor-memory round trip); otherwise P is simply computed against the older offset, which is the same
// mathematics.
//
// Q, K and V tiles are laid out in shared memory as the canonical 128-byte-swizzled layout the matrix
// descriptors name: two blocks of 64 channels, each [row][128 bytes] with the 16-byte chunk index XOR-ed
// with (row & 7) - which is also what a tensor-map copy with the 128-byte swizzle writes.  K and V use the
// same physical layout; only their descriptors differ (K: K-major, rows = N; V: N-major, rows = K).
// A prefix block that is not full is copied with cp.async and zero-filled instead (see the fetching warp).
//
// The kernel has two forms.  The dense one (kPaged = false, prefill_attn_tc5.cu) attends [prefix | own chunk] as above with
// head size 128.  The paged one (kPaged = true, paged_prefill_tc5.cu) reads keys and values of the whole sequence, the
// chunk's own included, by page from a cache of bf16 rows, with key and value sizes of up to 128 each: copies beyond a
// size read as zero, products run over the blocks of 64 channels there are, and a query at position p sees keys 0..p.
// With kOptions a sliding window leaves out the blocks in front of the tile's first row's window and masks the rest, a
// sink is what the first warpgroup's softmax state starts from, and the output gate multiplies in the last step.
//
// Every wait on an mbarrier is bounded: if a completion never arrives the waiting role records it, stops
// issuing work and the CTA skips its stores, sets B200KV_S_TIMEOUT in the status word, frees its tensor
// memory and returns.
#pragma once
#include <cuda.h>  // CUtensorMap and the cuTensorMapEncodeTiled prototype only; the entry point is fetched at run time

#include "common.cuh"
#include "dec_common.cuh"
#include "tmem_ldst.cuh"

namespace b200kv {

constexpr int kT5Threads = 384;                       // two softmax warpgroups, two warps issuing products, two fetching tiles
constexpr int kT5Tile = 128;                         // query rows per CTA
constexpr int kT5Keys = 64;                          // keys per block
constexpr uint32_t kT5QBytes = kT5Tile * kD * 2;     // Q tile: 32 KB, two 64-channel blocks of 16 KB
constexpr uint32_t kT5KvBytes = kT5Keys * kD * 2;    // K or V tile: 16 KB, two 64-channel blocks of 8 KB
constexpr uint32_t kT5WgBytes = 6 * kT5KvBytes;      // per warpgroup: K ring of 3, V ring of 3
constexpr uint32_t kT5Smem = kT5QBytes + 2 * kT5WgBytes + 1024 /* alignment slack */ + 384 /* barriers, flags */;
constexpr uint32_t kT5Cols = 512;                    // tensor memory: warpgroup w has S0/P0 at 256w, S1/P1 at 256w+64, O at 256w+128
constexpr uint32_t kT5SpinLimit = 1u << 20;
constexpr float kT5Lazy = 8.f;                      // log2 of the growth of the row maximum that forces a rescale

__device__ __forceinline__ uint32_t t5_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void t5_cp16(uint32_t dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void t5_commit_group() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void t5_wait_group() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ void t5_fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
__device__ __forceinline__ void t5_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void t5_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

__device__ __forceinline__ void t5_mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
// Bounded wait for the phase with the given parity; false when the limit ran out.  Each lane has a limit of its own, so a warp whose lanes go on
// to do something together votes on the outcome.
__device__ __forceinline__ bool t5_mbar_wait(uint32_t bar, uint32_t parity, uint32_t limit) {
  for (uint32_t spin = 0; spin < limit; ++spin) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void t5_mbar_arrive(uint32_t bar) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}\n" ::"r"(bar) : "memory");
}
// One arrival that also announces `bytes` of bulk-copy traffic the phase has to see before it completes.
__device__ __forceinline__ void t5_mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}\n" ::"r"(bar), "r"(bytes) : "memory");
}
// Tensor-map (TMA) tile load of one box into shared memory; completion is counted in bytes on `bar`.
// c0 (the channel coordinate) must keep the 16-byte rule: it is 0 or 64 bf16 here.
__device__ __forceinline__ void t5_tma_3d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
// Arrive on `bar` when every tcgen05.mma issued so far by this thread has completed.
__device__ __forceinline__ void t5_mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}

// Shared-memory matrix descriptor: 128-byte swizzle, start address / leading / stride byte offsets
// in units of 16 bytes, descriptor version 1.
__device__ __forceinline__ uint64_t t5_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo_bytes >> 4) << 16) | ((uint64_t)(sbo_bytes >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}
// Instruction descriptor of kind::f16: fp32 accumulator, bf16 A and B, M = 128, N as given.
__host__ __device__ constexpr uint32_t t5_idesc(uint32_t n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24); }
constexpr uint32_t kT5IdescQK = t5_idesc(kT5Keys);        // A (Q) K-major, B (K tile) K-major, N = 64 keys
constexpr uint32_t kT5IdescPV = t5_idesc(kD) | (1u << 16); // B (V tile) N-major, N = 128 channels

__device__ __forceinline__ void t5_mma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void t5_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}

__device__ __forceinline__ float t5_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
// Two 32-bit numbers in one register pair.
typedef unsigned long long t5_pair;
__device__ __forceinline__ t5_pair t5_two(float a, float b) {
  t5_pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void t5_split(t5_pair p, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p)); }
__device__ __forceinline__ t5_pair t5_fma2(t5_pair a, t5_pair b, t5_pair c) {
  t5_pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ t5_pair t5_add2(t5_pair a, t5_pair b) {
  t5_pair r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float t5_max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ uint32_t t5_pack_bf16x2(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// Copied by kThreads threads (tid in [0, kThreads)): `count` (<= kRows) rows of 8 * cols (<= 128) bf16 (row j at
// src + j*stride elements) into a swizzled tile of kRows rows; what lies past `count` or `cols` is zero-filled.
template <int kThreads, int kRows>
__device__ __forceinline__ void t5_load_tile(uint32_t dst, const uint16_t* src, long long stride, int count, int tid, int cols = 16) {
#pragma unroll
  for (int i = 0; i < (kRows * 16) / kThreads; ++i) {
    const int c = tid + i * kThreads, r = c >> 4, col = c & 15;
    const bool valid = r < count && col < cols;
    const uint32_t d = dst + (col >> 3) * (kRows * 128) + r * 128 + (((col & 7) ^ (r & 7)) << 4);
    t5_cp16(d, valid ? src + r * stride + col * 8 : src, valid ? 16 : 0);
  }
}

__device__ __forceinline__ void t5_wg_sync(int wg) { asm volatile("bar.sync %0, 128;\n" ::"r"(wg + 1) : "memory"); }
__device__ __forceinline__ void t5_sts_u32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t t5_lds_u32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(addr) : "memory");
  return v;
}

// What the paged form adds: the cache, the entries' cached lengths and the rows of a tensor-map box.
struct T5Paged {
  DecCache c;
  const int32_t* cached_lens;
  int box_rows;
  DecAttnOpt opt;
};

// With more CTAs of one head and tile than multiprocessors, the CTAs of tiles with few keys do two heads each, one a warpgroup: what
// comes in front of and behind a CTA's products (Q, the first tiles, the last P V, the merge of the warpgroups, which falls away)
// is as long as its products then, and is there once instead of twice.  16 heads in bf16, us per pass with the row writes: five portions
// of 1000 rows 34.9 -> 25.0, and on 2000 cached keys 53.3 -> 37.0; two portions on 4000 114 -> 90.  With
// tiles of up to 6 blocks only that second one took 53.4, with 10 41.1 and with 16 as long, and the first 27.9 and 28.7 (before the loops
// behind the products were rolled up).
constexpr int kT5PairBlocks = 10;

template <bool kPaged, int kKeyBlocks = 2, bool kOptions = false>  // kKeyBlocks: 64-channel blocks of a key (2 covers up to 128 channels)
__global__ void __launch_bounds__(kT5Threads, 1)
prefill_attn_tc5_kernel(const uint16_t* q, long long q_sn, long long q_sh, const uint16_t* k,
                        long long k_sn, long long k_sh, const uint16_t* v, long long v_sn, long long v_sh,
                        const int32_t* __restrict__ seq_ids, const int32_t* __restrict__ cu_seqlens,
                        const int32_t* __restrict__ tile_start, int block_m, int subs,
                        const uint16_t* k_prefix, const uint16_t* v_prefix, long long p_sh,
                        long long p_sn, const int32_t* __restrict__ cu_cached, uint16_t* __restrict__ out, long long o_sn,
                        long long o_sh, int N, int G, float scale_log2, int32_t* status,
                        const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                        const __grid_constant__ CUtensorMap tm_kp, const __grid_constant__ CUtensorMap tm_vp, int prefix_tma,
                        int idle_issuers, int full_tiles, const __grid_constant__ T5Paged pg) {
  extern __shared__ uint8_t t5_raw[];
  // idle_issuers (a test mode): the issuing warps do nothing and every wait gives up after a few thousand polls,
  // so that all bounded waits of the kernel run out and the time-out path is exercised without a fault
  const uint32_t spin = idle_issuers ? 4096u : kT5SpinLimit;
  // The first CTA waits for the predecessor on every path (a grid in which no CTA waited could complete before
  // it); the trigger for the successor comes late, from the softmax threads when their last block is done: a
  // successor brought up while this kernel is in full swing would only sit on the SMs.
  if ((blockIdx.x | blockIdx.y) == 0) pdl_wait();
  // heads run fastest in the grid: the caller's real tiles come first in tile_start, so every CTA with work
  // is dispatched before the idle ones behind them
  const int tile = blockIdx.y / subs, sub = blockIdx.y - tile * subs, Hq = gridDim.x;
  // full_tiles: the tiles with which every CTA of one head and tile has a multiprocessor of its own (the real tiles come first)
  const int past = full_tiles * subs < (int)gridDim.y ? tile_start[full_tiles] : -1;
  const int tile_row = tile_start[tile];
  if (tile_row < 0 || tile_row >= N) return;
  const int seq = seq_ids[tile_row];
  // a step in which no entry has a cached prefix may pass empty prefix tensors (no storage: NULL pointers)
  const int prefix_start = kPaged ? 0 : cu_cached[seq], prefix_len = (!kPaged && k_prefix && v_prefix) ? cu_cached[seq + 1] - prefix_start : 0;
  const int cached = kPaged ? pg.cached_lens[seq] : 0;  // keys in front of the chunk's first row, in the same list
  const int vdim = kPaged ? pg.c.v_dim : kD;
  const int seq_start = cu_seqlens[seq], seq_end = min(cu_seqlens[seq + 1], N);
  const int row_end = min(tile_row + block_m, seq_end);
  const int row0 = tile_row + sub * kT5Tile;  // first query row of this CTA
  if (row0 >= row_end) return;
  const int cta_last = min(row0 + kT5Tile, row_end) - 1;
  const int own_keys = cached + cta_last - seq_start + 1;  // causal: keys up to the CTA's last query
  const int nb_pre = (prefix_len + kT5Keys - 1) / kT5Keys, nb_own = (own_keys + kT5Keys - 1) / kT5Keys;
  // blocks in front of every row's window
  const int skipped = kOptions && pg.opt.window > 0 ? max(0, cached + row0 - seq_start - pg.opt.window + 1) / kT5Keys : 0;
  const int nb = nb_pre + nb_own - skipped;
  // Each warpgroup a head of its own (pair), or both the keys of one?
  const bool pair = past >= 0 && past < N && nb <= kT5PairBlocks;
  if (pair && 2 * (int)blockIdx.x >= Hq) return;
  auto head = [&](int w) { return pair ? min(2 * (int)blockIdx.x + w, Hq - 1) : (int)blockIdx.x; };

  float m_ref_keep = -INFINITY, l_keep = 0.f;
  // roles: warps 0-3 and 4-7 = softmax warpgroups 0 and 1, warps 8 and 9 = issue the products of warpgroup 0
  // and 1, warps 10 and 11 = fetch the K and V tiles of warpgroup 0 and 1
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wg = tid >> 7, wt = tid & 127;
  // warpgroup w owns blocks w, w + 2, ..., or all of its own head (one head too few: none)
  auto n_blk = [&](int w) { return pair ? (2 * (int)blockIdx.x + w < Hq ? nb : 0) : (nb + 1 - w) >> 1; };
  auto block_of = [&](int w, int h) { return pair ? h : w + 2 * h; };
  const int ring = pair ? 2 : 3;  // slots of a ring; a pair has a second Q tile where the third ones were
  const uint32_t base = (t5_smem_u32(t5_raw) + 1023u) & ~1023u;
  auto q_tile = [&](int w) { return base + (pair ? w * kT5QBytes : 0u); };
  const uint32_t rings = base + (pair ? 2 * kT5QBytes : kT5QBytes);
  const uint32_t bars = base + kT5QBytes + 2 * kT5WgBytes;
  // per warpgroup w, 18 barriers at bars + 144 w:
  //   s_done[2]  S buffer b holds a complete S (arrival = tcgen05.commit)
  //   o_done[2]  the last-but-one and the last P V are complete (one phase each: a parity wait must never fall
  //              two phases behind, so these two do not share a barrier)
  //   ready[2]   P is stored in S buffer b (128 arrivals)
  //   kfull[3], vfull[3]    ring slot holds its tile (one arrival by the fetching warp, plus the tile's bytes
  //                         when it is a tensor-map copy)
  //   kempty[3], vempty[3]  the product that read the slot is complete (tcgen05.commit)
  auto ring_k = [&](int w) { return rings + w * 2 * ring * kT5KvBytes; };
  auto ring_v = [&](int w) { return ring_k(w) + ring * kT5KvBytes; };
  auto bar_s = [&](int w, int buf) { return bars + 144 * w + 8 * buf; };
  auto bar_o = [&](int w, int which) { return bars + 144 * w + 16 + 8 * which; };
  auto bar_r = [&](int w, int buf) { return bars + 144 * w + 32 + 8 * buf; };
  auto bar_kf = [&](int w, int sl) { return bars + 144 * w + 48 + 8 * sl; };
  auto bar_vf = [&](int w, int sl) { return bars + 144 * w + 72 + 8 * sl; };
  auto bar_ke = [&](int w, int sl) { return bars + 144 * w + 96 + 8 * sl; };
  auto bar_ve = [&](int w, int sl) { return bars + 144 * w + 120 + 8 * sl; };
  const uint32_t bar_q = bars + 288;  // the Q tile has landed (256 arrivals)
  const uint32_t slot = bars + 296, dead_flag = bars + 304;

  if (tid == 0) {
    for (int w = 0; w < 2; ++w) {
      for (int i = 0; i < 18; ++i) t5_mbar_init(bars + 144 * w + 8 * i, (i == 4 || i == 5) ? 128 : 1);  // 4, 5: ready
    }
    t5_mbar_init(bar_q, 256);
    t5_sts_u32(dead_flag, 0);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(slot), "r"(kT5Cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  t5_fence_before();
  __syncthreads();  // barriers and the tensor-memory base are visible to every role
  t5_fence_after();
  pdl_wait();  // q, k, v and the prefix come from the kernels before this one; only metadata was read so far
  const uint32_t tmem = t5_lds_u32(slot);
  bool dead = false;
  if (wg < 2) {
    // The softmax threads copy the Q tile while the fetching warps already stream K and V.  Q rows past the end
    // of the packed batch are zero-filled; rows of other entries inside the tile are read and computed but
    // never stored.
    // a pair's warpgroups bring a tile each, others one half of the same
    const int half = pair ? 0 : wg * (kT5Tile / 2), rows = min(kT5Tile, N - row0), cols = kPaged ? pg.c.k_row / 8 : 16;
    const uint16_t* src = q + (long long)row0 * q_sn + head(wg) * q_sh;
    const int col = wt & 15;
    const uint32_t to = q_tile(wg) + (col >> 3) * (kT5Tile * 128);
#pragma unroll 8
    for (int r = half + (wt >> 4); r < half + (pair ? kT5Tile : kT5Tile / 2); r += 8) {
      const bool valid = r < rows && col < cols;
      t5_cp16(to + r * 128 + (((col & 7) ^ (r & 7)) << 4), valid ? src + r * q_sn + col * 8 : src, valid ? 16 : 0);
    }
    t5_commit_group();
    t5_wait_group<0>();
    t5_fence_async_smem();
    t5_mbar_arrive(bar_q);
  }

  if (warp >= 10) {
    // ---- a fetching warp: streams the K and V tiles of warpgroup w into its rings.  Block h of the warpgroup
    // is block w + 2h (of a pair: h) of the tile and lives in slot h % ring.  Full tiles come by tensor-map copies started by
    // lane 0 (two boxes of 64 rows x 64 channels, swizzled by the copy engine into the layout described
    // above).  A prefix block that is not full is copied by the warp's 32 lanes with cp.async instead, because
    // the rows behind a prefix may be uninitialised memory and have to be zero in shared memory (0 x NaN would
    // poison O); so is every prefix block when the caller gave no row capacity for the prefix tensors.
    const int w = warp - 10, n = n_blk(w), hk = head(w) / G;
    const uint16_t* kpre = k_prefix + hk * p_sh + (long long)prefix_start * p_sn;
    const uint16_t* vpre = v_prefix + hk * p_sh + (long long)prefix_start * p_sn;
    const uint16_t* kown = k + (long long)seq_start * k_sn + hk * k_sh;
    const uint16_t* vown = v + (long long)seq_start * v_sn + hk * v_sh;
    bool live = true;
    if constexpr (kPaged) {
      // A step is a chain of instructions of one warp beside two busy softmax warps.  With the divisions and the page table in
      // it the chain took 2200 cycles and the kernel waited for it, so places are found 32 boxes of rows at a time, a box
      // per lane, and handed to the issuing lane.  A step fetches the K of a block and the V of the one in front: the K slot
      // is free when S is complete, a product before the V slot.  992 rows on 3072, 16 heads: 52.6 -> 41.5 us; five prompts
      // of 1000 rows on up to 2000: 49.9 -> 39.0.
      const int R = pg.box_rows, lg = R == 64 ? 0 : (R == 32 ? 1 : 2), boxes = 1 << lg;  // boxes of a block
      const int v_blocks = vdim > 64 ? 2 : 1;
      int my_ph = 0, my_row = 0;     // this lane's box: (page, head) and the first row there
      int k_ph[4], k_row[4];         // the boxes of the block at hand
      int k_sl = 0, k_par = 1, v_sl = 0, v_par = 1;
#pragma unroll
      for (int x = 0; x < 4; ++x) k_ph[x] = k_row[x] = 0;
      for (int step = 0; step <= n; ++step) {
        int v_ph[4], v_row[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) { v_ph[x] = k_ph[x]; v_row[x] = k_row[x]; }
        if (step < n) {
          if (((step << lg) & 31) == 0) {
            const int box = (step << lg) + lane, j = (block_of(w, box >> lg) + skipped) * kT5Keys + (box & (boxes - 1)) * R;
            const int col = j / pg.c.P;
            int page = 0;
            if (j < own_keys) {
              page = col < pg.c.max_pages ? pg.c.table[(long long)seq * pg.c.table_stride + col] : -1;
              if (page < 0 || page >= pg.c.num_pages) {  // reported, and page 0 read in its place
                if (status) atomicOr(status, col < pg.c.max_pages ? B200KV_S_BAD_PAGE : B200KV_S_BAD_POSITION);
                page = 0;
              }
            }
            my_row = j - col * pg.c.P;
            my_ph = page * pg.c.heads + hk;
          }
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            if (x >= boxes) break;
            k_ph[x] = __shfl_sync(0xffffffffu, my_ph, ((step << lg) + x) & 31);
            k_row[x] = __shfl_sync(0xffffffffu, my_row, ((step << lg) + x) & 31);
          }
          if (step >= ring && !__all_sync(0xffffffffu, t5_mbar_wait(bar_ke(w, k_sl), k_par, spin))) { live = false; break; }
          if (lane == 0) {
            // keys behind the last one may be anything: their scores are never looked at
            const int count = min(kT5Keys, own_keys - (block_of(w, step) + skipped) * kT5Keys);
            const int some = count == kT5Keys ? boxes : (count + R - 1) / R;
            const uint32_t dst = ring_k(w) + k_sl * kT5KvBytes, full = bar_kf(w, k_sl);
            t5_mbar_expect_tx(full, (uint32_t)(some * R * 128 * kKeyBlocks));
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              if (x >= some) break;
#pragma unroll
              for (int bl = 0; bl < kKeyBlocks; ++bl)
                t5_tma_3d(dst + bl * (kT5Keys * 128) + x * R * 128, &tm_k, 64 * bl, k_row[x], k_ph[x], full);
            }
          }
          __syncwarp();
        }
        if (step > 0) {
          const int j0 = (block_of(w, step - 1) + skipped) * kT5Keys, count = min(kT5Keys, own_keys - j0);
          const uint32_t dst = ring_v(w) + v_sl * kT5KvBytes, full = bar_vf(w, v_sl);
          if (step > ring && !__all_sync(0xffffffffu, t5_mbar_wait(bar_ve(w, v_sl), v_par, spin))) { live = false; break; }
          if (count == kT5Keys) {
            if (lane == 0) {
              t5_mbar_expect_tx(full, (uint32_t)(kT5Keys * 128 * v_blocks));
#pragma unroll
              for (int x = 0; x < 4; ++x) {
                if (x >= boxes) break;
                t5_tma_3d(dst + x * R * 128, &tm_v, 0, v_row[x], v_ph[x], full);
                if (v_blocks > 1) t5_tma_3d(dst + kT5Keys * 128 + x * R * 128, &tm_v, 64, v_row[x], v_ph[x], full);
              }
            }
          } else {  // values behind the last key must be zero in shared memory (0 x NaN would poison O)
            // (a lane keeps its 16-byte column and takes every other row; this ends nearly every tile)
            const int col = lane & 15;
            const bool some = col < pg.c.v_row / 8;
            const uint32_t to = dst + (col >> 3) * (kT5Keys * 128);
#pragma unroll
            for (int x = 0; x < 4; ++x) {
              if (x >= boxes) break;
              const uint16_t* src = (const uint16_t*)pg.c.v + ((long long)v_ph[x] * pg.c.P + v_row[x] + (lane >> 4)) * pg.c.v_row + (some ? col * 8 : 0);
#pragma unroll 4
              for (int r = x * R + (lane >> 4); r < (x + 1) * R; r += 2) {
                const bool valid = some && r < count;
                t5_cp16(to + r * 128 + (((col & 7) ^ (r & 7)) << 4), valid ? src : (const uint16_t*)pg.c.v, valid ? 16 : 0);
                src += 2 * pg.c.v_row;
              }
            }
            t5_commit_group();
            t5_wait_group<0>();
            t5_fence_async_smem();
            __syncwarp();
            if (lane == 0) t5_mbar_arrive(full);
          }
          __syncwarp();
        }
        v_sl = k_sl;
        v_par = k_par;
        if (++k_sl == ring) {
          k_sl = 0;
          k_par ^= 1;
        }
      }
    } else {
      for (int h = 0, sl = 0, par = 1; h < n && live; ++h) {
        const int kb = block_of(w, h);
        const bool pre = kb < nb_pre;
        const int j0 = pre ? kb * kT5Keys : (kb - nb_pre) * kT5Keys;
        const int count = min(kT5Keys, (pre ? prefix_len : own_keys) - j0);
        const bool tma = !pre || (prefix_tma && count == kT5Keys);
        const int row = pre ? prefix_start + j0 : seq_start + j0;
        for (int is_v = 0; is_v < 2 && live; ++is_v) {
          const uint32_t dst = (is_v ? ring_v(w) : ring_k(w)) + sl * kT5KvBytes;
          const uint32_t full = is_v ? bar_vf(w, sl) : bar_kf(w, sl), empty = is_v ? bar_ve(w, sl) : bar_ke(w, sl);
          // the product that read this slot a ring of blocks ago has completed
          if (h >= ring && !__all_sync(0xffffffffu, t5_mbar_wait(empty, par, spin))) { live = false; break; }
          if (tma) {
            if (lane == 0) {
              t5_mbar_expect_tx(full, kT5KvBytes);
              const CUtensorMap* map = pre ? (is_v ? &tm_vp : &tm_kp) : (is_v ? &tm_v : &tm_k);
              t5_tma_3d(dst, map, 0, pre ? row : hk, pre ? hk : row, full);
              t5_tma_3d(dst + kT5Keys * 128, map, 64, pre ? row : hk, pre ? hk : row, full);
            }
          } else {
            const uint16_t* src = pre ? (is_v ? vpre : kpre) + (long long)j0 * p_sn
                                      : (is_v ? vown + (long long)j0 * v_sn : kown + (long long)j0 * k_sn);
            t5_load_tile<32, kT5Keys>(dst, src, pre ? p_sn : (is_v ? v_sn : k_sn), count, lane);
            t5_commit_group();
            t5_wait_group<0>();
            t5_fence_async_smem();
            __syncwarp();
            if (lane == 0) t5_mbar_arrive(full);
          }
        }
        if (++sl == ring) {
          sl = 0;
          par ^= 1;
        }
      }
    }
    if (!live && lane == 0) t5_sts_u32(dead_flag, 1);
  } else if (warp >= 8) {
    // ---- an issuing warp: one lane queues every product of warpgroup w.  The descriptors are built once; per
    // instruction only the start-address field moves.  The issue of a product blocks while the tensor core's
    // queue is full, and this lane's waits and commits are not hidden behind its own products; with one
    // issuing lane per warpgroup the bookkeeping of one overlaps the products of the other.
    if (lane == 0 && !idle_issuers) {
      const int w = warp - 8, n = n_blk(w);
      const uint64_t dq = t5_desc(q_tile(w), 16, 1024), dk = t5_desc(ring_k(w), 16, 1024);
      const uint64_t dv = t5_desc(ring_v(w), kT5Keys * 128, 1024);
      const uint32_t tw = tmem + 256 * w;
      const uint32_t idesc_pv = kPaged ? t5_idesc((uint32_t)((vdim + 15) / 16 * 16)) | (1u << 16) : kT5IdescPV;
      bool live = t5_mbar_wait(bar_q, 0, spin);
      int k_sl = 0, k_par = 0;
      auto issue_s = [&](int h) {  // S(h) = Q K(h)^T into S buffer h & 1, then the arrivals; called for h = 0, 1, ...
        const int sl = k_sl;
        if (!t5_mbar_wait(bar_kf(w, sl), k_par, spin)) { live = false; return; }
        if (++k_sl == ring) {
          k_sl = 0;
          k_par ^= 1;
        }
        const uint64_t kd = dk + (uint64_t)(sl * (kT5KvBytes >> 4));
        const uint32_t d = tw + 64 * (h & 1);
#pragma unroll
        for (int j = 0; j < 4 * kKeyBlocks; ++j)  // 16 channels per instruction
          t5_mma_ss(d, dq + (uint64_t)(((j >> 2) * (kT5Tile * 128) + (j & 3) * 32) >> 4),
                    kd + (uint64_t)(((j >> 2) * (kT5Keys * 128) + (j & 3) * 32) >> 4), kT5IdescQK, j > 0);
        t5_mma_commit(bar_s(w, h & 1));
        t5_mma_commit(bar_ke(w, sl));
      };
      for (int h = 0; h < 2; ++h)
        if (h < n && live) issue_s(h);
      for (int h = 0, sl = 0, par = 0; h < n && live; ++h) {
        // P(h) is stored and V(h) has landed
        if (!t5_mbar_wait(bar_r(w, h & 1), (h >> 1) & 1, spin) || !t5_mbar_wait(bar_vf(w, sl), par, spin)) {
          live = false;
          break;
        }
        t5_fence_after();
        const uint64_t vd = dv + (uint64_t)(sl * (kT5KvBytes >> 4));
#pragma unroll
        for (int j = 0; j < 4; ++j)  // 16 keys per instruction: 8 columns of packed P, 2 KB of V rows
          t5_mma_ts(tw + 128, tw + 64 * (h & 1) + 8 * j, vd + (uint64_t)(j * (2048 >> 4)), idesc_pv, (h > 0) || (j > 0));
        t5_mma_commit(bar_ve(w, sl));
        if (h + 2 < n) issue_s(h + 2);  // executes behind P V(h): it overwrites the columns P(h) is read from
        else t5_mma_commit(bar_o(w, h + 1 < n ? 0 : 1));  // the last-but-one / the last P V of the warpgroup
        if (++sl == ring) {
          sl = 0;
          par ^= 1;
        }
      }
      if (!live) t5_sts_u32(dead_flag, 1);
    }
  } else {
    const int n_mine = n_blk(wg);
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t tS = tmem + 256 * wg + lane_base, tO = tS + 128;  // this thread's lane
    const int my_keys = min(own_keys, cached + row0 + wt - seq_start + 1);  // own-chunk keys this row may see
    const int first_keys = min(own_keys, cached + row0 - seq_start + 1);    // ... and the tile's first row
    float m_ref = -INFINITY, l = 0.f;  // offset of the exponentials (log2 units, scaled), running sum
    int my_first = 0, last_first = 0;  // first key in the window of this row and of the tile's last row
    if constexpr (kOptions) {
      if (pg.opt.window > 0) {
        my_first = cached + row0 + wt - seq_start - pg.opt.window + 1;
        last_first = cached + cta_last - seq_start - pg.opt.window + 1;
      }
      if (pg.opt.sink && (wg == 0 || pair)) {
        m_ref = pg.opt.sink[head(wg)] * 1.4426950408889634f;
        l = 1.f;
      }
    }
    bool ok = true;
    for (int h = 0; h < n_mine && ok; ++h) {
      ok = t5_mbar_wait(bar_s(wg, h & 1), (h >> 1) & 1, spin);  // S(h) is complete
      t5_fence_after();
      // ---- softmax of this thread's row
      const int kb = block_of(wg, h);
      const bool pre = kb < nb_pre;
      const int j0 = pre ? kb * kT5Keys : (kb - nb_pre + skipped) * kT5Keys;
      const int lim = (pre ? prefix_len : my_keys) - j0;                // keys [0, lim) visible to this row
      const int low = kOptions ? my_first - j0 : 0;                      // ... but for those in front of its window
      // ... all 64 to every row of the tile
      const bool full = (pre ? prefix_len : first_keys) - j0 >= kT5Keys && (!kOptions || last_first <= j0);
      uint32_t u[64];
      t5_ld64(tS + 64 * (h & 1), u);
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // four chains instead of one of 64
      if (full) {
#pragma unroll
        for (int c = 0; c < 64; c += 2) mx4[(c >> 1) & 3] = t5_max3(mx4[(c >> 1) & 3], __uint_as_float(u[c]), __uint_as_float(u[c + 1]));
      } else {
#pragma unroll
        for (int c = 0; c < 64; ++c) mx4[c & 3] = fmaxf(mx4[c & 3], c < lim && (!kOptions || c >= low) ? __uint_as_float(u[c]) : -INFINITY);
      }
      const float r = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2;
      const bool move = r > m_ref + kT5Lazy;  // also true for the first visible key of a row (m_ref = -inf)
      if (__any_sync(0xffffffffu, move)) {
        const float alpha = move ? t5_exp2(m_ref - r) : 1.f;  // 0 when nothing was accumulated yet
        if (move) { m_ref = r; l *= alpha; }
        if (h > 0) {
          // O must be at rest: P V(h-1) may still be queued.  Its completion is what S(h+1)'s barrier (or, for
          // the last block, the barrier of the last-but-one P V) reports; waiting for that phase here and again
          // at the top of the next block is harmless.
          ok = ok && (h + 1 < n_mine ? t5_mbar_wait(bar_s(wg, (h + 1) & 1), ((h + 1) >> 1) & 1, spin) : t5_mbar_wait(bar_o(wg, 0), 0, spin));
          t5_fence_after();
#pragma unroll 1  // here and below: code that runs once or twice has to be fetched, which is what a short tile waits for
          for (int c = 0; c < 4; ++c) {
            if (kPaged && 32 * c >= vdim) break;
            uint32_t w[32];
            t5_ld32(tO + 32 * c, w);
#pragma unroll
            for (int e = 0; e < 32; ++e) w[e] = __float_as_uint(__uint_as_float(w[e]) * alpha);
            t5_st32(tO + 32 * c, w);
          }
        }
      }
      const float off = m_ref == -INFINITY ? 0.f : m_ref;  // kernels.py:1062
      float ps4[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t pk[32];
      if (full) {  // two scores per instruction where there is one for it: what paces a block is its warps' instructions
        const t5_pair scale2 = t5_two(scale_log2, scale_log2), off2 = t5_two(-off, -off);
        t5_pair sum2[2] = {t5_two(0.f, 0.f), t5_two(0.f, 0.f)};
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          float p0, p1;
          t5_split(t5_fma2(t5_two(__uint_as_float(u[2 * c]), __uint_as_float(u[2 * c + 1])), scale2, off2), p0, p1);
          p0 = t5_exp2(p0);
          p1 = t5_exp2(p1);
          sum2[c & 1] = t5_add2(sum2[c & 1], t5_two(p0, p1));
          pk[c] = t5_pack_bf16x2(p0, p1);
        }
        t5_split(sum2[0], ps4[0], ps4[1]);
        t5_split(sum2[1], ps4[2], ps4[3]);
      } else {
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          const float p0 = 2 * c < lim && (!kOptions || 2 * c >= low) ? t5_exp2(fmaf(__uint_as_float(u[2 * c]), scale_log2, -off)) : 0.f;
          const float p1 = 2 * c + 1 < lim && (!kOptions || 2 * c + 1 >= low) ? t5_exp2(fmaf(__uint_as_float(u[2 * c + 1]), scale_log2, -off)) : 0.f;
          ps4[c & 3] += p0 + p1;
          pk[c] = t5_pack_bf16x2(p0, p1);
        }
      }
      l += (ps4[0] + ps4[1]) + (ps4[2] + ps4[3]);
      t5_st32(tS + 64 * (h & 1), pk);  // P over the first 32 columns of this S buffer
      asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
      t5_fence_before();
      ok = __all_sync(0xffffffffu, ok);  // the warp goes on or stops as a whole
      if (ok) t5_mbar_arrive(bar_r(wg, h & 1));  // hand P(h) to the issuing warp
    }
    pdl_trigger();
    if (n_mine > 0 && ok) ok = t5_mbar_wait(bar_o(wg, 1), 0, spin);  // the last P V
    t5_fence_after();
    if (!ok) t5_sts_u32(dead_flag, 1);
    m_ref_keep = m_ref;
    l_keep = l;
  }

  // ---- merge the two warpgroups (a pair has nothing to merge): warpgroup 1 hands its (offset, sum, O) over through shared memory
  // (the first 64 KB of its rings, [channel][row] fp32 so that both sides touch consecutive banks)
  const uint32_t xO = base + kT5QBytes + kT5WgBytes, xML = base + kT5QBytes;  // (unless a pair) scalars: start of warpgroup 0's rings
  const uint32_t tO = tmem + 256 * (wg & 1) + 128 + ((uint32_t)(((tid >> 5) & 3) * 32) << 16);
  const int my_row = row0 + wt;
  t5_fence_before();
  __syncthreads();  // every product of the CTA is complete (or given up), nobody uses the rings any more
  t5_fence_after();
  dead = t5_lds_u32(dead_flag) != 0;
  if (wg == 1 && !pair) {
#pragma unroll 1
    for (int c = 0; c < 4; ++c) {
      if (kPaged && 32 * c >= vdim) break;
      uint32_t w[32];
      if (n_blk(1) > 0 && !dead) {
        t5_ld32(tO + 32 * c, w);
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) w[e] = 0u;
      }
#pragma unroll
      for (int e = 0; e < 32; ++e) t5_sts_u32(xO + ((32 * c + e) * 128 + wt) * 4, w[e]);
    }
    t5_sts_u32(xML + wt * 4, __float_as_uint(m_ref_keep));
    t5_sts_u32(xML + 512 + wt * 4, __float_as_uint(l_keep));
  }
  __syncthreads();
  if (wg == 0 || (pair && wg == 1 && n_blk(1) > 0)) {
    const int hq = head(wg);
    const float m0 = m_ref_keep, l0 = l_keep;
    const float m1 = pair ? -INFINITY : __uint_as_float(t5_lds_u32(xML + wt * 4)), l1 = pair ? 0.f : __uint_as_float(t5_lds_u32(xML + 512 + wt * 4));
    if (dead && wt == 0 && status) atomicOr(status, B200KV_S_TIMEOUT);
    if (!dead) {
      const float mm = fmaxf(m0, m1);
      const float a0 = m0 == -INFINITY ? 0.f : t5_exp2(m0 - mm), a1 = m1 == -INFINITY ? 0.f : t5_exp2(m1 - mm);
      const float lt = l0 * a0 + l1 * a1;
      float inv = lt != 0.f ? 1.f / lt : 0.f;  // kernels.py:1118
      if constexpr (kOptions) inv *= my_row < row_end ? pg.opt.factor<uint16_t>(my_row, hq) : 0.f;
      const float f0 = a0 * inv, f1 = a1 * inv;
      uint4* dst = reinterpret_cast<uint4*>(out + (long long)my_row * o_sn + hq * o_sh);
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        if (kPaged && 32 * c >= vdim) break;
        uint32_t w[32];
        t5_ld32(tO + 32 * c, w);
        float o[32];
#pragma unroll
        for (int e = 0; e < 32; ++e) {
          uint32_t x = 0u;
          if (!pair) x = t5_lds_u32(xO + ((32 * c + e) * 128 + wt) * 4);
          o[e] = __uint_as_float(w[e]) * f0 + __uint_as_float(x) * f1;
        }
        if (kPaged && vdim % 8 != 0) {
          if (my_row < row_end) {
            uint16_t* p = out + (long long)my_row * o_sn + hq * o_sh + 32 * c;
#pragma unroll
            for (int e = 0; e < 32; ++e)
              if (32 * c + e < vdim) p[e] = (uint16_t)float_to_bf16_bits(o[e]);
          }
        } else if (my_row < row_end) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            if (kPaged && 32 * c + 8 * e >= vdim) break;
            uint4 x;
            x.x = t5_pack_bf16x2(o[8 * e], o[8 * e + 1]);
            x.y = t5_pack_bf16x2(o[8 * e + 2], o[8 * e + 3]);
            x.z = t5_pack_bf16x2(o[8 * e + 4], o[8 * e + 5]);
            x.w = t5_pack_bf16x2(o[8 * e + 6], o[8 * e + 7]);
            dst[4 * c + e] = x;
          }
        }
      }
    }
  }
  t5_fence_before();
  __syncthreads();
  if (tid < 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kT5Cols) : "memory");
}

}  // namespace b200kv
