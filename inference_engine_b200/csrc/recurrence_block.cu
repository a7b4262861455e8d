// Prompt portions of the delta rule (one decay per key channel), eight tokens at a time and all in 32-bit.
//
// With L_i the running product of a block's decays up to token i (per key channel), S0 the state in front of the block, and
//   kd_i = k_i * L_i     qd_i = q_i * L_i     kr_j = k_j * (L_8 / L_j)     (quotients as products of the decays between: all <= 1)
//   A_ij = sum_d k_i k_j L_i / L_j  (j < i)     B_ij = sum_d q_i k_j L_i / L_j  (j <= i)
// the block's writes solve a triangular system, u = (I + diag(beta) A)^-1 diag(beta) (v - S0^T kd), the outputs are
// o = S0^T qd + B u, and the state behind is S = L_8 * S0 + sum_j kr_j u_j^T.
//   prepare  one block of threads per (8 tokens, head), all independent: the vectors, the inverse T and B, to a workspace.
//   scan     (rb_scan_kernel; rb_scan_split_kernel with the read-out in warps of its own)
//            groups of lanes own four state columns each, block after block: two sums over the key channels per token on the
//            same state, one exchange of the eight tokens' sums between the lanes, the eight writes in one pass.
//            A block's vectors come by bulk copies into a ring; packed 32-bit arithmetic (two rows per instruction).
// Every wait is bounded: when one runs out the block writes nothing more and sets B200KV_S_TIMEOUT.
#include <algorithm>

#include "dec_tma.cuh"
#include "recurrence.cuh"

namespace b200kv {

constexpr int kRbTok = 8;        // tokens per block
constexpr int kRbWarps = 2;      // of a block of the scan
constexpr int kRbCols = 4;       // state columns of a group of lanes
constexpr int kRbStages = 3;

// Workspace of one (block, head) in floats: kd, qd, kr [8][Dp], L_8 [Dp], T [8][8], B [8][8].
__host__ __device__ constexpr int rb_floats(int Dp) { return 3 * kRbTok * Dp + Dp + 2 * kRbTok * kRbTok; }

// First block of entry e in the list of all blocks: never less than the number of blocks of the entries in front.
__device__ __forceinline__ int rb_first(const b200dec_entries& ent, int e) { return ent.cu_seqlens[e] / kRbTok + e; }

// ---------------------------------------------------------------- prepare
constexpr int kRpSums = 80;  // A (28), B (36), squares of q and of k (8 each)

__host__ __device__ constexpr int rp_a(int i, int j) { return i * (i - 1) / 2 + j; }       // j < i
__host__ __device__ constexpr int rp_b(int i, int j) { return 28 + i * (i + 1) / 2 + j; }  // j <= i
constexpr int kRpQ = 64, kRpK = 72;

// Sums of 16 values over 16 lanes, of which lane l keeps the l-th.
__device__ __forceinline__ float rp_exchange(float (&v)[16], int lane) {
  int n = 8;
#pragma unroll
  for (int bit = 8; bit > 0; bit >>= 1) {
    const bool hi = lane & bit;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float keep = hi ? v[i + n] : v[i], give = hi ? v[i] : v[i + n];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
    }
    n >>= 1;
  }
  return v[0];
}

// Two mappings of the threads: a key channel of all or half of the eight tokens each (kParts 1, 2), and, for the sums over the channels, 16 or
// 32 lanes per token j, which find the products of token j with every later one in a handful of registers.  With all 64 sums of its
// channel in one thread's registers three blocks fitted a multiprocessor, and a warp spent a third of its instructions exchanging them: 1000
// rows of 16 heads of 128 27.0 -> 20.0 us.  Twice the threads shorten the chain where all blocks are at work at once (50 rows) and are
// slower where they are not (23.5).
template <typename T, int Dp, int kParts>
__global__ void __launch_bounds__(128 * kParts)
rb_prepare_kernel(const b200dec_recurrence rec, const b200dec_recurrence_in in, const T* conv, int conv_stride,
                  const b200dec_entries ent, float* __restrict__ ws, int32_t* status) {
  constexpr int kChannels = 128, kRpHalf = kRbTok / kParts, kLanes = 16 * kParts;
  constexpr bool kOne = Dp <= kChannels;  // a thread's channel stays in registers
  __shared__ float2 kq[kRbTok][Dp];  // k, q
  __shared__ float decay[kRbTok][Dp];
  __shared__ float sums[kRpSums], beta[kRbTok], fq[kRbTok], fk[kRbTok];
  pdl_enter();
  const int s = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  int lo = 0, hi = ent.num_entries;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (rb_first(ent, mid) <= s) lo = mid; else hi = mid;
  }
  if (lo < *ent.num_decoding) { pdl_wait(); return; }
  const RecEntry x = rec_entry(ent, rec, lo, status);
  const int t0 = (s - rb_first(ent, lo)) * kRbTok, nt = min(kRbTok, x.n - t0);
  pdl_wait();
  if (nt <= 0) return;
  const int D = rec.dim, hq = h / (rec.heads / rec.qk_heads);
  const long long row0 = x.first + t0;
  const float na = rec.neg_a[h];
  const T* steps = (const T*)in.step + row0 * in.step_stride + h * D;
  const T* src = conv + row0 * conv_stride + hq * D;
  if (tid < kRbTok) beta[tid] = tid < nt ? sigmoid_f(ld_elem((const T*)in.beta + (row0 + tid) * in.beta_stride + h)) : 0.f;
  const int half = tid / kChannels, i0 = half * kRpHalf;  // this thread's tokens: kRpHalf from i0 on
  float q[kRpHalf], k[kRpHalf], g[kRpHalf];
  auto load = [&](int d) {
    const float bias = d < D ? rec.dt_bias[h * D + d] : 0.f;
    const T *pq = src + i0 * (long long)conv_stride + rec.off_q + d, *pk = src + i0 * (long long)conv_stride + rec.off_k + d,
            *ps = steps + i0 * (long long)in.step_stride + d;
#pragma unroll
    for (int i = 0; i < kRpHalf; ++i) {
      const bool some = i0 + i < nt && d < D;
      q[i] = some ? ld_elem(pq) : 0.f;
      k[i] = some ? ld_elem(pk) : 0.f;
      g[i] = some ? ld_elem(ps) + bias : 0.f;
      pq += conv_stride;
      pk += conv_stride;
      ps += in.step_stride;
    }
#pragma unroll
    for (int i = 0; i < kRpHalf; ++i) g[i] = i0 + i < nt && d < D ? expf(na * softplus_f(g[i])) : 1.f;
  };
  for (int d = tid % kChannels; d < Dp; d += kChannels) {
    load(d);
#pragma unroll
    for (int i = 0; i < kRpHalf; ++i) {
      kq[i0 + i][d] = make_float2(k[i], q[i]);
      decay[i0 + i][d] = g[i];
    }
  }
  __syncthreads();
  {
    const int j = tid / kLanes, l = tid % kLanes;
    float v[16], nk = 0.f, nq = 0.f;  // A of tokens 0 to 7 with j, B
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = 0.f;
    for (int d = l; d < Dp; d += kLanes) {
      float2 x[kRbTok];
      float g8[kRbTok];
#pragma unroll
      for (int i = 0; i < kRbTok; ++i) {
        x[i] = kq[i][d];
        g8[i] = decay[i][d];
      }
      float f = 0.f;  // k_j times the decays since
#pragma unroll
      for (int i = 0; i < kRbTok; ++i) {
        if (i < j) continue;
        if (i == j) {
          f = x[i].x;
          nk = fmaf(x[i].x, x[i].x, nk);
          nq = fmaf(x[i].y, x[i].y, nq);
        } else {
          f *= g8[i];
          v[i] = fmaf(x[i].x, f, v[i]);
        }
        v[8 + i] = fmaf(x[i].y, f, v[8 + i]);
      }
    }
    float mine = rp_exchange(v, l);
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) {
      nk += __shfl_xor_sync(0xffffffffu, nk, o);
      nq += __shfl_xor_sync(0xffffffffu, nq, o);
    }
    if (kParts == 2) mine += __shfl_xor_sync(0xffffffffu, mine, 16);
    const int i = l & 7;
    if (l < 8 ? i > j : (l < 16 && i >= j)) sums[l < 8 ? rp_a(i, j) : rp_b(i, j)] = mine;
    if (l == 0) {
      sums[kRpQ + j] = nq;
      sums[kRpK + j] = nk;
    }
  }
  __syncthreads();
  if (tid < kRbTok) {
    fq[tid] = rec.q_scale * (rec.unit_norm ? 1.0f / sqrtf(sums[kRpQ + tid] + rec.unit_eps) : 1.f);
    fk[tid] = rec.unit_norm ? 1.0f / sqrtf(sums[kRpK + tid] + rec.unit_eps) : 1.f;
  }
  __syncthreads();
  float* dst = ws + ((long long)s * rec.heads + h) * rb_floats(Dp);
  float* tb = dst + 3 * kRbTok * Dp + Dp;
  for (int d = tid % kChannels; d < Dp; d += kChannels) {
    if (!kOne) load(d);
    float f = 1.f, rest = 1.f;  // the decays up to here, and those of the other half's tokens, if they come later
    if (kParts == 2) {
#pragma unroll
      for (int i = 0; i < kRpHalf; ++i) {
        const float other = decay[kRpHalf - i0 + i][d];
        if (half) f *= other; else rest *= other;
      }
    }
#pragma unroll
    for (int i = 0; i < kRpHalf; ++i) {
      f *= g[i];
      dst[(i0 + i) * Dp + d] = k[i] * fk[i0 + i] * f;
      dst[(kRbTok + i0 + i) * Dp + d] = q[i] * fq[i0 + i] * f;
    }
    if (half == kParts - 1) dst[3 * kRbTok * Dp + d] = f;
    f = rest;
#pragma unroll
    for (int i = kRpHalf - 1; i >= 0; --i) {
      dst[(2 * kRbTok + i0 + i) * Dp + d] = k[i] * fk[i0 + i] * f;
      f *= g[i];
    }
  }
  if (tid < kRbTok) {  // column tid of the inverse
    float c[kRbTok];
#pragma unroll
    for (int i = 0; i < kRbTok; ++i) {
      float a = i == tid ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < i; ++j) a = fmaf(-sums[rp_a(i, j)] * fk[i] * fk[j], c[j], a);
      c[i] = beta[i] * a;
      tb[i * kRbTok + tid] = c[i];
    }
  } else if (tid >= 64 && tid < 128) {
    const int i = (tid - 64) / kRbTok, j = tid % kRbTok;
    tb[kRbTok * kRbTok + tid - 64] = j <= i ? sums[28 + i * (i + 1) / 2 + j] * fq[i] * fk[j] : 0.f;
  }
}

// ---------------------------------------------------------------- scan
typedef unsigned long long rb_pair;  // two 32-bit numbers of neighbouring rows
__device__ __forceinline__ rb_pair rb_pack(float a, float b) {
  rb_pair r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float rb_both(rb_pair p) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p));
  return a + b;
}
__device__ __forceinline__ rb_pair rb_fma(rb_pair a, rb_pair b, rb_pair c) {
  rb_pair r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ rb_pair rb_mul(rb_pair a, rb_pair b) {
  rb_pair r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// Volatile, so that the loads stay in front of the arithmetic they feed instead of beside it.
__device__ __forceinline__ ulonglong2 rb_lds(uint32_t addr) {
  ulonglong2 v;
  asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ void rb_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// Sums of 32 values over kLanes lanes, of which each keeps 32 / kLanes: those of token lane / (kLanes / 8) and of columns
// kC * (lane % (kLanes / 8)) on, kC = 32 / kLanes.  A lane holds token i ^ (the token it will keep) in places 4 i .., so that what it gives away in the exchanges over tokens always stands in the same places.
template <int kLanes>
__device__ __forceinline__ void rb_exchange(float (&v)[kRbCols * kRbTok], int lane) {
  int n = kRbCols * kRbTok / 2;
#pragma unroll
  for (int bit = kLanes / 2; bit > 0; bit >>= 1) {
    const bool hi = n < kRbCols && (lane & bit);
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float keep = hi ? v[i + n] : v[i], give = hi ? v[i] : v[i + n];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
    }
    n >>= 1;
  }
}

// What a lane does with its rows of the state, kR of kRbCols columns as pairs of rows: rows 4 kLanes j + 4 l + (0..3), j < kR / 4.
template <int kLanes, int kR>
__device__ __forceinline__ void rb_state_load(rb_pair (&S)[kRbCols][kR / 2], const float* state, bool some, int D, int P4, int p0, int l) {
#pragma unroll
  for (int i = 0; i < kR / 2; ++i) {
    const int d = (i / 2) * 4 * kLanes + 4 * l + 2 * (i & 1);
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), c = a;
    if (some) {
      if (d < D) a = __ldcg(reinterpret_cast<const float4*>(state + (long long)d * P4 + p0));
      if (d + 1 < D) c = __ldcg(reinterpret_cast<const float4*>(state + (long long)(d + 1) * P4 + p0));
    }
    S[0][i] = rb_pack(a.x, c.x);
    S[1][i] = rb_pack(a.y, c.y);
    S[2][i] = rb_pack(a.z, c.z);
    S[3][i] = rb_pack(a.w, c.w);
  }
}
template <int kLanes, int kR>
__device__ __forceinline__ void rb_state_store(const rb_pair (&S)[kRbCols][kR / 2], float* state, int D, int P, int P4, int p0, int l) {
#pragma unroll
  for (int i = 0; i < kR / 2; ++i) {
    const int d = (i / 2) * 4 * kLanes + 4 * l + 2 * (i & 1);
    float a[kRbCols], c[kRbCols];
#pragma unroll
    for (int k = 0; k < kRbCols; ++k) {
      asm("mov.b64 {%0, %1}, %2;" : "=f"(a[k]), "=f"(c[k]) : "l"(S[k][i]));
      if (p0 + k >= P) a[k] = c[k] = 0.f;
    }
    if (p0 < P4) {
      if (d < D) st_elem4(state + (long long)d * P4 + p0, a);
      if (d + 1 < D) st_elem4(state + (long long)(d + 1) * P4 + p0, c);
    }
  }
}
// its rows of a stage's eight vectors (of token i ^ swap in place i); mine: the stage, 16 l bytes on
template <int kLanes, int kR>
__device__ __forceinline__ void rb_rows(uint32_t mine, int vec, int swap, ulonglong2 (&k)[kRbTok][kR / 4]) {
#pragma unroll
  for (int i = 0; i < kRbTok; ++i)
#pragma unroll
    for (int j = 0; j < kR / 4; ++j) k[i][j] = rb_lds(mine + 4 * ((vec * kRbTok + (i ^ swap)) * kLanes * kR + 4 * kLanes * j));
}
// ... and their sums with the state
template <int kR>
__device__ __forceinline__ void rb_sums(const rb_pair (&S)[kRbCols][kR / 2], const ulonglong2 (&vec)[kRbTok][kR / 4], float (&r)[kRbCols * kRbTok]) {
#pragma unroll
  for (int i = 0; i < kRbTok; ++i) {
    rb_pair acc[kRbCols];
#pragma unroll
    for (int j = 0; j < kR / 4; ++j) {
      const ulonglong2 k = vec[i][j];
#pragma unroll
      for (int c = 0; c < kRbCols; ++c) {
        acc[c] = j == 0 ? rb_mul(S[c][0], k.x) : rb_fma(S[c][2 * j], k.x, acc[c]);
        acc[c] = rb_fma(S[c][2 * j + 1], k.y, acc[c]);
      }
    }
#pragma unroll
    for (int c = 0; c < kRbCols; ++c) r[kRbCols * i + c] = rb_both(acc[c]);
  }
}
// S <- decay S + sum of k_i u_i^T
template <int kR>
__device__ __forceinline__ void rb_update(rb_pair (&S)[kRbCols][kR / 2], const ulonglong2 (&decay)[kR / 4], const ulonglong2 (&k)[kRbTok][kR / 4],
                                          const float (&u)[kRbTok][kRbCols]) {
#pragma unroll
  for (int j = 0; j < kR / 4; ++j)
#pragma unroll
    for (int c = 0; c < kRbCols; ++c) {
      S[c][2 * j] = rb_mul(S[c][2 * j], decay[j].x);
      S[c][2 * j + 1] = rb_mul(S[c][2 * j + 1], decay[j].y);
    }
#pragma unroll
  for (int i = 0; i < kRbTok; ++i) {
    const float4 uu = *reinterpret_cast<const float4*>(u[i]);
    const rb_pair up[kRbCols] = {rb_pack(uu.x, uu.x), rb_pack(uu.y, uu.y), rb_pack(uu.z, uu.z), rb_pack(uu.w, uu.w)};
#pragma unroll
    for (int j = 0; j < kR / 4; ++j) {
#pragma unroll
      for (int c = 0; c < kRbCols; ++c) {
        S[c][2 * j] = rb_fma(k[i][j].x, up[c], S[c][2 * j]);
        S[c][2 * j + 1] = rb_fma(k[i][j].y, up[c], S[c][2 * j + 1]);
      }
    }
  }
}
// a token's row of T or B
__device__ __forceinline__ void rb_row8(const float* p, float (&row)[kRbTok]) {
  const float4 a = *reinterpret_cast<const float4*>(p), c = *reinterpret_cast<const float4*>(p + 4);
  row[0] = a.x; row[1] = a.y; row[2] = a.z; row[3] = a.w;
  row[4] = c.x; row[5] = c.y; row[6] = c.z; row[7] = c.w;
}

// kLanes lanes share kRbCols state columns; lane l owns rows 4 kLanes j + 4 l + (0..3), j < kR / 4, of all of them.
// One block: kRbWarps warps, 32 kRbCols / kLanes columns each, of one head of one entry.
template <typename T, int kLanes, int kR>
__global__ void __launch_bounds__(32 * kRbWarps)
rb_scan_kernel(const b200dec_recurrence rec, const b200dec_recurrence_in in, const T* conv, int conv_stride,
               const b200dec_entries ent, const float* ws, float* __restrict__ out, int slabs, int32_t* status) {
  constexpr int Dp = kLanes * kR, kFloats = rb_floats(Dp), kQuads = kR / 4, kGroups = 32 / kLanes;
  constexpr int kM = kLanes / 8, kC = kRbCols / kM;  // after the exchange a lane holds kC columns of one token
  extern __shared__ __align__(128) float rb_smem[];  // [kRbStages][kFloats]
  __shared__ __align__(16) float ubuf[kRbWarps][kGroups][kRbTok][kRbCols];
  __shared__ __align__(8) uint64_t bars[kRbStages];
  pdl_enter();
  const int e = blockIdx.y, h = blockIdx.x / slabs, slab = blockIdx.x - h * slabs, tid = threadIdx.x;
  if (e < *ent.num_decoding) { pdl_wait(); return; }
  const RecEntry x = rec_entry(ent, rec, e, status);
  if (tid == 0) {
    for (int i = 0; i < kRbStages; ++i) dt_mbar_init(dt_smem(bars + i), 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  pdl_wait();
  if (x.n == 0) return;
  const int D = rec.dim, P = rec.vdim, P4 = rec_round4(P), blocks = (x.n + kRbTok - 1) / kRbTok;
  const int warp = tid >> 5, grp = (tid & 31) / kLanes, l = tid % kLanes;
  const int p0 = ((slab * kRbWarps + warp) * kGroups + grp) * kRbCols;  // the first column
  const int tok = l / kM, pc = p0 + kC * (l % kM);                  // what this lane holds after the exchange
  const long long at0 = (long long)rb_first(ent, e) * rec.heads + h;
  auto fetch = [&](int b) {
    const uint32_t bar = dt_smem(bars + b % kRbStages);
    dt_expect_tx(bar, kFloats * 4);
    rb_bulk(dt_smem(rb_smem + (b % kRbStages) * kFloats), ws + (at0 + (long long)b * rec.heads) * kFloats, kFloats * 4, bar);
  };
  if (tid == 0)
    for (int b = 0; b < min(kRbStages, blocks); ++b) fetch(b);
  float* state = rec.state + ((long long)x.slot * rec.heads + h) * D * P4;
  rb_pair S[kRbCols][kR / 2];  // [column][pair of rows]
  rb_state_load<kLanes, kR>(S, state, x.pos > 0 && p0 < P4, D, P4, p0, l);
  // v of this lane's token and columns in block b; kept as loaded until it is used, so that nothing waits for it
  auto value = [&](int b, T (&v)[kC]) {
    const int t = b * kRbTok + tok;
    const T* src = conv + (long long)(x.first + t) * conv_stride + rec.off_v + h * P + pc;
#pragma unroll
    for (int c = 0; c < kC; ++c) v[c] = t < x.n && pc + c < P ? src[c] : T(0);
  };
  T v_next[kC];
  value(0, v_next);
  bool dead = false;
  for (int b = 0; b < blocks; ++b) {
    float w[kC];
#pragma unroll
    for (int c = 0; c < kC; ++c) w[c] = ld_elem(v_next + c);
    value(b + 1, v_next);
    if (!dt_mbar_wait(dt_smem(bars + b % kRbStages), (b / kRbStages) & 1)) dead = true;
    const float* st = rb_smem + (b % kRbStages) * kFloats;
    const uint32_t mine = dt_smem(st) + 16 * l;
    ulonglong2 ka[kRbTok][kQuads], kb[kRbTok][kQuads], decay[kQuads];
    float r[kRbCols * kRbTok], o[kRbCols * kRbTok];
    rb_rows<kLanes, kR>(mine, 0, tok, ka);
    rb_rows<kLanes, kR>(mine, 1, tok, kb);
    rb_sums<kR>(S, ka, r);
    rb_rows<kLanes, kR>(mine, 2, 0, ka);
    rb_exchange<kLanes>(r, l);
    rb_sums<kR>(S, kb, o);
#pragma unroll
    for (int j = 0; j < kQuads; ++j) decay[j] = rb_lds(mine + 4 * (3 * kRbTok * Dp + 4 * kLanes * j));
    rb_exchange<kLanes>(o, l);
    const float* tb = st + 3 * kRbTok * Dp + Dp;
    float row[2][kRbTok];
    rb_row8(tb + tok * kRbTok, row[0]);
    rb_row8(tb + (kRbTok + tok) * kRbTok, row[1]);
    float u[kC];
#pragma unroll
    for (int c = 0; c < kC; ++c) {
      w[c] -= r[c];
      float even = 0.f, odd = 0.f;
#pragma unroll
      for (int j = 0; j < kRbTok; ++j) {
        const float wj = __shfl_sync(0xffffffffu, w[c], j * kM + l % kM, kLanes);
        if (j & 1) odd = fmaf(row[0][j], wj, odd); else even = fmaf(row[0][j], wj, even);
      }
      u[c] = even + odd;
      ubuf[warp][grp][tok][kC * (l % kM) + c] = u[c];
    }
    __syncwarp();
    const int t = b * kRbTok + tok;
#pragma unroll
    for (int c = 0; c < kC; ++c) {
      float even = o[c], odd = 0.f;
#pragma unroll
      for (int j = 0; j < kRbTok; ++j) {
        const float uj = ubuf[warp][grp][j][kC * (l % kM) + c];
        if (j & 1) odd = fmaf(row[1][j], uj, odd); else even = fmaf(row[1][j], uj, even);
      }
      if (t < x.n && pc + c < P && !dead) out[((long long)(x.first + t) * rec.heads + h) * P + pc + c] = even + odd;
    }
    rb_update<kR>(S, decay, ka, ubuf[warp][grp]);
    if (__syncthreads_or(dead)) {  // (otherwise: the stage and ubuf are free)
      if (tid == 0) {
        if (status) atomicOr(status, B200KV_S_TIMEOUT);
        for (int i = b; i < min(b + kRbStages, blocks); ++i) dt_mbar_wait(dt_smem(bars + i % kRbStages), (i / kRbStages) & 1);
      }
      __syncthreads();
      return;
    }
    if (tid == 0 && b + kRbStages < blocks) fetch(b + kRbStages);
  }
  rb_state_store<kLanes, kR>(S, state, D, P, P4, p0, l);
  rec_keep_inputs<T>(rec, in, x, blockIdx.x, gridDim.x, 32 * kRbWarps);
}

// The same with two warps for the columns of one, for steps with so few portions that their blocks leave schedulers idle: the first finds
// the writes (sums with k, u), the second reads out (sums with q, the outputs) on a copy of the state, which both advance.  The chain of a
// block of eight tokens is then without the read-out, and nothing holds the warps together but what they hand on: u by a barrier, a stage's
// end by another, which the fetching lane of a reading warp waits for.  The arithmetic is the same, bit for bit.
template <typename T, int kLanes, int kR>
__global__ void __launch_bounds__(64 * kRbWarps, 3)
rb_scan_split_kernel(const b200dec_recurrence rec, const b200dec_recurrence_in in, const T* conv, int conv_stride,
                     const b200dec_entries ent, const float* ws, float* __restrict__ out, int slabs, int32_t* status) {
  constexpr int Dp = kLanes * kR, kFloats = rb_floats(Dp), kQuads = kR / 4, kGroups = 32 / kLanes;
  constexpr int kM = kLanes / 8, kC = kRbCols / kM;  // after the exchange a lane holds kC columns of one token
  extern __shared__ __align__(128) float rb_smem[];  // [kRbStages][kFloats]
  __shared__ __align__(16) float ubuf[kRbStages][kRbWarps][kGroups][kRbTok][kRbCols];
  __shared__ __align__(8) uint64_t full[kRbStages], empty[kRbStages], written[kRbStages][kRbWarps];
  pdl_enter();
  const int e = blockIdx.y, h = blockIdx.x / slabs, slab = blockIdx.x - h * slabs, tid = threadIdx.x;
  if (e < *ent.num_decoding) { pdl_wait(); return; }
  const RecEntry x = rec_entry(ent, rec, e, status);
  if (tid == 0) {
    for (int i = 0; i < kRbStages; ++i) {
      dt_mbar_init(dt_smem(full + i), 1);
      dt_mbar_init(dt_smem(empty + i), 2 * kRbWarps);
      for (int w = 0; w < kRbWarps; ++w) dt_mbar_init(dt_smem(&written[i][w]), 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  __syncthreads();
  pdl_wait();
  if (x.n == 0) return;
  const int D = rec.dim, P = rec.vdim, P4 = rec_round4(P), blocks = (x.n + kRbTok - 1) / kRbTok;
  const int lane = tid & 31, warp = (tid >> 5) % kRbWarps, grp = lane / kLanes, l = tid % kLanes;
  const bool reads = tid >= 32 * kRbWarps;
  const int p0 = ((slab * kRbWarps + warp) * kGroups + grp) * kRbCols;  // the first column
  const int tok = l / kM, pc = p0 + kC * (l % kM);                  // what this lane holds after the exchange
  const long long at0 = (long long)rb_first(ent, e) * rec.heads + h;
  const bool fetches = tid == 32 * kRbWarps;
  int sent = 0;
  auto fetch = [&]() {
    const uint32_t bar = dt_smem(full + sent % kRbStages);
    dt_expect_tx(bar, kFloats * 4);
    rb_bulk(dt_smem(rb_smem + (sent % kRbStages) * kFloats), ws + (at0 + (long long)sent * rec.heads) * kFloats, kFloats * 4, bar);
    ++sent;
  };
  if (fetches)
    while (sent < min(kRbStages, blocks)) fetch();
  float* state = rec.state + ((long long)x.slot * rec.heads + h) * D * P4;
  rb_pair S[kRbCols][kR / 2];  // [column][pair of rows]
  rb_state_load<kLanes, kR>(S, state, x.pos > 0 && p0 < P4, D, P4, p0, l);
  bool dead = false;
  ulonglong2 ka[kRbTok][kQuads], decay[kQuads];
  float r[kRbCols * kRbTok], row[kRbTok];
  // block b's phase of a barrier of its stage, alike for all lanes of the warp
  auto warp_wait = [&](const uint64_t* bar, int b) { return __all_sync(0xffffffffu, dt_mbar_wait(dt_smem(bar), (b / kRbStages) & 1)) != 0; };
  // the sums of vectors `vec` with the state in front of block b; then what advances the state, and the token's row of T (0) or B (1)
  auto look = [&](int b, int vec) {
    const int s = b % kRbStages;
    if (!warp_wait(full + s, b)) return false;
    const float* st = rb_smem + s * kFloats;
    const uint32_t mine = dt_smem(st) + 16 * l;
    rb_rows<kLanes, kR>(mine, vec, tok, ka);
    rb_sums<kR>(S, ka, r);
    rb_rows<kLanes, kR>(mine, 2, 0, ka);
    rb_exchange<kLanes>(r, l);
#pragma unroll
    for (int j = 0; j < kQuads; ++j) decay[j] = rb_lds(mine + 4 * (3 * kRbTok * Dp + 4 * kLanes * j));
    rb_row8(st + 3 * kRbTok * Dp + Dp + (vec * kRbTok + tok) * kRbTok, row);
    return true;
  };
  if (!reads) {
    // v of this lane's token and columns in block b; kept as loaded until it is used, so that nothing waits for it
    auto value = [&](int b, T (&v)[kC]) {
      const int t = b * kRbTok + tok;
      const T* src = conv + (long long)(x.first + t) * conv_stride + rec.off_v + h * P + pc;
#pragma unroll
      for (int c = 0; c < kC; ++c) v[c] = t < x.n && pc + c < P ? src[c] : T(0);
    };
    T v_next[kC];
    value(0, v_next);
    for (int b = 0; b < blocks; ++b) {
      float w[kC];
#pragma unroll
      for (int c = 0; c < kC; ++c) w[c] = ld_elem(v_next + c);
      value(b + 1, v_next);
      if (!look(b, 0)) { dead = true; break; }
      const int s = b % kRbStages;
      float (&mine)[kRbTok][kRbCols] = ubuf[s][warp][grp];
#pragma unroll
      for (int c = 0; c < kC; ++c) {
        w[c] -= r[c];
        float even = 0.f, odd = 0.f;
#pragma unroll
        for (int j = 0; j < kRbTok; ++j) {
          const float wj = __shfl_sync(0xffffffffu, w[c], j * kM + l % kM, kLanes);
          if (j & 1) odd = fmaf(row[j], wj, odd); else even = fmaf(row[j], wj, even);
        }
        mine[tok][kC * (l % kM) + c] = even + odd;
      }
      __syncwarp();
      if (lane == 0) dt_mbar_arrive(dt_smem(&written[s][warp]));
      rb_update<kR>(S, decay, ka, mine);
      __syncwarp();
      if (lane == 0) dt_mbar_arrive(dt_smem(empty + s));
    }
  } else {
    for (int b = 0; b < blocks; ++b) {
      if (!look(b, 1)) { dead = true; break; }
      const int s = b % kRbStages, t = b * kRbTok + tok;
      if (!warp_wait(&written[s][warp], b)) { dead = true; break; }
      const float (&theirs)[kRbTok][kRbCols] = ubuf[s][warp][grp];
      rb_update<kR>(S, decay, ka, theirs);
#pragma unroll
      for (int c = 0; c < kC; ++c) {
        float even = r[c], odd = 0.f;
#pragma unroll
        for (int j = 0; j < kRbTok; ++j) {
          const float uj = theirs[j][kC * (l % kM) + c];
          if (j & 1) odd = fmaf(row[j], uj, odd); else even = fmaf(row[j], uj, even);
        }
        if (t < x.n && pc + c < P) out[((long long)(x.first + t) * rec.heads + h) * P + pc + c] = even + odd;
      }
      __syncwarp();
      if (lane == 0) dt_mbar_arrive(dt_smem(empty + s));
      if (fetches && sent < blocks) {
        if (dt_mbar_wait(dt_smem(empty + s), (b / kRbStages) & 1)) fetch(); else dead = true;
      }
      if (__any_sync(0xffffffffu, dead)) break;
    }
  }
  if (__syncthreads_or(dead)) {
    if (fetches) {
      if (status) atomicOr(status, B200KV_S_TIMEOUT);
      for (int i = max(sent - kRbStages, 0); i < sent; ++i) dt_mbar_wait(dt_smem(full + i % kRbStages), (i / kRbStages) & 1);
    }
    return;
  }
  if (!reads) rb_state_store<kLanes, kR>(S, state, D, P, P4, p0, l);
  rec_keep_inputs<T>(rec, in, x, blockIdx.x, gridDim.x, 64 * kRbWarps);
}

template <typename T, int kLanes, int kR>
static int rb_launch(const b200dec_recurrence& rec, const b200dec_recurrence_in& in, const void* conv, const b200dec_entries& ent, float* ws,
                     float* out, int32_t* status, cudaStream_t s) {
  constexpr int Dp = kLanes * kR, kCols = kRbWarps * 32 / kLanes * kRbCols;
  const int stride = (rec.channels + 7) / 8 * 8, slabs = (rec.vdim + kCols - 1) / kCols;
  const int list = ent.num_rows / kRbTok + ent.num_entries;
  // Blocks of 256 threads in one round; those of the list that have a decoding entry's place leave at once and do not
  // count: 185 rows, 16 heads of 128 beside 16 decoding entries, with the convolution and the scan 45.2 -> 42.5 us.
  const bool few = (long long)(ent.num_rows / kRbTok + 1) * rec.heads <= 4 * device_sms();
  const int rc = launch_result(launch_chained(few ? rb_prepare_kernel<T, Dp, 2> : rb_prepare_kernel<T, Dp, 1>, dim3(list, rec.heads),
                                              dim3(few ? 256 : 128), 0, s, rec, in, (const T*)conv, stride, ent, ws, status));
  if (rc != B200KV_OK) return rc;
  const size_t smem = (size_t)kRbStages * rb_floats(Dp) * 4;
  // Warps of their own for the read-out where a portion's blocks have a multiprocessor each and all portions' blocks are one round; or, where three fit a
  // multiprocessor, two portions', or nearly three rounds.  us a layer, without and with, blocks of all portions in brackets: one of 614 rows [64] 106.6 and 100.0, [96] 110.7 and
  // 104.5, [128] 114.8 and 106.7, [160] 131.8 and 137.4, [192] 135.8 and 142.7; several of 1000 rows in all [96] 75.9 and 69.8, [128] 73.8 and
  // 67.7, [168] 88.7 and 90.7, [192] 90.2 and 93.3 (of two portions 134.2 and 133.2), [256] of two 142.4 and 141.4, [336] 92.3 and 98.7 (129.2 and 129.1), [384] 129.3 and
  // 122.0, [420] 138.3 and 129.1, [512] 114.8 and 131.1.  A step's entries are counted but for the padding one; entries that bring nothing are known on the
  // device only, and with many of them the form with fewer warps is taken, as with many portions.
  const int portions = std::max(1, ent.num_entries - 1);
  const long long sms = device_sms(), portion = (long long)rec.heads * slabs, all = portion * portions;
  const bool three = 3 * (smem + 4096) <= 227 * 1024;  // (with the static part and the reserved kilobyte)
  const bool split = portion <= sms && (all <= sms || (three && (portions == 2 || (2 * all > 5 * sms && all <= 3 * sms))));
  auto* scan = split ? rb_scan_split_kernel<T, kLanes, kR> : rb_scan_kernel<T, kLanes, kR>;
  if (!allow_smem(scan, smem)) return B200KV_E_LAUNCH;
  // Not chained: brought up beside the kernel in front, its few long-running blocks would crowd on the multiprocessors that
  // come free first.
  return launch_result(launch_kernel(false, scan, dim3(rec.heads * slabs, ent.num_entries), dim3((split ? 64 : 32) * kRbWarps), smem, s, rec, in,
                                      (const T*)conv, stride, ent, (const float*)ws, out, slabs, status));
}

template <typename T>
static int rb_run(const b200dec_recurrence& rec, const b200dec_recurrence_in& in, const void* conv, const b200dec_entries& ent, float* ws, float* out,
                  int32_t* status, cudaStream_t s) {
  if (rec.dim <= 32) return rb_launch<T, 8, 4>(rec, in, conv, ent, ws, out, status, s);
  if (rec.dim <= 64) return rb_launch<T, 16, 4>(rec, in, conv, ent, ws, out, status, s);
  if (rec.dim <= 128) return rb_launch<T, 16, 8>(rec, in, conv, ent, ws, out, status, s);
  return rb_launch<T, 32, 8>(rec, in, conv, ent, ws, out, status, s);
}

}  // namespace b200kv

using namespace b200kv;

extern "C" size_t b200dec_recurrence_blocked_workspace(const b200dec_recurrence* rec, const b200dec_entries* ent) {
  if (!rec || !ent || !rec->correct || !rec->channel_decay || rec->dim < 1 || rec->dim > 256 || rec->heads < 1) return 0;
  const int Dp = rec->dim <= 32 ? 32 : rec->dim <= 64 ? 64 : rec->dim <= 128 ? 128 : 256;
  return (size_t)(ent->num_rows / kRbTok + ent->num_entries) * rec->heads * rb_floats(Dp) * 4;
}

extern "C" int b200dec_recurrence_blocked(const b200dec_recurrence* rec, const b200dec_recurrence_in* in, const void* conv_out,
                                          const b200dec_entries* ent, float* out, void* workspace, size_t workspace_bytes, int32_t* status,
                                          void* stream) {
  const int rc = check_recurrence(rec, in, ent);
  if (rc != B200KV_OK) return rc;
  if (!ent->cu_seqlens || !conv_out || !out || !workspace) return B200KV_E_NULL;
  const size_t need = b200dec_recurrence_blocked_workspace(rec, ent);
  if (need == 0 || rec->heads > 65535 || rec->skip) return B200KV_E_SHAPE;
  if (workspace_bytes < need) return B200KV_E_WORKSPACE;
  if (!aligned(workspace, 128)) return B200KV_E_ALIGN;
  if (ent->num_entries == 0 || ent->num_rows == 0) return B200KV_OK;
  cudaStream_t s = (cudaStream_t)stream;
  return rec->elem == 2 ? rb_run<uint16_t>(*rec, *in, conv_out, *ent, (float*)workspace, out, status, s)
                        : rb_run<float>(*rec, *in, conv_out, *ent, (float*)workspace, out, status, s);
}
