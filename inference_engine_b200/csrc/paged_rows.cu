// The paged cache of unquantised rows: rotary positions + unit norm + write of keys and values (one kernel; a second one
// norms whole projections first and rotates neighbouring channels), and the
// general attention over it (any sizes, bf16 or fp32, prompt portions and decoding alike) on the CUDA cores.
#include <algorithm>
#include <type_traits>

#include "dec_common.cuh"

namespace b200kv {

constexpr int kRwWarps = 8;
constexpr int kRwMaxPairs = 16;  // a lane holds up to 32 channels: heads of up to 1024 (2: heads of up to 128)

__device__ __forceinline__ float2 rw_load2(const uint16_t* p) {
  const uint32_t u = *reinterpret_cast<const uint32_t*>(p);
  return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
}
__device__ __forceinline__ float2 rw_load2(const float* p) { return *reinterpret_cast<const float2*>(p); }

// One warp per (row, head), heads in the order q | k | v.  A lane owns channels 2 * lane + 64 * i and the next one.
// kPairs: head sizes, half and the row stride are even, so both channels are loaded and rotated together.
template <typename T, bool kPairs, int kMax>
__global__ void __launch_bounds__(kRwWarps * 32)
rope_write_kernel(const T* qkv, long long qkv_stride, b200dec_rows rows, DecCache c, const float* cos_sin,
                  int table_len, int half, int heads, int write_kv, int unit_norm, float eps, T* __restrict__ q_out, int32_t* status) {
  pdl_enter();
  const int hkv = write_kv ? c.heads : 0, per_row = heads + 2 * hkv;
  const int item = blockIdx.x * kRwWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= rows.num_rows * per_row) return;
  const int r = item / per_row, j = item - r * per_row;
  const int kind = j < heads ? 0 : (j < heads + hkv ? 1 : 2);  // q, k, v
  int seq = r, pos;
  if (rows.seq_ids) {
    seq = rows.seq_ids[r];
    pos = rows.positions[r];
  } else {
    if (r >= *rows.num_decoding) {  // an idle row: nothing is written to the cache, q reads as zero
      pdl_wait();
      if (kind == 0)
        for (int ch = lane; ch < c.k_row; ch += 32) st_elem(q_out + ((long long)r * heads + j) * c.k_row + ch, 0.f);
      return;
    }
    pos = rows.cached_lens[r];
  }
  const bool ok = pos >= 0 && (half == 0 || pos < table_len);
  if (!ok) {
    if (lane == 0 && status) atomicOr(status, B200KV_S_BAD_POSITION);
    pos = 0;
  }
  T* dst;
  int dim = c.k_dim, row_len = c.k_row;
  long long src_off;
  if (kind == 0) {
    dst = q_out + ((long long)r * heads + j) * c.k_row;
    src_off = (long long)j * c.k_dim;
  } else {
    const int h = kind == 1 ? j - heads : j - heads - hkv;
    const int page = ok ? dec_page(c, seq, pos, lane == 0 ? status : nullptr) : -1;
    if (page < 0) return;
    const long long at = dec_row(c, page, h, pos % c.P);
    if (kind == 1) {
      dst = (T*)c.k + at * c.k_row;
      src_off = (long long)(heads + h) * c.k_dim;
    } else {
      dst = (T*)c.v + at * c.v_row;
      src_off = (long long)(heads + hkv) * c.k_dim + (long long)h * c.v_dim;
      dim = c.v_dim;
      row_len = c.v_row;
    }
  }
  pdl_wait();
  const T* src = qkv + r * qkv_stride + src_off;
  float y[kMax][2];
  float ss = 0.f;
  const float2* cs = reinterpret_cast<const float2*>(cos_sin) + (long long)pos * half;
#pragma unroll
  for (int i = 0; i < kMax; ++i) {
    y[i][0] = y[i][1] = 0.f;
    if (kPairs && 64 * i < dim) {
      const int ch = 64 * i + 2 * lane;
      if (ch < dim) {
        float2 v = rw_load2(src + ch);
        if (kind < 2 && ch < 2 * half) {
          const bool low = ch < half;
          const float2 other = rw_load2(src + (low ? ch + half : ch - half));
          const float4 a = *reinterpret_cast<const float4*>(cs + (low ? ch : ch - half));  // cos, sin of both
          const float s0 = low ? -a.y : a.y, s1 = low ? -a.w : a.w;
          v = make_float2(v.x * a.x + other.x * s0, v.y * a.z + other.y * s1);
        }
        y[i][0] = v.x;
        y[i][1] = v.y;
        ss = fmaf(v.x, v.x, fmaf(v.y, v.y, ss));
      }
    } else if (64 * i < dim) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int ch = 64 * i + 2 * lane + e;
        float v = 0.f;
        if (ch < dim) {
          v = ld_elem(src + ch);
          if (kind < 2 && ch < 2 * half) {
            const bool low = ch < half;
            const float other = ld_elem(src + (low ? ch + half : ch - half));
            const float2 a = cs[low ? ch : ch - half];
            v = low ? v * a.x - other * a.y : v * a.x + other * a.y;
          }
        }
        y[i][e] = v;
        ss = fmaf(v, v, ss);
      }
    }
  }
  float inv = 1.f;
  if (kind < 2 && unit_norm) inv = 1.0f / sqrtf(warp_sum(ss) / (float)dim + eps);
#pragma unroll
  for (int i = 0; i < kMax; ++i) {
    const int ch = 64 * i + 2 * lane;
    if (ch < row_len) {  // row_len is even; channels behind dim are zero
      if (sizeof(T) == 2)
        *reinterpret_cast<uint32_t*>(dst + ch) = float_to_bf16_bits(y[i][0] * inv) | (float_to_bf16_bits(y[i][1] * inv) << 16);
      else
        *reinterpret_cast<float2*>(dst + ch) = make_float2(y[i][0] * inv, y[i][1] * inv);
    }
  }
}

// ---------------------------------------------------------------- the same by whole rows
// Eight channels as they lie in memory, until their arithmetic.
template <typename T>
struct Raw8 {
  uint4 v[sizeof(T) / 2];
};
template <typename T>
__device__ __forceinline__ Raw8<T> ld_raw8(const T* p) {
  Raw8<T> r;
#pragma unroll
  for (int i = 0; i < (int)sizeof(T) / 2; ++i) r.v[i] = reinterpret_cast<const uint4*>(p)[i];
  return r;
}
__device__ __forceinline__ void raw_floats(const Raw8<uint16_t>& r, float (&f)[8]) { unpack8(r.v[0], f); }
__device__ __forceinline__ void raw_floats(const Raw8<float>& r, float (&f)[8]) {
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    f[4 * i] = __uint_as_float(r.v[i].x); f[4 * i + 1] = __uint_as_float(r.v[i].y);
    f[4 * i + 2] = __uint_as_float(r.v[i].z); f[4 * i + 3] = __uint_as_float(r.v[i].w);
  }
}
// Four (cos, sin) or eight floats
__device__ __forceinline__ void ld_floats8(const float* p, float (&f)[8]) { ld_vec(p, f); }

// One block per row, kLanes lanes per head, eight channels a lane: what rope_write_kernel's warps each find for themselves (the
// row's position and page, divisions, a lane's angles) is found once for all heads, and memory moves in 16 bytes.  For sizes and strides
// that are multiples of eight channels.  Bound by the chain of a row's loads; its own come before the page is looked at, and two heads
// of a group of lanes at a time leave room for more blocks than four (1024 rows 7.5 against 10.8 us).  us, rope_write_kernel -> this:
// 1024 rows of 32 heads of 128 13.4 -> 7.5, 300 rows 6.1 -> 5.2, 60 rows 4.0 -> 4.4; 200 rows in fp32 7.7 -> 6.9.
template <typename T, int kLanes>
__global__ void __launch_bounds__(512)
rope_rows_kernel(const T* qkv, long long qkv_stride, b200dec_rows rows, DecCache c, const float* cos_sin,
                 int table_len, int half, int heads, int write_kv, int unit_norm, float eps, T* __restrict__ q_out, int32_t* status) {
  constexpr int kAtOnce = 2;  // heads of a group of lanes whose loads are in flight together
  pdl_enter();
  const int r = blockIdx.x, tid = threadIdx.x, gl = tid % kLanes, groups = blockDim.x / kLanes;
  const int hkv = write_kv ? c.heads : 0, per_row = heads + 2 * hkv;
  int seq = r, pos;
  if (rows.seq_ids) {
    seq = rows.seq_ids[r];
    pos = rows.positions[r];
  } else {
    if (r >= *rows.num_decoding) {  // an idle row: nothing is written to the cache, q reads as zero
      pdl_wait();
      for (int i = tid; i < heads * c.k_row; i += blockDim.x) st_elem(q_out + (long long)r * heads * c.k_row + i, 0.f);
      return;
    }
    pos = rows.cached_lens[r];
  }
  const bool ok = pos >= 0 && (half == 0 || pos < table_len);
  if (!ok) {
    if (tid == 0 && status) atomicOr(status, B200KV_S_BAD_POSITION);
    pos = 0;
  }
  const int col = pos / c.P, prow = pos - col * c.P;  // the page, asked for here and looked at behind the row's loads
  const bool listed = ok && hkv > 0 && col < c.max_pages;
  const int id = listed ? c.table[(long long)seq * c.table_stride + col] : -1;
  const int ch = 8 * gl;
  const bool turned = ch < 2 * half, low = ch < half;
  const int partner = (tid & 31) + (turned ? (low ? half / 8 : -(half / 8)) : 0);
  pdl_wait();
  float cs[8], sn[8];
  if (turned) {
    const float* a = cos_sin + 2 * ((long long)pos * half + (low ? ch : ch - half));
    float x[2][8];
    ld_floats8(a, x[0]);
    ld_floats8(a + 8, x[1]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      cs[i] = x[i / 4][2 * (i % 4)];
      const float v = x[i / 4][2 * (i % 4) + 1];
      sn[i] = low ? -v : v;
    }
  }
  const unsigned lanes = kLanes == 32 ? 0xffffffffu : ((1u << kLanes) - 1) << ((tid & 31) / kLanes * kLanes);
  const T* src = qkv + r * qkv_stride;
  long long at0 = 0;
  bool stored = false;
  for (int j0 = tid / kLanes; j0 < per_row; j0 += kAtOnce * groups) {
    Raw8<T> own[kAtOnce];
#pragma unroll
    for (int u = 0; u < kAtOnce; ++u) {
      const int j = j0 + u * groups;
      if (j >= per_row) break;
      const bool is_v = j >= heads + hkv;
      const T* from = src + (is_v ? (heads + hkv) * c.k_dim + (j - heads - hkv) * c.v_dim : j * c.k_dim) + ch;
      if (ch < (is_v ? c.v_dim : c.k_dim)) own[u] = ld_raw8(from);
    }
    stored = listed && id >= 0 && id < c.num_pages;
    at0 = stored ? dec_row(c, id, 0, prow) : 0;
#pragma unroll
    for (int u = 0; u < kAtOnce; ++u) {
      const int j = j0 + u * groups;
      if (j >= per_row) break;
      const bool is_v = j >= heads + hkv, some = ch < (is_v ? c.v_dim : c.k_dim);
      float y[8];
      raw_floats(own[u], y);
      if (!is_v) {
        float ss = 0.f;
        if (half > 0) {
          Raw8<T> other;  // the partner's channels
#pragma unroll
          for (int i = 0; i < (int)sizeof(T) / 2; ++i) {
            other.v[i].x = __shfl_sync(lanes, own[u].v[i].x, partner);
            other.v[i].y = __shfl_sync(lanes, own[u].v[i].y, partner);
            other.v[i].z = __shfl_sync(lanes, own[u].v[i].z, partner);
            other.v[i].w = __shfl_sync(lanes, own[u].v[i].w, partner);
          }
          if (turned) {
            float o[8];
            raw_floats(other, o);
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = y[i] * cs[i] + o[i] * sn[i];
          }
        }
        if (some) {
#pragma unroll
          for (int i = 0; i < 8; ++i) ss = fmaf(y[i], y[i], ss);
        }
        if (unit_norm) {
#pragma unroll
          for (int o = kLanes / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(lanes, ss, o);
          const float inv = 1.0f / sqrtf(ss / (float)c.k_dim + eps);
#pragma unroll
          for (int i = 0; i < 8; ++i) y[i] *= inv;
        }
      }
      if (!some || (j >= heads && !stored)) continue;
      T* dst = j < heads ? q_out + ((long long)r * heads + j) * c.k_row
               : is_v    ? (T*)c.v + (at0 + (long long)(j - heads - hkv) * c.P) * c.v_row
                         : (T*)c.k + (at0 + (long long)(j - heads) * c.P) * c.k_row;
      st_vec(dst + ch, y);
    }
  }
  if (ok && hkv > 0 && tid == 0 && status && !(listed && id >= 0 && id < c.num_pages))
    atomicOr(status, listed ? B200KV_S_BAD_PAGE : B200KV_S_BAD_POSITION);
}

// ---------------------------------------------------------------- norm of whole projections, interleaved rotation, write
// Sizes and strides that are multiples of eight channels: one block per row, kVecs times eight channels a thread.  Against pairs of channels
// (norm_rope_write_kernel below) a quarter of the loads, and a row's inputs as they lie, so that with many rows twice as many blocks
// fit a multiprocessor.  1024 rows of 32 heads of 128 16.4 -> 7.1 us; of 48 heads of 64 15.4 -> 6.7, 64 rows of these 6.0 -> 4.1.
template <typename T, int kVecs>
__global__ void __launch_bounds__(512)
norm_rope_rows_kernel(const T* qkv, long long qkv_stride, b200dec_rows rows, DecCache c, const float* q_norm,
                      const float* k_norm, float eps, const float* cos_sin, int table_len, int half, int heads,
                      int k_shift, int v_shift, T* __restrict__ q_out, int32_t* status) {
  __shared__ float part[2][16];
  pdl_enter();
  const int r = blockIdx.x, tid = threadIdx.x, threads = blockDim.x;
  T* qdst = q_out + (long long)r * heads * c.k_row;
  int seq = r, pos;
  if (rows.seq_ids) {
    seq = rows.seq_ids[r];
    pos = rows.positions[r];
  } else {
    if (r >= *rows.num_decoding) {  // an idle row: nothing is written to the cache, q reads as zero
      pdl_wait();
      for (int i = tid; i < heads * c.k_row; i += threads) st_elem(qdst + i, 0.f);
      return;
    }
    pos = rows.cached_lens[r];
  }
  const bool ok = pos >= 0 && (half == 0 || pos < table_len);
  if (!ok) {
    if (tid == 0 && status) atomicOr(status, B200KV_S_BAD_POSITION);
    pos = 0;
  }
  const int col = pos / c.P, prow = pos - col * c.P;  // the page, asked for here and looked at behind the row's loads
  const bool listed = ok && col < c.max_pages;
  const int id = listed ? c.table[(long long)seq * c.table_stride + col] : -1;
  const float* cs = cos_sin + 2 * (long long)pos * half;
  const int kv8 = c.k_dim / 8, vv8 = c.v_dim / 8, nq = heads * kv8, nqk = nq + c.heads * kv8, all = nqk + c.heads * vv8;  // in eights
  // head and channel of the i-th eight of this thread (of q | k heads, or of v heads)
  auto locate = [&](int p, int& h, int& ch) {
    const bool is_v = p >= nqk;
    const int m = is_v ? p - nqk : p, per = is_v ? vv8 : kv8, shift = is_v ? v_shift : k_shift;
    h = shift >= 0 ? m >> shift : m / per;
    ch = 8 * (m - h * per);
  };
  float w[8], t[8];  // of a thread's eight channels: weights, (cos, sin) of their pairs
  auto constants = [&](int p, int ch) {
    ld_floats8(p < nq ? q_norm + 8 * p : k_norm + 8 * (p - nq), w);
    if (ch < 2 * half) ld_floats8(cs + ch, t);
  };
  pdl_wait();
  if (kVecs == 1 && tid < nqk) {
    int h, ch;
    locate(tid, h, ch);
    constants(tid, ch);
  }
  Raw8<T> raw[kVecs];
  const T* src = qkv + r * qkv_stride;
#pragma unroll
  for (int i = 0; i < kVecs; ++i)
    if (tid + i * threads < all) raw[i] = ld_raw8(src + 8 * (tid + i * threads));
  const bool stored = listed && id >= 0 && id < c.num_pages;
  if (ok && !stored && tid == 0 && status) atomicOr(status, listed ? B200KV_S_BAD_PAGE : B200KV_S_BAD_POSITION);
  const long long at0 = stored ? dec_row(c, id, 0, prow) : 0;
  float sq = 0.f, sk = 0.f;
#pragma unroll
  for (int i = 0; i < kVecs; ++i) {
    const int p = tid + i * threads;
    if (p < nqk) {
      float x[8], s = 0.f;
      raw_floats(raw[i], x);
#pragma unroll
      for (int e = 0; e < 8; ++e) s = fmaf(x[e], x[e], s);
      if (p < nq) sq += s; else sk += s;
    }
  }
  sq = warp_sum(sq);
  sk = warp_sum(sk);
  if ((tid & 31) == 0) {
    part[0][tid >> 5] = sq;
    part[1][tid >> 5] = sk;
  }
  __syncthreads();
  sq = sk = 0.f;
  for (int i = 0; i < threads / 32; ++i) {
    sq += part[0][i];
    sk += part[1][i];
  }
  sq = 1.0f / sqrtf(sq / (float)(heads * c.k_dim) + eps);
  sk = 1.0f / sqrtf(sk / (float)(c.heads * c.k_dim) + eps);
#pragma unroll
  for (int i = 0; i < kVecs; ++i) {
    const int p = tid + i * threads;
    if (p >= all || (p >= nq && !stored)) continue;
    int h, ch;
    locate(p, h, ch);
    float x[8];
    raw_floats(raw[i], x);
    T* dst = (T*)c.v + (at0 + (long long)h * c.P) * c.v_row;
    if (p < nqk) {
      if (kVecs > 1) constants(p, ch);
      const float inv = p < nq ? sq : sk;
#pragma unroll
      for (int e = 0; e < 8; ++e) x[e] = x[e] * inv * w[e];
      if (ch < 2 * half) {
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          const float a = x[e], b = x[e + 1];
          x[e] = a * t[e] - b * t[e + 1];
          x[e + 1] = b * t[e] + a * t[e + 1];
        }
      }
      dst = p < nq ? qdst + h * c.k_row : (T*)c.k + (at0 + (long long)(h - heads) * c.P) * c.k_row;
    }
    st_vec(dst + ch, x);
  }
}

// Any sizes: one block per row; a thread owns channel pairs tid, tid + 256, ... of q | k | v.
constexpr int kNrThreads = 256;

// Pair p of a group of heads of `pairs` pairs each (shift: log2 of it, or -1).
__device__ __forceinline__ void nr_split(int p, int pairs, int shift, int& head, int& pr) {
  head = shift >= 0 ? p >> shift : p / pairs;
  pr = p - head * pairs;
}

// kKeep > 0: sizes and the row stride are even and a row has at most kKeep * 256 pairs, which stay in registers; their
// weights and angles are loaded beside them.  0: any sizes, the row is read twice.
template <typename T, int kKeep>
__global__ void __launch_bounds__(kNrThreads)
norm_rope_write_kernel(const T* qkv, long long qkv_stride, b200dec_rows rows, DecCache c, const float* q_norm,
                       const float* k_norm, float eps, const float* cos_sin, int table_len, int half, int heads,
                       int k_shift, int v_shift, T* __restrict__ q_out, int32_t* status) {
  __shared__ float part[2][kNrThreads / 32];
  pdl_enter();
  const int r = blockIdx.x, tid = threadIdx.x;
  T* qdst = q_out + (long long)r * heads * c.k_row;
  int seq = r, pos;
  if (rows.seq_ids) {
    seq = rows.seq_ids[r];
    pos = rows.positions[r];
  } else {
    if (r >= *rows.num_decoding) {  // an idle row: nothing is written to the cache, q reads as zero
      pdl_wait();
      for (int ch = tid; ch < heads * c.k_row; ch += kNrThreads) st_elem(qdst + ch, 0.f);
      return;
    }
    pos = rows.cached_lens[r];
  }
  const bool ok = pos >= 0 && (half == 0 || pos < table_len);
  if (!ok) {
    if (tid == 0 && status) atomicOr(status, B200KV_S_BAD_POSITION);
    pos = 0;
  }
  const int page = ok ? dec_page(c, seq, pos, tid == 0 ? status : nullptr) : -1;
  const float2* cs = reinterpret_cast<const float2*>(cos_sin) + (long long)pos * half;
  const T* src = qkv + r * qkv_stride;
  const int nq = heads * c.k_dim, nk = c.heads * c.k_dim, all_heads = heads + c.heads;
  const long long at0 = page < 0 ? 0 : dec_row(c, page, 0, pos % c.P);
  auto put2 = [](T* dst, float a, float b) {
    if (sizeof(T) == 2) *reinterpret_cast<uint32_t*>(dst) = float_to_bf16_bits(a) | (float_to_bf16_bits(b) << 16);
    else *reinterpret_cast<float2*>(dst) = make_float2(a, b);
  };
  // where channel ch of q / k head h (q heads first) goes; only for k heads a page is needed
  auto place = [&](int h, int ch) {
    return h < heads ? qdst + h * c.k_row + ch : (T*)c.k + (at0 + (long long)(h - heads) * c.P) * c.k_row + ch;
  };
  float sq = 0.f, sk = 0.f;
  auto means = [&] {
    sq = warp_sum(sq);
    sk = warp_sum(sk);
    if ((tid & 31) == 0) {
      part[0][tid >> 5] = sq;
      part[1][tid >> 5] = sk;
    }
    __syncthreads();
    sq = sk = 0.f;
#pragma unroll
    for (int i = 0; i < kNrThreads / 32; ++i) {
      sq += part[0][i];
      sk += part[1][i];
    }
    sq = 1.0f / sqrtf(sq / (float)nq + eps);
    sk = 1.0f / sqrtf(sk / (float)nk + eps);
  };
  if constexpr (kKeep > 0) {
    const int qkp = (nq + nk) / 2, all = qkp + c.heads * c.v_dim / 2;
    float2 v[kKeep], w[kKeep], t[kKeep];
    pdl_wait();
#pragma unroll
    for (int i = 0; i < kKeep; ++i) {
      const int p = tid + i * kNrThreads;
      if (p < qkp) {
        int h, pr;
        nr_split(p, c.k_dim / 2, k_shift, h, pr);
        w[i] = *reinterpret_cast<const float2*>(2 * p < nq ? q_norm + 2 * p : k_norm + (2 * p - nq));
        t[i] = pr < half ? cs[pr] : make_float2(1.f, 0.f);
      }
    }
#pragma unroll
    for (int i = 0; i < kKeep; ++i) {
      const int p = tid + i * kNrThreads;
      if (p < all) v[i] = rw_load2(src + 2 * p);
    }
#pragma unroll
    for (int i = 0; i < kKeep; ++i) {
      const int p = tid + i * kNrThreads;
      if (p < qkp) {
        const float s2 = fmaf(v[i].x, v[i].x, v[i].y * v[i].y);
        if (2 * p < nq) sq += s2; else sk += s2;
      }
    }
    means();
#pragma unroll
    for (int i = 0; i < kKeep; ++i) {
      const int p = tid + i * kNrThreads;
      int h, pr;
      if (p < qkp) {
        nr_split(p, c.k_dim / 2, k_shift, h, pr);
        if (h >= heads && page < 0) continue;
        const float inv = h < heads ? sq : sk, a = v[i].x * inv * w[i].x, b = v[i].y * inv * w[i].y;
        put2(place(h, 2 * pr), a * t[i].x - b * t[i].y, b * t[i].x + a * t[i].y);
      } else if (p < all && page >= 0) {
        nr_split(p - qkp, c.v_dim / 2, v_shift, h, pr);
        put2((T*)c.v + (at0 + (long long)h * c.P) * c.v_row + 2 * pr, v[i].x, v[i].y);
      }
    }
    // channels behind a size are written as zero
    const int k_pad = (c.k_row - c.k_dim) / 2, v_pad = (c.v_row - c.v_dim) / 2;
    for (int i = tid; i < all_heads * k_pad; i += kNrThreads)
      if (i / k_pad < heads || page >= 0) put2(place(i / k_pad, c.k_dim + 2 * (i % k_pad)), 0.f, 0.f);
    if (page >= 0)
      for (int i = tid; i < c.heads * v_pad; i += kNrThreads)
        put2((T*)c.v + (at0 + (long long)(i / v_pad) * c.P) * c.v_row + c.v_dim + 2 * (i % v_pad), 0.f, 0.f);
  } else {
    pdl_wait();
    for (int i = tid; i < nq + nk; i += kNrThreads) {
      const float f = ld_elem(src + i);
      if (i < nq) sq = fmaf(f, f, sq); else sk = fmaf(f, f, sk);
    }
    means();
    for (int i = tid; i < all_heads * (c.k_row / 2); i += kNrThreads) {
      const int h = i / (c.k_row / 2), pr = i - h * (c.k_row / 2), ch = 2 * pr, off = h * c.k_dim + ch;  // q and k heads lie end to end
      if (h >= heads && page < 0) continue;
      const float* w = h < heads ? q_norm + off : k_norm + (off - nq);
      const float inv = h < heads ? sq : sk;
      float a = ch < c.k_dim ? ld_elem(src + off) * inv * w[0] : 0.f;
      float b = ch + 1 < c.k_dim ? ld_elem(src + off + 1) * inv * w[1] : 0.f;
      if (pr < half) {
        const float2 t = cs[pr];
        const float u = a;
        a = u * t.x - b * t.y;
        b = b * t.x + u * t.y;
      }
      put2(place(h, ch), a, b);
    }
    if (page < 0) return;
    for (int i = tid; i < c.heads * (c.v_row / 2); i += kNrThreads) {
      const int h = i / (c.v_row / 2), ch = 2 * (i - h * (c.v_row / 2));
      const T* p = src + nq + nk + h * c.v_dim + ch;
      put2((T*)c.v + (at0 + (long long)h * c.P) * c.v_row + ch, ch < c.v_dim ? ld_elem(p) : 0.f, ch + 1 < c.v_dim ? ld_elem(p + 1) : 0.f);
    }
  }
}

// ---------------------------------------------------------------- attention, one block per (row, query head)
constexpr int kArThreads = 128;
constexpr int kArKeys = 128;  // keys per block step, one score per thread
constexpr int kArPieces = 8;  // channels of the output per thread: v_dim up to 1024

template <typename T>
__global__ void __launch_bounds__(kArThreads)
attn_rows_kernel(const T* q, DecCache c, b200dec_rows rows, int heads, float scale, DecAttnOpt opt, T* __restrict__ out,
                 int32_t* status) {
  extern __shared__ float ar_smem[];
  float* qs = ar_smem;                                                  // [k_dim]
  float* ps = qs + ((c.k_dim + 3) / 4) * 4;                             // [kArKeys]
  int* pages = reinterpret_cast<int*>(ps + kArKeys);                    // [kArKeys] row index of each key in the cache
  __shared__ float red[2][kArThreads / 32];
  pdl_enter();
  const int r = blockIdx.y, h = blockIdx.x, hk = h / (heads / c.heads), tid = threadIdx.x;
  T* dst = out + r * opt.out_stride + h * c.v_dim;
  int seq = r, pos;
  if (rows.seq_ids) {
    seq = rows.seq_ids[r];
    pos = rows.positions[r];
  } else {
    pos = r < *rows.num_decoding ? rows.cached_lens[r] : -1;
  }
  pdl_wait();
  if (pos < 0) {  // idle row
    for (int ch = tid; ch < c.v_dim; ch += kArThreads) st_elem(dst + ch, 0.f);
    return;
  }
  const T* qrow = q + ((long long)r * heads + h) * c.k_row;
  for (int ch = tid; ch < c.k_dim; ch += kArThreads) qs[ch] = ld_elem(qrow + ch) * scale;
  float m = opt.sink ? opt.sink[h] : -INFINITY, l = opt.sink ? 1.f : 0.f, o[kArPieces];
#pragma unroll
  for (int i = 0; i < kArPieces; ++i) o[i] = 0.f;
  for (int j0 = opt.window > 0 ? max(0, pos - opt.window + 1) : 0; j0 <= pos; j0 += kArKeys) {
    const int n = min(kArKeys, pos + 1 - j0);
    __syncthreads();
    int at = -1;
    float s = -INFINITY;
    if (tid < n) {
      const int page = dec_page(c, seq, j0 + tid, status);
      if (page >= 0) {
        at = page * c.P + (j0 + tid) % c.P;  // token slot; head and row strides are applied below
        const T* krow = (const T*)c.k + dec_row(c, page, hk, (j0 + tid) % c.P) * c.k_row;
        float acc = 0.f;
        for (int ch = 0; ch < c.k_row; ch += 4) {
          float f[4];
          ld_elem4(krow + ch, f);
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (ch + e < c.k_dim) acc = fmaf(qs[ch + e], f[e], acc);
        }
        s = acc;
      }
    }
    pages[tid] = at;
    float mx = s;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    if ((tid & 31) == 0) red[0][tid >> 5] = mx;
    __syncthreads();
    mx = fmaxf(fmaxf(red[0][0], red[0][1]), fmaxf(red[0][2], red[0][3]));
    const float mn = fmaxf(m, mx), base = mn == -INFINITY ? 0.f : mn;
    const float p = expf(s - base), alpha = expf(m - base);
    m = mn;
    ps[tid] = p;
    const float sum = warp_sum(p);
    if ((tid & 31) == 0) red[1][tid >> 5] = sum;
    __syncthreads();
    l = l * alpha + (red[1][0] + red[1][1]) + (red[1][2] + red[1][3]);
#pragma unroll
    for (int i = 0; i < kArPieces; ++i) o[i] *= alpha;
    for (int k = 0; k < n; ++k) {
      const int slot = pages[k];
      if (slot < 0) continue;
      const int page = slot / c.P;
      const T* vrow = (const T*)c.v + dec_row(c, page, hk, slot - page * c.P) * c.v_row;
      const float w = ps[k];
#pragma unroll
      for (int i = 0; i < kArPieces; ++i) {
        const int ch = tid + i * kArThreads;
        if (ch < c.v_dim) o[i] = fmaf(w, ld_elem(vrow + ch), o[i]);
      }
    }
  }
  const float inv = (l > 0.f ? 1.f / l : 0.f) * opt.factor<T>(r, h);
#pragma unroll
  for (int i = 0; i < kArPieces; ++i) {
    const int ch = tid + i * kArThreads;
    if (ch < c.v_dim) st_elem(dst + ch, o[i] * inv);
  }
}


// ---------------------------------------------------------------- attention, one block per (tile of rows, kv head)
// The rows of a tile are neighbours of one entry, and with the query heads of their kv head they make up to kAtSlots query
// rows that share every key and value: kAtKeys keys and values at a time come to shared memory in whole lines, a thread
// computes one key's scores with four query rows, and a warp keeps two query rows' softmax and output, a lane's channels
// 4 lane + 128 i + (0..3).  A score is the same chain of multiply-adds as in attn_rows_kernel, where every thread reads a key
// row of its own from L1, a line per 16 bytes: that, not the arithmetic, bounded it.  Here it is the shared-memory reads (a key
// against four query rows, a value against two) and, with few entries, one block's chain of steps.
// fp32, us, attn_rows_kernel -> this: 200 rows, 16 heads of 112 and 96, 183 -> 43; 8 entries of 550 decoding, 16 heads of 128, 420 -> 51 (with half
// the threads 67).
// A tile's keys are shared by the blocks of a cluster (at_splits), whose parts meet in its shared memory, in the order of the keys.
constexpr int kAtThreads = 256;
constexpr int kAtSlots = 16;
constexpr int kAtKeys = 64;
constexpr int kAtDots = kAtSlots * kAtKeys / kAtThreads;  // query rows of a thread's scores
constexpr int kAtOwn = kAtSlots * 32 / kAtThreads;         // query rows a warp keeps
constexpr int kAtPitch = 20;  // of the scores of one key: 16 and 4 that spread the banks
constexpr size_t kAtMostSmem = 112 * 1024;  // two blocks per multiprocessor

// 16 bytes of which the first `bytes` are copied and the others zero
__device__ __forceinline__ void at_copy16(float* dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(max(bytes, 0))
               : "memory");
}
__device__ __forceinline__ void at_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void at_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ void at_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared memory of block `rank` of the cluster, at the place where `p` lies in this one's
__device__ __forceinline__ uint32_t at_peer(const float* p, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ float2 at_peer2(const float* p, int rank) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at_peer(p, rank)) : "memory");
  return v;
}
__device__ __forceinline__ float4 at_peer4(const float* p, int rank) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at_peer(p, rank)) : "memory");
  return v;
}
template <int N>
__device__ __forceinline__ void at_read(const float* p, float (&f)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const float2 v = *reinterpret_cast<const float2*>(p + i);
    f[i] = v.x; f[i + 1] = v.y;
  }
}

__host__ __device__ constexpr size_t at_floats(int k_row, int v_row) {
  return (size_t)kAtSlots * k_row + (size_t)kAtKeys * (k_row + 4) + (size_t)kAtKeys * v_row + kAtKeys * kAtPitch;
}

template <typename T, int kPieces, bool kListed>  // kPieces: output channels, in pieces of 128; kListed: with the entries' first rows
__global__ void __launch_bounds__(kAtThreads, 2)
attn_tile_kernel(const T* q, DecCache c, b200dec_rows rows, const int32_t* __restrict__ cu_seqlens, int num_entries, int heads, int slice_heads, float scale, DecAttnOpt opt,
                 T* __restrict__ out, int32_t* status) {
  extern __shared__ __align__(16) float at_smem[];
  const int splits = gridDim.z, part = blockIdx.z;  // of the cluster's blocks
  const int kp = c.k_row + 4;  // an odd number of 16-byte words: neighbouring keys lie in different banks
  float* qs = at_smem;                  // [kAtSlots][k_row]
  float* ks = qs + kAtSlots * c.k_row;  // [kAtKeys][kp]
  float* vs = ks + kAtKeys * kp;        // [kAtKeys][v_row]
  float* ps = vs + kAtKeys * c.v_row;   // [kAtKeys][kAtPitch]
  __shared__ long long at[2][kAtKeys];  // a key's row in the cache, -1: none; of this step and the next
  constexpr int kWarps = kAtThreads / 32;
  pdl_enter();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = heads / c.heads, slices = (G + kAtSlots - 1) / kAtSlots;
  const int hk = blockIdx.x / slices, g0 = blockIdx.x % slices * slice_heads, gs = min(slice_heads, G - g0);
  // Rows r0 to r0 + n - 1, of entry seq at the positions from pos on.
  auto run = [&](const int r0, const int n, const int seq, const int pos) {
    const int slots = n * gs;
    // The block's steps.  Where the table has room for more keys than there are, only the first `parts` blocks of the cluster have some.
    int first = opt.window > 0 ? max(0, pos - opt.window + 1) : 0, end = pos + n, parts = 1;
    if (splits > 1) {
      const int steps = (end - first + kAtKeys - 1) / kAtKeys, share = (steps + splits - 1) / splits;
      parts = (steps + share - 1) / share;
      if (part >= parts) {
        if (parts > 1) {  // the others meet
          at_cluster_sync();
          at_cluster_sync();
        }
        return;
      }
      first += part * share * kAtKeys;
      end = min(end, first + share * kAtKeys);
    }
    for (int s = warp; s < kAtSlots; s += kWarps) {
      const T* src = q + ((long long)(r0 + s / gs) * heads + hk * G + g0 + s % gs) * c.k_row;
      for (int ch = lane; ch < c.k_row; ch += 32) qs[s * c.k_row + ch] = s < slots && ch < c.k_dim ? ld_elem(src + ch) * scale : 0.f;
    }
    // what this warp keeps: query rows kAtOwn warp + i
    float m[kAtOwn], l[kAtOwn], o[kAtOwn][kPieces][4];
    int last[kAtOwn], low[kAtOwn];  // the keys each of them sees
#pragma unroll
    for (int i = 0; i < kAtOwn; ++i) {
      const int s = kAtOwn * warp + i, h = hk * G + g0 + s % gs;
      last[i] = s < slots ? pos + s / gs : -1;
      low[i] = s < slots && opt.window > 0 ? max(0, last[i] - opt.window + 1) : 0;
      m[i] = opt.sink && s < slots && part == 0 ? opt.sink[h] : -INFINITY;
      l[i] = opt.sink && part == 0 ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < kPieces; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) o[i][j][k] = 0.f;
    }
    const bool mine = kAtOwn * warp < slots;
    // Keys [all_low, all_last] are seen by every query row of the tile; the others are looked at one by one, so that what a row
    // does not see (a later token, perhaps not a number) never meets it.
    const int all_last = pos, all_low = opt.window > 0 ? max(0, pos + n - opt.window) : 0;
    // the rows of the keys from j0 on
    auto look_up = [&](int j0, long long* at_rows) {
      if (tid < kAtKeys) {
        const int page = j0 + tid < end ? dec_page(c, seq, j0 + tid, status) : -1;
        at_rows[tid] = page < 0 ? -1 : dec_row(c, page, hk, (j0 + tid) % c.P);
      }
    };
    // their keys or values to shared memory, zero where there is none and behind `dim`
    auto fetch = [&](const long long* at_rows, const void* cache, int row, int dim, float* to, int pitch) {
      for (int k0 = warp; k0 < kAtKeys; k0 += 4 * kWarps) {
        long long src[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) src[u] = at_rows[k0 + u * kWarps] * row;
        for (int ch = 4 * lane; ch < row; ch += 128) {
          float* d = to + k0 * pitch + ch;
          if constexpr (sizeof(T) == 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u)
              at_copy16(d + u * kWarps * pitch, (const float*)cache + max(src[u], 0ll) + ch, src[u] < 0 ? 0 : min(16, 4 * (dim - ch)));
          } else {
            float f[4][4];
#pragma unroll
            for (int u = 0; u < 4; ++u) ld_elem4((const T*)cache + max(src[u], 0ll) + ch, f[u]);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (src[u] < 0 || ch + e >= dim) f[u][e] = 0.f;
              st_elem4(d + u * kWarps * pitch, f[u]);
            }
          }
        }
      }
      at_commit();
    };
    // The keys of a step are fetched while the values of the one before are used, its values while its scores are made.
    if (first < end) {
      look_up(first, at[0]);
      __syncthreads();
      fetch(at[0], c.k, c.k_row, c.k_dim, ks, kp);
      fetch(at[0], c.v, c.v_row, c.v_dim, vs, c.v_row);
    }
    for (int j0 = first, turn = 0; j0 < end; j0 += kAtKeys, turn ^= 1) {
      const int count = min(kAtKeys, end - j0);
      const bool more = j0 + kAtKeys < end;
      look_up(j0 + kAtKeys, at[turn ^ 1]);
      at_wait<1>();
      __syncthreads();  // the keys are there, the scores of the step before are used
      const int key = tid & (kAtKeys - 1), s0 = tid / kAtKeys * kAtDots;
      if (s0 < slots) {
        const float *kr = ks + key * kp, *qr = qs + s0 * c.k_row;
        float acc[kAtDots];
#pragma unroll
        for (int i = 0; i < kAtDots; ++i) acc[i] = 0.f;
        auto dots = [&](auto rows_at_once) {
          constexpr int kN = decltype(rows_at_once)::value;
#pragma unroll 2
          for (int ch = 0; ch < c.k_row; ch += 4) {
            const float4 kv = *reinterpret_cast<const float4*>(kr + ch);
#pragma unroll
            for (int i = 0; i < kN; ++i) {
              const float4 x = *reinterpret_cast<const float4*>(qr + i * c.k_row + ch);
              acc[i] = fmaf(x.w, kv.w, fmaf(x.z, kv.z, fmaf(x.y, kv.y, fmaf(x.x, kv.x, acc[i]))));
            }
          }
        };
        if (slots - s0 <= 2) dots(std::integral_constant<int, 2>{}); else dots(std::integral_constant<int, kAtDots>{});
#pragma unroll
        for (int i = 0; i < kAtDots; i += 4)
          *reinterpret_cast<float4*>(ps + key * kAtPitch + s0 + i) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
      }
      __syncthreads();  // the keys are used
      if (more) fetch(at[turn ^ 1], c.k, c.k_row, c.k_dim, ks, kp); else at_commit();
      at_wait<1>();
      __syncthreads();  // every thread's part of the values is there
      if (mine) {
        // softmax of the warp's query rows, keys lane and lane + 32
        float p[2][kAtOwn];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int k = lane + 32 * u, j = j0 + k;
          at_read(ps + k * kAtPitch + kAtOwn * warp, p[u]);
          const bool some = at[turn][k] >= 0;
#pragma unroll
          for (int i = 0; i < kAtOwn; ++i)
            if (!some || j > last[i] || j < low[i]) p[u][i] = -INFINITY;
        }
#pragma unroll
        for (int i = 0; i < kAtOwn; ++i) {
          float mx = fmaxf(p[0][i], p[1][i]);
#pragma unroll
          for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
          const float mn = fmaxf(m[i], mx), base = mn == -INFINITY ? 0.f : mn, alpha = expf(m[i] - base);
          m[i] = mn;
#pragma unroll
          for (int u = 0; u < 2; ++u) p[u][i] = expf(p[u][i] - base);
          l[i] = l[i] * alpha + warp_sum(p[0][i] + p[1][i]);
#pragma unroll
          for (int a = 0; a < kPieces; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) o[i][a][b] *= alpha;
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int i = 0; i < kAtOwn; i += 2)
            *reinterpret_cast<float2*>(ps + (lane + 32 * u) * kAtPitch + kAtOwn * warp + i) = make_float2(p[u][i], p[u][i + 1]);
        __syncwarp();
        auto add = [&](int k, bool every) {
          float w[kAtOwn];
          at_read(ps + k * kAtPitch + kAtOwn * warp, w);
#pragma unroll
          for (int a = 0; a < kPieces; ++a) {
            const int ch = 4 * lane + 128 * a;
            if (ch >= c.v_row) break;
            const float4 v = *reinterpret_cast<const float4*>(vs + k * c.v_row + ch);
#pragma unroll
            for (int i = 0; i < kAtOwn; ++i) {
              if (!every && (j0 + k > last[i] || j0 + k < low[i])) continue;
              o[i][a][0] = fmaf(w[i], v.x, o[i][a][0]);
              o[i][a][1] = fmaf(w[i], v.y, o[i][a][1]);
              o[i][a][2] = fmaf(w[i], v.z, o[i][a][2]);
              o[i][a][3] = fmaf(w[i], v.w, o[i][a][3]);
            }
          }
        };
        // (a key without a page has a weight and a value of zero)
        const int e0 = min(max(all_low - j0, 0), count), e1 = max(e0, min(all_last + 1 - j0, count));
        for (int k = 0; k < e0; ++k) add(k, false);
#pragma unroll 4
        for (int k = e0; k < e1; ++k) add(k, true);
        for (int k = e1; k < count; ++k) add(k, false);
      }
      __syncthreads();  // the values are used
      if (more) fetch(at[turn ^ 1], c.v, c.v_row, c.v_dim, vs, c.v_row); else at_commit();
    }
    auto store = [&](int s, float sum, const float (&v)[kPieces][4]) {
      const int r = r0 + s / gs, h = hk * G + g0 + s % gs;
      const float inv = (sum > 0.f ? 1.f / sum : 0.f) * opt.factor<T>(r, h);
#pragma unroll
      for (int a = 0; a < kPieces; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int ch = 4 * lane + 128 * a + b;
          if (ch < c.v_dim) st_elem(out + r * opt.out_stride + (long long)h * c.v_dim + ch, v[a][b] * inv);
        }
    };
    if (parts == 1) {
#pragma unroll
      for (int i = 0; i < kAtOwn; ++i)
        if (kAtOwn * warp + i < slots) store(kAtOwn * warp + i, l[i], o[i]);
      return;
    }
    // the cluster's parts meet in its shared memory: outputs where the values were, maxima and sums where the scores were
#pragma unroll
    for (int i = 0; i < kAtOwn; ++i) {
      const int s = kAtOwn * warp + i;
      if (lane == 0) *reinterpret_cast<float2*>(ps + 2 * s) = make_float2(m[i], l[i]);
#pragma unroll
      for (int a = 0; a < kPieces; ++a)
        if (4 * lane + 128 * a < c.v_row) st_elem4(vs + s * c.v_row + 4 * lane + 128 * a, o[i][a]);
    }
    at_cluster_sync();
    for (int s = part + parts * warp; s < slots; s += parts * kWarps) {
      float top = -INFINITY, sum = 0.f, v[kPieces][4] = {};
      for (int j = 0; j < parts; ++j) top = fmaxf(top, at_peer2(ps + 2 * s, j).x);
      const float base = top == -INFINITY ? 0.f : top;
      for (int j = 0; j < parts; ++j) {
        const float2 ml = at_peer2(ps + 2 * s, j);
        const float w = expf(ml.x - base);
        sum = fmaf(ml.y, w, sum);
#pragma unroll
        for (int a = 0; a < kPieces; ++a) {
          if (4 * lane + 128 * a >= c.v_row) break;
          const float4 x = at_peer4(vs + s * c.v_row + 4 * lane + 128 * a, j);
          v[a][0] = fmaf(x.x, w, v[a][0]);
          v[a][1] = fmaf(x.y, w, v[a][1]);
          v[a][2] = fmaf(x.z, w, v[a][2]);
          v[a][3] = fmaf(x.w, w, v[a][3]);
        }
      }
      store(s, sum, v);
    }
    at_cluster_sync();  // a block's shared memory stays until its peers have read it
  };
  // A tile starts at the first row of an entry and then every `most` rows.  With the entries' first rows a block finds its tile, of a list with
  // a few places too many (the rows behind the last entry are one entry more); without, there is a block for every row, and those that start
  // nothing leave.  What a row is stands in seq_ids and positions alone: the rows of a tile are done in runs of one entry's consecutive
  // positions, as a rule one run.
  const int most = kAtSlots / slice_heads;
  int r0 = blockIdx.y, left = 1, seq = r0, pos, n = 1;
  if (rows.seq_ids) {
    left = min(most, rows.num_rows - r0);
    if (kListed) {
      int lo = 0, hi = num_entries + 1;  // the last entry whose first place is not behind this block's
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (cu_seqlens[mid] / most + mid <= r0) lo = mid; else hi = mid;
      }
      const int first = lo > 0 ? cu_seqlens[lo] : 0, end = lo < num_entries ? min(cu_seqlens[lo + 1], rows.num_rows) : rows.num_rows;
      r0 = first + (r0 - (lo > 0 ? first / most + lo : 0)) * most;
      if (r0 < 0 || r0 >= end) return;
      left = min(most, end - r0);
    } else if (r0 > 0) {
      pos = rows.positions[r0];
      if (pos >= 0 && pos % most != 0 && rows.seq_ids[r0 - 1] == rows.seq_ids[r0] && rows.positions[r0 - 1] == pos - 1) return;
    }
  }
  pdl_wait();
  for (; left > 0; r0 += n, left -= n) {  // (not listed: once)
    if (rows.seq_ids) {  // the run from r0 on: lane i looks at row r0 + i
      static_assert(kAtSlots < 32, "a warp sees where a run ends");
      const int s = lane < left ? rows.seq_ids[r0 + lane] : 0, p = lane < left ? rows.positions[r0 + lane] : -1;
      seq = __shfl_sync(0xffffffffu, s, 0);
      pos = __shfl_sync(0xffffffffu, p, 0);
      const bool same = p >= 0 && s == seq && p == pos + lane && (lane == 0 || kListed || p % most != 0);
      n = max(1, __ffs(~__ballot_sync(0xffffffffu, same)) - 1);
    } else {
      pos = r0 < *rows.num_decoding ? rows.cached_lens[r0] : -1;
    }
    if (pos >= 0) {
      run(r0, n, seq, pos);
    } else if (part == 0) {  // idle row
      for (int i = tid; i < gs * c.v_dim; i += kAtThreads) st_elem(out + r0 * opt.out_stride + (hk * G + g0) * c.v_dim + i, 0.f);
    }
    if (!kListed) break;
  }
}

}  // namespace b200kv

using namespace b200kv;

// Blocks that share a tile's keys: as many as are resident at a time (two per multiprocessor), but no more than the steps that the table has
// room for; what a tile has is known on the device only, where blocks without a step leave the others to it.  A block's
// fixed cost is about two steps, so that with more than a round of blocks sharing only adds work.  us with 1 / 2 / 4 / 8, 16 heads of
// 128 over 8: an entry of 550 decoding 51.3 / 34.9 / 24.7 / 20.6, of 4000 314 / 166 / 89 / 51; 8 of 550 55.4 / 34.9 / 26.7 / 37.0, 64 of
// 550 118 / 133 / 164 / 240; 200 rows of a prompt 41.0 / 41.7 / 49.1 / 90.
static int at_splits(long long blocks, int tile_rows, long long most_keys, int window) {
  if (window > 0 && window + tile_rows < most_keys) most_keys = window + tile_rows;
  int splits = 1;
  const int resident = 2 * device_sms();
  while (splits < 8 && 2 * splits * blocks <= resident && splits * kAtKeys < most_keys) splits *= 2;
  return splits;
}

// launch_chained with the grid's z extent as clusters
template <typename... KArgs, typename... Args>
static cudaError_t launch_clusters(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
  if (grid.z == 1) return launch_chained(kernel, grid, block, smem, stream, args...);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = grid.z;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = take_chained_launch(stream) ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

static int check_rows(const b200dec_rows* r) {
  if (!r) return B200KV_E_NULL;
  if (r->num_rows < 0) return B200KV_E_SHAPE;
  if ((r->seq_ids == nullptr) != (r->positions == nullptr)) return B200KV_E_NULL;
  if (!r->seq_ids && (!r->cached_lens || !r->num_decoding)) return B200KV_E_NULL;
  return B200KV_OK;
}

// Threads of a block that does one row of `items` threads' shares.  With few rows a share each, so that a row's chain is short; with more, as
// many shares a thread, up to `most`, as let all blocks be one round (about 1024 threads of these kernels fit a multiprocessor).
// Rotation, attention and all, us with 64 / 128 / 256 / 512 threads: 1000 rows 30.8 / 28.8 / 30.8 / 34.9, 300 rows 22.6 / 21.2 / 20.6 / 22.6,
// 64 rows 45.6 / 43.2 / 42.3 / 42.2.
static int row_threads(int num_rows, int items, int most) {
  const long long round = 1024ll * device_sms();
  int threads = 512;
  while (threads > 64 && (threads / 2 >= items || (2 * items <= most * threads && (long long)num_rows * threads > round))) threads /= 2;
  return threads;
}

extern "C" int b200dec_rope_write(const void* qkv, int64_t qkv_stride, const b200dec_rows* rows, const b200dec_cache* cache,
                                  const b200kv_table* table, const float* cos_sin, int32_t table_len, int32_t half, int32_t heads,
                                  int32_t write_kv, int32_t unit_norm, float eps, void* q_out, int32_t* status, void* stream) {
  if (rows && rows->num_rows == 0) return B200KV_OK;
  if (!qkv || !q_out) return B200KV_E_NULL;
  int rc = check_rows(rows);
  if (rc == B200KV_OK) rc = check_dec_cache(cache, table);
  if (rc != B200KV_OK) return rc;
  if (half < 0 || 2 * half > cache->k_dim || (half > 0 && (!cos_sin || table_len < 1))) return B200KV_E_SHAPE;
  if (heads < 1 || heads % cache->kv_heads || cache->k_row > 64 * kRwMaxPairs || cache->v_row > 64 * kRwMaxPairs) return B200KV_E_SHAPE;
  if (!aligned(q_out, 16) || !aligned(cos_sin, 8)) return B200KV_E_ALIGN;
  const long long items = (long long)rows->num_rows * (heads + (write_kv ? 2 * cache->kv_heads : 0));
  const long long blocks = (items + kRwWarps - 1) / kRwWarps;
  if (items > 0x7FFFFFF0ll) return B200KV_E_RANGE;
  const DecCache c = dec_view(cache, table);
  cudaStream_t s = (cudaStream_t)stream;
  const bool pairs = cache->k_dim % 2 == 0 && cache->v_dim % 2 == 0 && half % 2 == 0 && qkv_stride % 2 == 0 &&
                     aligned(qkv, 2 * cache->elem) && aligned(cos_sin, 16);
  auto run = [&](auto* kernel, auto* in, auto* q) {
    return launch_result(launch_chained(kernel, dim3((unsigned)blocks), dim3(kRwWarps * 32), 0, s, in, (long long)qkv_stride, *rows, c, cos_sin,
                                        table_len, half, heads, write_kv, unit_norm, eps, q, status));
  };
  const bool eights = cache->k_dim % 8 == 0 && cache->v_dim % 8 == 0 && half % 8 == 0 && qkv_stride % 8 == 0 && aligned(qkv, 16) &&
                      aligned(cos_sin, 16) && cache->k_row <= 128 && cache->v_row <= 128;
  if (eights && rows->num_rows >= 128) {  // (fewer rows: 60 of 16 + 2 x 8 heads 4.4 us by rows, 3.8 by warps; one entry decoding 14.4 and 12.4 with its attention)
    const int lanes = cache->k_row <= 64 && cache->v_row <= 64 ? 8 : 16, per_row = heads + (write_kv ? 2 * cache->kv_heads : 0);
    const int threads = row_threads(rows->num_rows, per_row * lanes, 4);
    auto by_rows = [&](auto* kernel, auto* in, auto* q) {
      return launch_result(launch_chained(kernel, dim3(rows->num_rows), dim3(threads), 0, s, in, (long long)qkv_stride, *rows, c, cos_sin, table_len,
                                          half, heads, write_kv, unit_norm, eps, q, status));
    };
    if (cache->elem == 2)
      return by_rows(lanes == 8 ? rope_rows_kernel<uint16_t, 8> : rope_rows_kernel<uint16_t, 16>, (const uint16_t*)qkv, (uint16_t*)q_out);
    return by_rows(lanes == 8 ? rope_rows_kernel<float, 8> : rope_rows_kernel<float, 16>, (const float*)qkv, (float*)q_out);
  }
  if (cache->elem == 2) {
    if (pairs && cache->k_row <= 128 && cache->v_row <= 128) return run(rope_write_kernel<uint16_t, true, 2>, (const uint16_t*)qkv, (uint16_t*)q_out);
    return run(pairs ? rope_write_kernel<uint16_t, true, kRwMaxPairs> : rope_write_kernel<uint16_t, false, kRwMaxPairs>, (const uint16_t*)qkv,
               (uint16_t*)q_out);
  }
  return run(pairs ? rope_write_kernel<float, true, kRwMaxPairs> : rope_write_kernel<float, false, kRwMaxPairs>, (const float*)qkv, (float*)q_out);
}

extern "C" int b200dec_norm_rope_write(const void* qkv, int64_t qkv_stride, const b200dec_rows* rows, const b200dec_cache* cache,
                                       const b200kv_table* table, const float* q_norm, const float* k_norm, float eps,
                                       const float* cos_sin, int32_t table_len, int32_t half, int32_t heads, void* q_out, int32_t* status,
                                       void* stream) {
  if (rows && rows->num_rows == 0) return B200KV_OK;
  if (!qkv || !q_out || !q_norm || !k_norm) return B200KV_E_NULL;
  int rc = check_rows(rows);
  if (rc == B200KV_OK) rc = check_dec_cache(cache, table);
  if (rc != B200KV_OK) return rc;
  if (half < 0 || 2 * half > cache->k_dim || (half > 0 && (!cos_sin || table_len < 1))) return B200KV_E_SHAPE;
  if (heads < 1 || heads % cache->kv_heads) return B200KV_E_SHAPE;
  if (!aligned(q_out, 16) || !aligned(cos_sin, 8)) return B200KV_E_ALIGN;
  const DecCache c = dec_view(cache, table);
  cudaStream_t s = (cudaStream_t)stream;
  const bool even = cache->k_dim % 2 == 0 && cache->v_dim % 2 == 0 && qkv_stride % 2 == 0 && aligned(qkv, 2 * cache->elem) &&
                    aligned(q_norm, 8) && aligned(k_norm, 8);
  const long long pairs = ((long long)(heads + cache->kv_heads) * cache->k_dim + (long long)cache->kv_heads * cache->v_dim) / 2;
  auto log2_of = [](int n) {
    for (int i = 0; i < 30; ++i)
      if (n == 1 << i) return i;
    return -1;
  };
  auto run = [&](auto* kernel, auto* in, auto* q) {
    return launch_result(launch_chained(kernel, dim3(rows->num_rows), dim3(kNrThreads), 0, s, in, (long long)qkv_stride, *rows, c, q_norm,
                                        k_norm, eps, cos_sin, table_len, half, heads, log2_of(cache->k_dim / 2), log2_of(cache->v_dim / 2), q,
                                        status));
  };
  const int items = (int)std::min<long long>(pairs / 4, 1 << 20), threads = row_threads(rows->num_rows, items, 4), vecs = (items + threads - 1) / threads;
  if (even && cache->k_dim % 8 == 0 && cache->v_dim % 8 == 0 && half % 4 == 0 && qkv_stride % 8 == 0 && aligned(qkv, 16) && aligned(q_norm, 16) &&
      aligned(k_norm, 16) && aligned(cos_sin, 16) && vecs <= 4) {
    auto by_rows = [&](auto* kernel, auto* in, auto* q) {
      return launch_result(launch_chained(kernel, dim3(rows->num_rows), dim3(threads), 0, s, in, (long long)qkv_stride, *rows, c, q_norm, k_norm,
                                          eps, cos_sin, table_len, half, heads, log2_of(cache->k_dim / 8), log2_of(cache->v_dim / 8), q, status));
    };
    if (cache->elem == 2)
      return by_rows(vecs == 1   ? norm_rope_rows_kernel<uint16_t, 1>
                     : vecs == 2 ? norm_rope_rows_kernel<uint16_t, 2> : norm_rope_rows_kernel<uint16_t, 4>,
                     (const uint16_t*)qkv, (uint16_t*)q_out);
    return by_rows(vecs == 1 ? norm_rope_rows_kernel<float, 1> : vecs == 2 ? norm_rope_rows_kernel<float, 2> : norm_rope_rows_kernel<float, 4>,
                   (const float*)qkv, (float*)q_out);
  }
  const int keep = !even ? 0 : pairs <= 4 * kNrThreads ? 4 : pairs <= 8 * kNrThreads ? 8 : pairs <= 16 * kNrThreads ? 16 : 0;
  if (cache->elem == 2)
    return run(keep == 4   ? norm_rope_write_kernel<uint16_t, 4>
               : keep == 8 ? norm_rope_write_kernel<uint16_t, 8>
               : keep      ? norm_rope_write_kernel<uint16_t, 16> : norm_rope_write_kernel<uint16_t, 0>,
               (const uint16_t*)qkv, (uint16_t*)q_out);
  return run(keep == 4   ? norm_rope_write_kernel<float, 4>
             : keep == 8 ? norm_rope_write_kernel<float, 8>
             : keep      ? norm_rope_write_kernel<float, 16> : norm_rope_write_kernel<float, 0>,
             (const float*)qkv, (float*)q_out);
}

extern "C" int b200dec_attn_rows_opt(const void* q, const b200dec_cache* cache, const b200kv_table* table, const b200dec_rows* rows,
                                     int32_t heads, float scale, const b200dec_attn_options* options, void* out, int32_t* status,
                                     void* stream) {
  return b200dec_attn_rows_entries(q, cache, table, rows, nullptr, 0, heads, scale, options, out, status, stream);
}

extern "C" int b200dec_attn_rows_entries(const void* q, const b200dec_cache* cache, const b200kv_table* table, const b200dec_rows* rows,
                                         const int32_t* cu_seqlens, int32_t num_entries, int32_t heads, float scale, const b200dec_attn_options* options, void* out,
                                         int32_t* status, void* stream) {
  if (rows && rows->num_rows == 0) return B200KV_OK;
  if (!q || !out) return B200KV_E_NULL;
  int rc = check_rows(rows);
  if (rc == B200KV_OK) rc = check_dec_cache(cache, table);
  DecAttnOpt opt;
  if (rc == B200KV_OK) rc = dec_attn_opt(options, heads, cache->v_dim, &opt);
  if (rc != B200KV_OK) return rc;
  if (heads < 1 || heads % cache->kv_heads || cache->v_dim > kArThreads * kArPieces || cache->k_dim > 1024 || num_entries < 0) return B200KV_E_SHAPE;
  if ((long long)cache->num_pages * cache->page_size > 0x7FFFFFFFll || rows->num_rows > 65535) return B200KV_E_RANGE;
  const DecCache c = dec_view(cache, table);
  cudaStream_t s = (cudaStream_t)stream;
  // Tiles as long as two of their blocks fit a multiprocessor: heads up to about 190 channels (of key and value on average).  Larger ones
  // keep the block per row and head, whose shared memory does not grow with them.  Below the line tiles are 2.2 to 14 times as fast, us: 64
  // entries of 550, 8 heads of 160 over 8, bf16 479 -> 215; a lone entry of 4000, 16 heads of 160 over 1, bf16 2516 -> 792, 16 of 184, fp32
  // 3887 -> 666; 600 rows, 64 heads of 128 over 4, fp32 5208 -> 424.
  const size_t tile_smem = at_floats(cache->k_row, cache->v_row) * 4;
  if (tile_smem <= kAtMostSmem && cache->v_row <= 256) {
    const int G = heads / cache->kv_heads, slices = (G + kAtSlots - 1) / kAtSlots, slice_heads = (G + slices - 1) / slices;
    const int most = kAtSlots / slice_heads;
    const bool listed = rows->seq_ids && cu_seqlens && num_entries > 0 && rows->num_rows / most + (long long)num_entries < 65535;
    const int blocks = listed ? rows->num_rows / most + num_entries + 1 : rows->num_rows;
    const int splits = at_splits((long long)cache->kv_heads * slices * (listed || !rows->seq_ids ? blocks : blocks / most + 1), most, (long long)table->max_pages * cache->page_size, opt.window);
    auto tiles = [&](auto* kernel, auto* in, auto* o) -> int {
      if (!allow_smem(kernel, kAtMostSmem)) return B200KV_E_LAUNCH;
      return launch_result(launch_clusters(kernel, dim3(cache->kv_heads * slices, blocks, splits), dim3(kAtThreads), tile_smem, s, in, c,
                                           *rows, listed ? cu_seqlens : nullptr, (int)num_entries, heads, slice_heads, scale, opt, o, status));
    };
    auto by_list = [&](auto some) {
      constexpr bool kListed = decltype(some)::value;
      if (cache->elem == 2)
        return tiles(cache->v_row <= 128 ? attn_tile_kernel<uint16_t, 1, kListed> : attn_tile_kernel<uint16_t, 2, kListed>, (const uint16_t*)q,
                     (uint16_t*)out);
      return tiles(cache->v_row <= 128 ? attn_tile_kernel<float, 1, kListed> : attn_tile_kernel<float, 2, kListed>, (const float*)q, (float*)out);
    };
    return listed ? by_list(std::true_type{}) : by_list(std::false_type{});
  }
  const size_t smem = (size_t)((cache->k_dim + 3) / 4 * 4 + 2 * kArKeys) * 4;
  if (cache->elem == 2)
    return launch_result(launch_chained(attn_rows_kernel<uint16_t>, dim3(heads, rows->num_rows), dim3(kArThreads), smem, s,
                                        (const uint16_t*)q, c, *rows, heads, scale, opt, (uint16_t*)out, status));
  return launch_result(launch_chained(attn_rows_kernel<float>, dim3(heads, rows->num_rows), dim3(kArThreads), smem, s, (const float*)q, c,
                                      *rows, heads, scale, opt, (float*)out, status));
}

extern "C" int b200dec_attn_rows(const void* q, const b200dec_cache* cache, const b200kv_table* table, const b200dec_rows* rows,
                                 int32_t heads, float scale, void* out, int32_t* status, void* stream) {
  return b200dec_attn_rows_opt(q, cache, table, rows, heads, scale, nullptr, out, status, stream);
}
