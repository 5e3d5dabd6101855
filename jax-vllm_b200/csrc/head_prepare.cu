// Query/key/value preparation head by head, fused with the write of the new keys and values into the paged cache.
// One warp handles one head of one token of a packed projection row `proj` (queries at q_off, keys at k_off, values at
// v_off; element offsets).  Every step is optional and all arithmetic is 32-bit (sums of squares, angles, cosines,
// sines):
//
//   queries, keys   u <- u * rsqrt(mean(u^2) + eps) * weight[D]          one weight vector shared by all heads (or none)
//                   rotation of the first rot_dim elements of the head by position * freq[j]; the rest passes
//   values          v <- v * rsqrt(mean(v^2) + eps)                      no weight
//                   rotation of the first v_rot_dim elements by position * v_freq[j]: a value that carries its own
//                   position, so that the summed output can be turned back by the query's position (jv_head_rotate)
//
// The pairs of a rotation are (j, j + dims/2) ("halves") or (2j, 2j + 1) (`interleaved`); the pair (u, v) becomes
// (u cos a - v sin a, v cos a + u sin a), for queries and keys with both cos and sin times `rot_gain`.  Queries go to q_out [n, Hq*D]; keys to k_cache[page, slot, key head, :D];
// values to v_cache[page, slot, value head, :DV].
//
// jv_head_rotate turns every head of rows [n, heads*dim] by sign * position * freq[j] (in place or into `out`).
//
// jv_rms_rows: out[t, :] = in[t, :width] * rsqrt(mean(in[t, :width]^2) + eps) * weight, for rows that are a column
// range of a wider product (the normed latent that a second product reads).
#include "common.cuh"

namespace {
constexpr int WARPS = 4;

struct HeadPrepareParams {
  const void* proj; long long row_stride; int q_off, k_off, v_off;
  void* q_out;
  const int* positions; const int* token_entry; const int* block_table; int table_width;
  const float* freq; int rot_dim; float rot_gain;
  const float* v_freq; int v_rot_dim;
  int interleaved;
  const void* q_norm_w; const void* k_norm_w; float eps;
  int v_norm, qk_unit;               // values, and queries and keys without a weight, divided by their root mean square
  void* k_cache; void* v_cache;
  int n, n_q_heads, n_k_heads, n_v_heads, key_dim, value_dim, page_size, num_pages;
  int* status;
};

// One head: dim elements at src -> dst; optional unit norm (with a weight, or none), optional rotation of the first
// `rot` elements.  The whole warp calls it.
template <typename T, typename TW>
__device__ __forceinline__ void prepare_head(const T* __restrict__ src, T* __restrict__ dst, int dim, bool normed,
                                             const TW* __restrict__ w, float eps, const float* __restrict__ freq, int rot,
                                             int interleaved, float pos, float gain, int lane) {
  float inv = 1.f;
  if (normed) {
    float ss = 0.f;
    for (int d = lane; d < dim; d += 32) { const float v = to_f32(src[d]); ss += v * v; }
    inv = rsqrtf(warp_sum(ss) / (float)dim + eps);
  }
  const int half = rot >> 1;
  for (int j = lane; j < half; j += 32) {
    const int i0 = interleaved ? 2 * j : j, i1 = interleaved ? 2 * j + 1 : j + half;
    float u = to_f32(src[i0]) * inv, v = to_f32(src[i1]) * inv;
    if (w != nullptr) { u *= to_f32(w[i0]); v *= to_f32(w[i1]); }
    float sn, cs;
    sincosf(pos * freq[j], &sn, &cs);
    sn *= gain; cs *= gain;
    dst[i0] = from_f32<T>(u * cs - v * sn);
    dst[i1] = from_f32<T>(v * cs + u * sn);
  }
  for (int d = rot + lane; d < dim; d += 32) {
    float u = to_f32(src[d]) * inv;
    if (w != nullptr) u *= to_f32(w[d]);
    dst[d] = from_f32<T>(u);
  }
}

template <typename T, typename TW>
__global__ void __launch_bounds__(32 * WARPS) head_prepare_kernel(const HeadPrepareParams p) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const bool writes = p.k_cache != nullptr;
  const int per_token = p.n_q_heads + (writes ? p.n_k_heads + p.n_v_heads : 0);
  const long long item = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5);
  if (item >= (long long)p.n * per_token) return;
  const int t = (int)(item / per_token);
  int h = (int)(item - (long long)t * per_token);
  const int posi = p.positions[t];
  const float pos = (float)posi;
  const T* row = (const T*)p.proj + (size_t)t * p.row_stride;
  if (h < p.n_q_heads) {
    prepare_head<T, TW>(row + p.q_off + (size_t)h * p.key_dim, (T*)p.q_out + ((size_t)t * p.n_q_heads + h) * p.key_dim,
                        p.key_dim, p.q_norm_w != nullptr || p.qk_unit != 0, (const TW*)p.q_norm_w, p.eps, p.freq, p.rot_dim,
                        p.interleaved, pos, p.rot_gain, lane);
    return;
  }
  h -= p.n_q_heads;
  const int entry = p.token_entry[t];
  const int page_idx = posi / p.page_size;
  const int page = (posi >= 0 && page_idx < p.table_width) ? p.block_table[(size_t)entry * p.table_width + page_idx] : -1;
  if (page < 0 || page >= p.num_pages) {
    if (lane == 0) atomicOr(p.status, JV_STATUS_BAD_PAGE);
    return;
  }
  const size_t slot = (size_t)page * p.page_size + (posi - page_idx * p.page_size);
  if (h < p.n_k_heads) {
    prepare_head<T, TW>(row + p.k_off + (size_t)h * p.key_dim, (T*)p.k_cache + (slot * p.n_k_heads + h) * p.key_dim,
                        p.key_dim, p.k_norm_w != nullptr || p.qk_unit != 0, (const TW*)p.k_norm_w, p.eps, p.freq, p.rot_dim,
                        p.interleaved, pos, p.rot_gain, lane);
    return;
  }
  h -= p.n_k_heads;
  prepare_head<T, TW>(row + p.v_off + (size_t)h * p.value_dim, (T*)p.v_cache + (slot * p.n_v_heads + h) * p.value_dim,
                      p.value_dim, p.v_norm != 0, (const TW*)nullptr, p.eps, p.v_freq, p.v_rot_dim, p.interleaved, pos, 1.f, lane);
}

// Whole vectors: a head of 8 * lanes elements (lanes a power of two up to 32) lies eight elements a thread, and its `lanes`
// threads take HPG heads of one token one after another, all asked for before the first is used, with the cos and sin of their
// places formed once.  A pair (j, j + dims/2) lies in two threads, which exchange their elements.  The general kernel above was
// bound by its two-byte accesses and a sincosf for every pair of every head (2,999 tokens of 16 + 4 + 4 heads of 64: 20.5 us,
// 10.3 so).
template <typename TW, int HPG>
__global__ void __launch_bounds__(32 * WARPS) head_prepare_vec_kernel(const HeadPrepareParams p, int lanes, int groups) {
  typedef __nv_bfloat16 T;
  pdl_trigger();
  pdl_wait();
  const int l = threadIdx.x & (lanes - 1);
  const unsigned mask = (lanes == 32 ? 0xffffffffu : (1u << lanes) - 1) << (threadIdx.x & 31 & ~(lanes - 1));
  const bool writes = p.k_cache != nullptr;
  const int per_token = p.n_q_heads + (writes ? p.n_k_heads + p.n_v_heads : 0);
  const long long gid = (long long)blockIdx.x * (blockDim.x / lanes) + threadIdx.x / lanes;
  if (gid >= (long long)p.n * groups) return;
  const int t = (int)(gid / groups), first = (int)(gid - (long long)t * groups), dim = lanes * 8, d0 = l * 8;
  const int posi = p.positions[t];
  const float pos = (float)posi;
  const T* row = (const T*)p.proj + (size_t)t * p.row_stride;
  uint4 raw[HPG];
#pragma unroll
  for (int i = 0; i < HPG; ++i) {
    const int h = first + i * groups;
    if (h >= per_token) break;
    const int off = h < p.n_q_heads ? p.q_off + h * dim
                    : h < p.n_q_heads + p.n_k_heads ? p.k_off + (h - p.n_q_heads) * dim
                                                    : p.v_off + (h - p.n_q_heads - p.n_k_heads) * dim;
    raw[i] = *reinterpret_cast<const uint4*>(row + off + d0);
  }
  size_t slot = 0;
  if (first + (HPG - 1) * groups >= p.n_q_heads && writes) {       // some head of this group may go to the cache
    const int entry = p.token_entry[t], page_idx = posi / p.page_size;
    const int page = (posi >= 0 && page_idx < p.table_width) ? p.block_table[(size_t)entry * p.table_width + page_idx] : -1;
    if (page < 0 || page >= p.num_pages) {
      if (l == 0) atomicOr(p.status, JV_STATUS_BAD_PAGE);
      slot = (size_t)-1;
    } else {
      slot = (size_t)page * p.page_size + (posi - page_idx * p.page_size);
    }
  }
  float sn[8], cs[8];
  int formed = 0;                                                   // what sn and cs were formed for: 1 queries and keys, 2 values
#pragma unroll
  for (int k = 0; k < 8; ++k) { sn[k] = 0.f; cs[k] = 1.f; }
#pragma unroll
  for (int i = 0; i < HPG; ++i) {
    int h = first + i * groups;
    if (h >= per_token) return;
    const bool is_q = h < p.n_q_heads, is_k = !is_q && h < p.n_q_heads + p.n_k_heads, is_v = !is_q && !is_k;
    if (!is_q && slot == (size_t)-1) continue;
    T* dst = is_q ? (T*)p.q_out + ((size_t)t * p.n_q_heads + h) * dim
             : is_k ? (T*)p.k_cache + (slot * p.n_k_heads + (h - p.n_q_heads)) * dim
                    : (T*)p.v_cache + (slot * p.n_v_heads + (h - p.n_q_heads - p.n_k_heads)) * dim;
    const TW* w = is_q ? (const TW*)p.q_norm_w : is_k ? (const TW*)p.k_norm_w : nullptr;
    const bool normed = is_v ? p.v_norm != 0 : w != nullptr || p.qk_unit != 0;
    const int rot = is_v ? p.v_rot_dim : p.rot_dim, half = rot >> 1;
    const float* freq = is_v ? p.v_freq : p.freq;
    const float gain = is_v ? 1.f : p.rot_gain;
    float x[8];
    T* e = reinterpret_cast<T*>(&raw[i]);
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = to_f32(e[k]);
    if (normed) {
      float ss = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) ss += x[k] * x[k];
      for (int o = lanes >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(mask, ss, o);
      const float inv = rsqrtf(ss / (float)dim + p.eps);
#pragma unroll
      for (int k = 0; k < 8; ++k) { x[k] *= inv; if (w != nullptr) x[k] *= to_f32(w[d0 + k]); }
    }
    if (rot > 0) {
      if (formed != 1 + is_v) {
        formed = 1 + is_v;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (p.interleaved) {
            if ((k & 1) == 0 && d0 + k < rot) sincosf(pos * freq[(d0 + k) >> 1], &sn[k], &cs[k]);
          } else if (d0 < rot) {
            sincosf(pos * freq[d0 + k < half ? d0 + k : d0 + k - half], &sn[k], &cs[k]);
          }
          sn[k] *= gain; cs[k] *= gain;
        }
      }
      if (p.interleaved) {
#pragma unroll
        for (int k = 0; k < 8; k += 2)
          if (d0 + k < rot) {
            const float u = x[k], v = x[k + 1];
            x[k] = u * cs[k] - v * sn[k];
            x[k + 1] = v * cs[k] + u * sn[k];
          }
      } else {
        const int step = half >> 3;                                  // the partner holds the other elements of the pairs
        const int base = threadIdx.x & 31 & ~(lanes - 1), other = base + (d0 < half ? l + step : d0 < rot ? l - step : l);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float y = __shfl_sync(mask, x[k], other);
          if (d0 < half) x[k] = x[k] * cs[k] - y * sn[k];
          else if (d0 < rot) x[k] = x[k] * cs[k] + y * sn[k];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) e[k] = from_f32<T>(x[k]);
    *reinterpret_cast<uint4*>(dst + d0) = raw[i];
  }
}

// Heads that the vectors fit: a power of two of eight-element vectors, 16-byte aligned everywhere, halves of a rotation whole vectors.
bool head_vectors_fit(const HeadPrepareParams& p, int dtype) {
  const int lanes = p.key_dim / 8;
  const auto aligned = [](const void* x) { return ((uintptr_t)x % 16) == 0; };
  const auto whole = [&](int rot) { return p.interleaved || rot % 16 == 0; };
  return dtype == 1 && p.key_dim % 8 == 0 && lanes <= 32 && (lanes & (lanes - 1)) == 0 &&
         (p.k_cache == nullptr || p.value_dim == p.key_dim) && p.row_stride % 8 == 0 && p.q_off % 8 == 0 && p.k_off % 8 == 0 &&
         p.v_off % 8 == 0 && aligned(p.proj) && aligned(p.q_out) && aligned(p.k_cache) && aligned(p.v_cache) &&
         whole(p.rot_dim) && whole(p.v_rot_dim);
}

template <typename TI, typename TO>
__global__ void __launch_bounds__(32 * WARPS) head_rotate_kernel(const TI* in, long long in_stride, TO* out, long long out_stride,
                                                                const int* __restrict__ positions,
                                                                const float* __restrict__ freq, int rot, int interleaved,
                                                                float sign, int n, int heads, int dim) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long item = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5);
  if (item >= (long long)n * heads) return;
  const int t = (int)(item / heads), h = (int)(item - (long long)t * heads);
  const float pos = sign * (float)positions[t];
  const TI* src = in + (size_t)t * in_stride + (size_t)h * dim;
  TO* dst = out + (size_t)t * out_stride + (size_t)h * dim;
  const int half = rot >> 1;
  for (int j = lane; j < half; j += 32) {
    const int i0 = interleaved ? 2 * j : j, i1 = interleaved ? 2 * j + 1 : j + half;
    const float u = to_f32(src[i0]), v = to_f32(src[i1]);
    float sn, cs;
    sincosf(pos * freq[j], &sn, &cs);
    dst[i0] = from_f32<TO>(u * cs - v * sn);
    dst[i1] = from_f32<TO>(v * cs + u * sn);
  }
  for (int d = rot + lane; d < dim; d += 32) dst[d] = from_f32<TO>(to_f32(src[d]));
}

// Whole vectors of eight elements (width and strides multiples of 8, 16-byte aligned tensors), a row's elements and
// weights asked for together and kept in registers: up to ROW_VECS vectors a thread.  Bound by the chain load - sum -
// store (rows of 1,536: 8 of them 7.1 us, 2,048 of them 9.4 us read two bytes at a time and twice; 1.6 and 4.9 so).
constexpr int ROW_VECS = 4;

template <typename TW>
__global__ void __launch_bounds__(256) rms_rows_vec_kernel(const __nv_bfloat16* __restrict__ in, long long in_stride,
                                                           __nv_bfloat16* __restrict__ out, long long out_stride,
                                                           const TW* __restrict__ w, float eps, int width) {
  __shared__ float scratch[33];
  pdl_trigger();
  pdl_wait();
  const __nv_bfloat16* src = in + (size_t)blockIdx.x * in_stride;
  __nv_bfloat16* dst = out + (size_t)blockIdx.x * out_stride;
  constexpr int W_VECS = sizeof(TW) / 2;                // vectors of sixteen bytes that eight weights fill
  uint4 raw[ROW_VECS], weight[ROW_VECS][W_VECS];
#pragma unroll
  for (int k = 0; k < ROW_VECS; ++k) {
    const int d = (threadIdx.x + k * blockDim.x) * 8;
    if (d >= width) break;
    raw[k] = *reinterpret_cast<const uint4*>(src + d);
    if (w != nullptr) {
#pragma unroll
      for (int j = 0; j < W_VECS; ++j) weight[k][j] = reinterpret_cast<const uint4*>(w + d)[j];
    }
  }
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < ROW_VECS; ++k) {
    if ((threadIdx.x + k * blockDim.x) * 8 >= width) break;
    const __nv_bfloat16* e = reinterpret_cast<const __nv_bfloat16*>(&raw[k]);
#pragma unroll
    for (int j = 0; j < 8; ++j) { const float v = to_f32(e[j]); ss += v * v; }
  }
  const float inv = rsqrtf(block_sum(ss, scratch) / (float)width + eps);
#pragma unroll
  for (int k = 0; k < ROW_VECS; ++k) {
    const int d = (threadIdx.x + k * blockDim.x) * 8;
    if (d >= width) break;
    __nv_bfloat16* e = reinterpret_cast<__nv_bfloat16*>(&raw[k]);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float v = to_f32(e[j]) * inv;
      if (w != nullptr) v *= to_f32(reinterpret_cast<const TW*>(weight[k])[j]);
      e[j] = from_f32<__nv_bfloat16>(v);
    }
    *reinterpret_cast<uint4*>(dst + d) = raw[k];
  }
}

template <typename T, typename TW>
__global__ void __launch_bounds__(128) rms_rows_kernel(const T* __restrict__ in, long long in_stride, T* __restrict__ out,
                                                       long long out_stride, const TW* __restrict__ w, float eps,
                                                       int width) {
  __shared__ float scratch[33];
  pdl_trigger();
  pdl_wait();
  const T* src = in + (size_t)blockIdx.x * in_stride;
  T* dst = out + (size_t)blockIdx.x * out_stride;
  float ss = 0.f;
  for (int d = threadIdx.x; d < width; d += blockDim.x) { const float v = to_f32(src[d]); ss += v * v; }
  const float inv = rsqrtf(block_sum(ss, scratch) / (float)width + eps);
  for (int d = threadIdx.x; d < width; d += blockDim.x) {
    float v = to_f32(src[d]) * inv;
    if (w != nullptr) v *= to_f32(w[d]);
    dst[d] = from_f32<T>(v);
  }
}
}  // namespace

// proj: [n, row_stride] of `dtype`; q_out: [n, n_q_heads*key_dim] of `dtype`; q_norm_w, k_norm_w: [key_dim] of
// `w_dtype` or null; freq: [rot_dim/2] float or null (rot_dim 0); v_freq: [v_rot_dim/2] or null; v_norm: values
// are unit-normed (no weight); qk_unit: so are queries and keys where they have no weight; caches as for
// jv_attn_prepare, both null: queries only.
JV_EXPORT int jv_head_prepare(const void* proj, int dtype, long long row_stride, int q_off, int k_off, int v_off,
                              void* q_out, const int* positions, const int* token_entry, const int* block_table,
                              int table_width, const float* freq, int rot_dim, float rot_gain, const float* v_freq, int v_rot_dim,
                              int interleaved, const void* q_norm_w, const void* k_norm_w, int w_dtype, float eps,
                              int v_norm, int qk_unit, void* k_cache, void* v_cache, int n, int n_q_heads, int n_k_heads,
                              int n_v_heads, int key_dim, int value_dim, int page_size, int num_pages, int* status,
                              cudaStream_t stream) {
  if (n == 0) return JV_OK;
  if (rot_dim < 0 || rot_dim > key_dim || (rot_dim & 1) || (rot_dim > 0 && freq == nullptr) || v_rot_dim < 0 ||
      v_rot_dim > value_dim || (v_rot_dim & 1) || (v_rot_dim > 0 && v_freq == nullptr) || key_dim < 1 || value_dim < 1 ||
      page_size < 1 || (k_cache == nullptr) != (v_cache == nullptr))
    return JV_ERR_UNSUPPORTED;
  HeadPrepareParams p;
  p.proj = proj; p.row_stride = row_stride; p.q_off = q_off; p.k_off = k_off; p.v_off = v_off; p.q_out = q_out;
  p.positions = positions; p.token_entry = token_entry; p.block_table = block_table; p.table_width = table_width;
  p.freq = freq; p.rot_dim = rot_dim; p.rot_gain = rot_gain; p.v_freq = v_freq; p.v_rot_dim = v_rot_dim; p.interleaved = interleaved ? 1 : 0;
  p.q_norm_w = q_norm_w; p.k_norm_w = k_norm_w; p.eps = eps; p.v_norm = v_norm ? 1 : 0; p.qk_unit = qk_unit ? 1 : 0;
  p.k_cache = k_cache; p.v_cache = v_cache; p.n = n; p.n_q_heads = n_q_heads; p.n_k_heads = n_k_heads; p.n_v_heads = n_v_heads;
  p.key_dim = key_dim; p.value_dim = value_dim; p.page_size = page_size; p.num_pages = num_pages; p.status = status;
  const long long items = (long long)n * (n_q_heads + (k_cache != nullptr ? n_k_heads + n_v_heads : 0));
  if (head_vectors_fit(p, dtype) && (w_dtype == 0 || w_dtype == 1)) {
    // four heads a thread once that leaves 16 warps a multiprocessor (4,096 tokens of 48 heads of 128: 32.9 us
    // against 45.8 with one), else one
    const int lanes = key_dim / 8, per_token = (int)(items / n);
    const int hpg = items * lanes / 32 >= 4LL * 148 * 16 ? 4 : 1, groups = (per_token + hpg - 1) / hpg;
    const long long threads = (long long)n * groups * lanes;
    const dim3 vgrid((unsigned)((threads + 32 * WARPS - 1) / (32 * WARPS))), block(32 * WARPS);
    if (w_dtype == 0)
      return hpg == 4 ? jv_launch(head_prepare_vec_kernel<float, 4>, vgrid, block, 0, stream, p, lanes, groups)
                      : jv_launch(head_prepare_vec_kernel<float, 1>, vgrid, block, 0, stream, p, lanes, groups);
    return hpg == 4 ? jv_launch(head_prepare_vec_kernel<__nv_bfloat16, 4>, vgrid, block, 0, stream, p, lanes, groups)
                    : jv_launch(head_prepare_vec_kernel<__nv_bfloat16, 1>, vgrid, block, 0, stream, p, lanes, groups);
  }
  const dim3 grid((unsigned)((items + WARPS - 1) / WARPS));
  JV_DISPATCH_DTYPE(dtype, T, {
    if (w_dtype == 0) return jv_launch(head_prepare_kernel<T, float>, grid, dim3(32 * WARPS), 0, stream, p);
    if (w_dtype == 1) return jv_launch(head_prepare_kernel<T, __nv_bfloat16>, grid, dim3(32 * WARPS), 0, stream, p);
  });
  return JV_ERR_UNSUPPORTED;
}

// in: [n, in_stride] of in_dtype, out: [n, out_stride] of out_dtype (may be `in`, with equal types), heads of `dim`
// elements side by side; the first `rot` elements of every head turn by sign * position * freq[j].
JV_EXPORT int jv_head_rotate(const void* in, int in_dtype, long long in_stride, void* out, int out_dtype,
                             long long out_stride, const int* positions, const float* freq, int rot, int interleaved,
                             float sign, int n, int heads, int dim, cudaStream_t stream) {
  if (n == 0 || heads == 0) return JV_OK;
  if (rot < 0 || rot > dim || (rot & 1) || (rot > 0 && freq == nullptr)) return JV_ERR_UNSUPPORTED;
  const long long items = (long long)n * heads;
  const dim3 grid((unsigned)((items + WARPS - 1) / WARPS));
  JV_DISPATCH_DTYPE(in_dtype, TI, JV_DISPATCH_DTYPE(out_dtype, TO,
      return jv_launch(head_rotate_kernel<TI, TO>, grid, dim3(32 * WARPS), 0, stream, (const TI*)in, in_stride, (TO*)out,
                       out_stride, positions, freq, rot, interleaved ? 1 : 0, sign, n, heads, dim)));
  return JV_ERR_UNSUPPORTED;
}

// in: [n, in_stride], out: [n, out_stride] of `dtype`; w: [width] of w_dtype or null.
JV_EXPORT int jv_rms_rows(const void* in, long long in_stride, void* out, long long out_stride, int dtype, const void* w,
                          int w_dtype, float eps, int n, int width, cudaStream_t stream) {
  if (n == 0) return JV_OK;
  if (width < 1) return JV_ERR_UNSUPPORTED;
  if (dtype == 1 && width % 8 == 0 && width <= 256 * 8 * ROW_VECS && in_stride % 8 == 0 && out_stride % 8 == 0 &&
      ((uintptr_t)in % 16) == 0 && ((uintptr_t)out % 16) == 0 && ((uintptr_t)w % 16) == 0) {
    int threads = (width / 8 + 31) / 32 * 32;
    if (threads > 256) threads = 256;
    JV_DISPATCH_DTYPE(w_dtype, TW,
        return jv_launch(rms_rows_vec_kernel<TW>, dim3(n), dim3(threads), 0, stream, (const __nv_bfloat16*)in, in_stride,
                         (__nv_bfloat16*)out, out_stride, (const TW*)w, eps, width));
  }
  JV_DISPATCH_DTYPE(dtype, T, JV_DISPATCH_DTYPE(w_dtype, TW,
      return jv_launch(rms_rows_kernel<T, TW>, dim3(n), dim3(128), 0, stream, (const T*)in, in_stride, (T*)out, out_stride,
                       (const TW*)w, eps, width)));
  return JV_ERR_UNSUPPORTED;
}
