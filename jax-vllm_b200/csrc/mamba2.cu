// What stands around the state scan of a Mamba-2 mixer (state-space duality): per head a state S [N, E] (N state
// channels, E value channels) with
//
//   dt  = softplus(dt_raw + dt_bias)                 a = exp(-exp(A_log) * dt)
//   S  <- a S + dt * B x^T                           y = S^T C + D x
//
// which is the update of csrc/recurrent.cu's state scan (long portions: csrc/chunk_scan.cu) with the key dt * B, the
// query C and the decay a in every key channel.  B and C are shared by the heads of a group (head h uses group h / (heads / groups)).
//
// jv_mamba_prepare, one warp per (token, head): packed[t, h] = (C_g, dt * B_g, a) as float32 [3][N], from the
//   convolved rows xbc = [x | B | C] and the raw step sizes; softplus, both exponentials and the product with B in 32-bit.
// jv_mamba_finish, one block per (token, norm group): y = (o + D_h x) * silu(z), divided by the root mean square of its
//   norm group (inner / norm_groups elements), times the norm weight; 32-bit, written in the compute type.
#include "scan.cuh"
#include <math.h>

namespace {
constexpr int WARPS = 4;

template <typename T, typename TW>
__global__ void __launch_bounds__(32 * WARPS) mamba_prepare_kernel(const T* __restrict__ xbc, long long xbc_stride, int b_off,
                                                                  int c_off, const T* __restrict__ dt_raw,
                                                                  long long dt_stride, const TW* __restrict__ dt_bias,
                                                                  const TW* __restrict__ a_log, float* __restrict__ packed,
                                                                  int n, int heads, int groups, int state,
                                                                  const int* __restrict__ work,
                                                                  const int* __restrict__ cu_seqlens) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long item = (long long)blockIdx.x * WARPS + (threadIdx.x >> 5);
  if (item >= (long long)n * heads) return;
  const int row = (int)(item / heads), h = (int)(item - (long long)row * heads), t = token_of(row, work, cu_seqlens);
  const int g = h / (heads / groups);
  const float z = to_f32(dt_raw[(size_t)t * dt_stride + h]) + to_f32(dt_bias[h]);
  const float dt = fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)));             // softplus, no clamp
  const float a = expf(-expf(to_f32(a_log[h])) * dt);
  const T* B = xbc + (size_t)t * xbc_stride + b_off + (size_t)g * state;
  const T* C = xbc + (size_t)t * xbc_stride + c_off + (size_t)g * state;
  float* dst = packed + (size_t)item * 3 * state;
  for (int i = lane; i < state; i += 32) {
    dst[i] = to_f32(C[i]);
    dst[state + i] = dt * to_f32(B[i]);
    dst[2 * state + i] = a;
  }
}

// A thread keeps up to KEEP of its group's gated values in registers between the sum of squares and the write (a
// group of up to KEEP * blockDim elements is then read once); a longer group is formed twice.
constexpr int KEEP = 8;

template <typename T, typename TW>
__global__ void __launch_bounds__(1024) mamba_finish_kernel(const float* __restrict__ o, const T* __restrict__ x,
                                                            long long x_stride, const T* __restrict__ z, long long z_stride,
                                                            const TW* __restrict__ skip, const TW* __restrict__ w,
                                                            T* __restrict__ out, long long out_stride, float eps, int value_dim,
                                                            int group_size, int inner) {
  __shared__ float scratch[33];
  pdl_trigger();
  pdl_wait();
  const int t = blockIdx.x, first = blockIdx.y * group_size;
  const float* ot = o + (size_t)t * inner + first;
  const T* xt = x + (size_t)t * x_stride + first;
  const T* zt = z + (size_t)t * z_stride + first;
  auto gated = [&](int i) {
    const float zz = to_f32(zt[i]);
    return (ot[i] + to_f32(skip[(first + i) / value_dim]) * to_f32(xt[i])) * (zz / (1.f + expf(-zz)));
  };
  const bool kept = group_size <= KEEP * (int)blockDim.x;
  float ys[KEEP];
  float ss = 0.f;
  if (kept) {
#pragma unroll
    for (int u = 0; u < KEEP; ++u) {
      const int i = threadIdx.x + u * blockDim.x;
      ys[u] = i < group_size ? gated(i) : 0.f;
      ss += ys[u] * ys[u];
    }
  } else {
    for (int i = threadIdx.x; i < group_size; i += blockDim.x) { const float y = gated(i); ss += y * y; }
  }
  const float inv = rsqrtf(block_sum(ss, scratch) / (float)group_size + eps);
  T* dst = out + (size_t)t * out_stride + first;
  if (kept) {
#pragma unroll
    for (int u = 0; u < KEEP; ++u) {
      const int i = threadIdx.x + u * blockDim.x;
      if (i < group_size) dst[i] = from_f32<T>(ys[u] * inv * to_f32(w[first + i]));
    }
  } else {
    for (int i = threadIdx.x; i < group_size; i += blockDim.x) dst[i] = from_f32<T>(gated(i) * inv * to_f32(w[first + i]));
  }
}

// The same for groups in whole vectors: eight neighbouring elements a thread (all of one head), read once.
template <typename T> __device__ __forceinline__ void load_eight(float (&v)[8], const T* p) {
  if constexpr (sizeof(T) == 4) {
    const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
    const uint4 a = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  }
}
template <typename T> __device__ __forceinline__ void store_eight(T* p, const float (&v)[8]) {
  if constexpr (sizeof(T) == 4) {
    reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
  } else {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 b = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
      w[i] = *reinterpret_cast<const uint32_t*>(&b);
    }
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// EARLY: the weights are read before the kernels before this one have finished, which spares few tokens two loads' latency (one of 2,048 in
// 2.1 us against 2.3) and costs many the registers (4,096 of 8,192 in 60 against 58.6).
template <bool EARLY, typename T, typename TW>
__global__ void __launch_bounds__(1024) mamba_finish_vec_kernel(const float* __restrict__ o, const T* __restrict__ x,
                                                                long long x_stride, const T* __restrict__ z, long long z_stride,
                                                                const TW* __restrict__ skip, const TW* __restrict__ w,
                                                                T* __restrict__ out, long long out_stride, float eps,
                                                                int value_dim, int group_size, int inner) {
  __shared__ float scratch[33];
  pdl_trigger();
  const int t = blockIdx.x, i = threadIdx.x * 8, at = blockIdx.y * group_size + i;
  const bool live = i < group_size;
  float y[8] = {}, wv[8] = {}, D = 0.f;
  float ss = 0.f;
  if (EARLY && live) {
    D = to_f32(skip[at / value_dim]);
#pragma unroll
    for (int e = 0; e < 8; ++e) wv[e] = to_f32(w[at + e]);
  }
  pdl_wait();
  if (live) {
    float xv[8], zv[8];
    load_eight<float>(y, o + (size_t)t * inner + at);
    load_eight<T>(xv, x + (size_t)t * x_stride + at);
    load_eight<T>(zv, z + (size_t)t * z_stride + at);
    if (!EARLY) D = to_f32(skip[at / value_dim]);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      y[e] = (y[e] + D * xv[e]) * (zv[e] / (1.f + expf(-zv[e])));
      ss = fmaf(y[e], y[e], ss);
    }
  }
  const float inv = rsqrtf(block_sum(ss, scratch) / (float)group_size + eps);
  if (!live) return;
  if (!EARLY) {
#pragma unroll
    for (int e = 0; e < 8; ++e) wv[e] = to_f32(w[at + e]);
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) y[e] *= inv * wv[e];
  store_eight<T>(out + (size_t)t * out_stride + at, y);
}
}  // namespace

// xbc: rows of `dtype`, B at b_off and C at c_off ([groups][state] each); dt_raw: rows of `dtype`, [heads] used;
// dt_bias, a_log: [heads] of w_dtype; packed: float [n, heads, 3, state].  work, cu_seqlens: n entries of one token whose tokens
// alone are prepared, or null (all of the n rows).
JV_EXPORT int jv_mamba_prepare(const void* xbc, int dtype, long long xbc_stride, int b_off, int c_off, const void* dt_raw,
                               long long dt_stride, const void* dt_bias, const void* a_log, int w_dtype, float* packed,
                               int n, int heads, int groups, int state, const int* work, const int* cu_seqlens,
                               cudaStream_t stream) {
  if (n == 0) return JV_OK;
  if (heads < 1 || groups < 1 || heads % groups || state < 1) return JV_ERR_UNSUPPORTED;
  const long long items = (long long)n * heads;
  const dim3 grid((unsigned)((items + WARPS - 1) / WARPS));
  JV_DISPATCH_DTYPE(dtype, T, JV_DISPATCH_DTYPE(w_dtype, TW,
      return jv_launch(mamba_prepare_kernel<T, TW>, grid, dim3(32 * WARPS), 0, stream, (const T*)xbc, xbc_stride, b_off,
                       c_off, (const T*)dt_raw, dt_stride, (const TW*)dt_bias, (const TW*)a_log, packed, n, heads, groups,
                       state, work, cu_seqlens)));
  return JV_ERR_UNSUPPORTED;
}

// o: float [n, inner] (the scan's output); x, z: rows of `dtype`, [inner] used; skip: [heads] and w: [inner] of
// w_dtype; out: rows of `dtype`.  inner = heads * value_dim = norm_groups * group_size.  w_fixed: none of the kernels launched before this
// one writes skip or w, which may then be read before they have finished.
JV_EXPORT int jv_mamba_finish(const float* o, const void* x, long long x_stride, const void* z, long long z_stride,
                              int dtype, const void* skip, const void* w, int w_dtype, void* out, long long out_stride,
                              float eps, int n, int heads, int value_dim, int norm_groups, int w_fixed, cudaStream_t stream) {
  if (n == 0) return JV_OK;
  const int inner = heads * value_dim;
  if (heads < 1 || value_dim < 1 || norm_groups < 1 || inner % norm_groups) return JV_ERR_UNSUPPORTED;
  // Eight elements a thread where vectors fit (heads and groups in steps of 8, rows on 16-byte boundaries), whatever the number of
  // tokens: 4,096 tokens of 8 groups of 1,024 in 62 us against 222, 200 of 4,096 in 4.2 against 6.8, one of 4,096 in 2.8 against 4.0.
  const int group_size = inner / norm_groups, size = dtype == 0 ? 4 : 2;
  auto eights = [&](const void* q, long long stride, int bytes) { return ((uintptr_t)q & 15) == 0 && stride * bytes % 16 == 0; };
  if (value_dim % 8 == 0 && group_size % 8 == 0 && group_size <= 8192 && eights(o, inner, 4) && eights(x, x_stride, size) &&
      eights(z, z_stride, size) && eights(out, out_stride, size)) {
    const int threads = (group_size / 8 + 31) / 32 * 32;
    const bool early = w_fixed && (long long)n * norm_groups * threads <= 2048LL * jv_multiprocessors();
    JV_DISPATCH_DTYPE(dtype, T, JV_DISPATCH_DTYPE(w_dtype, TW,
        return jv_launch(early ? mamba_finish_vec_kernel<true, T, TW> : mamba_finish_vec_kernel<false, T, TW>, dim3(n, norm_groups), dim3(threads), 0, stream, o, (const T*)x, x_stride,
                         (const T*)z, z_stride, (const TW*)skip, (const TW*)w, (T*)out, out_stride, eps, value_dim, group_size,
                         inner)));
  }
  // two elements a thread where the group allows: many warps hide the loads' latency when there are few tokens
  int threads = ((inner / norm_groups + 1) / 2 + 31) / 32 * 32;
  threads = threads < 32 ? 32 : threads > 1024 ? 1024 : threads;
  JV_DISPATCH_DTYPE(dtype, T, JV_DISPATCH_DTYPE(w_dtype, TW,
      return jv_launch(mamba_finish_kernel<T, TW>, dim3(n, norm_groups), dim3(threads), 0, stream, o, (const T*)x, x_stride,
                       (const T*)z, z_stride, (const TW*)skip, (const TW*)w, (T*)out, out_stride, eps, value_dim,
                       inner / norm_groups, inner)));
  return JV_ERR_UNSUPPORTED;
}
