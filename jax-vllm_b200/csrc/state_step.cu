// The state update of recurrent.cu for steps of single tokens (decoding):
//
//     S <- diag(w) S - b (u^T S) + k v^T,   o = S^T r          (the removal term where packed holds u and b)
//
// It reads and writes every state once, which is all it costs, so a block is laid out for that and nothing else: 256 threads
// hold the whole key range of COLS columns of one (entry, head), eight rows of VEC neighbouring columns a thread, all eight loads
// under way at once; rows of a block are 128 to 512 bytes of memory in one piece.  The sums over the key channels go through
// shared memory.  An entry of several tokens is gone through in a loop with the state in registers.  Beside portions of prompts the
// entries of one token come in a list (`work`), and the rows of `packed` may be theirs alone.
//
// 48 requests of 8 heads of 128 x 256 (50 MB of states, read and written): 16.0 us (6.3 TB/s), 38.8 us on the scan for whole entries
// (which stages vectors and values for many tokens and keeps 16 channels x 4 columns a thread).
//
// The state-space layers' vectors are formed here (MAMBA) instead of being read: q = C and k = dt B of the head's group, one decay
// exp(-exp(A_log) dt) in every channel, dt = softplus(dt_raw + dt_bias), as mamba_prepare (mamba2.cu) forms them, which spares single
// tokens a launch (one token of 32 heads of 64 x 64: 1.7 and 2.75 us in two launches, 3.1 in one); those of gated linear attention (GLA) as
// gla_prepare (recurrent.cu) forms them (eight tokens of 8 heads of 128 x 256: 2.4 and 5.2, 5.1 in
// one), those of the delta rule (DELTA) as delta_prepare does (16 tokens of
// 32 heads of 64 x 64: 2.8 and 7.3, 8.0 in one).
#include "scan.cuh"
#include <math.h>
#include <type_traits>

namespace {
constexpr int THREADS = 256, ROWS = 8;     // state rows a thread

struct StepParams {
  const float* packed;                     // [n, heads, 3 or 5, D] = r, k, w (, u, b)
  const void* v; long long v_stride; int v_off;
  float* out;                              // [n, heads * V]
  float* state; long long slot_stride;
  float* state_n; float* nq; int nq_stride;  // the normaliser's column (value 1) and where its outputs go, or null
  const int* cu_seqlens; const int* slots;
  int n_slots, heads, D, V;
  const int* work; int compact;            // pairs (entry, -), or null: every entry; a row of packed for every pair, not every token
  int* status;
};
// What the kinds that form their vectors are given besides, instead of packed.
struct FormParams : StepParams {
  const void *b, *c, *dt_raw; long long bc_stride, dt_stride;      // MAMBA: rows of B, C and the raw step sizes
  const void *dt_bias, *a_log; int w_dtype, per_group;
  // GLA: q and k in b and c, the low-rank numbers in dt_raw; their matrix [heads * D, rank] and bias [heads * D] in dt_bias and a_log
  int rank; float inv_tau, q_scale;
  // DELTA: r and k in c and b, z_a in dt_raw, their biases a_bias and w_bias [heads * D] in dt_bias and a_log, zw rows of its own
  const void* zw; long long zw_stride;
};

// RG: row groups (D <= ROWS * RG); a thread's rows are rg, rg + RG, ...
enum : int { PLAIN, REMOVAL_TERM, MAMBA, GLA, DELTA };
template <int KIND> using ParamsOf = std::conditional_t<KIND == PLAIN || KIND == REMOVAL_TERM, StepParams, FormParams>;

__device__ __forceinline__ float weight_at(const void* w, int dtype, size_t i) {
  return dtype == 0 ? ((const float*)w)[i] : to_f32(((const __nv_bfloat16*)w)[i]);
}

template <int RG, int VEC, int KIND, typename T>
__global__ void __launch_bounds__(THREADS) state_step_kernel(const ParamsOf<KIND> p) {
  constexpr bool REMOVAL = KIND == REMOVAL_TERM || KIND == DELTA;
  constexpr int CQ = THREADS / RG, COLS = CQ * VEC, NV = REMOVAL ? 5 : 3;
  __shared__ float vec[NV * ROWS * RG];
  __shared__ __align__(16) float part[RG * COLS];
  __shared__ float scratch[33];
  pdl_trigger();
  pdl_wait();
  const int entry = p.work != nullptr ? p.work[2 * blockIdx.x] : blockIdx.x;
  const int h = blockIdx.y, tid = threadIdx.x, rg = tid / CQ, cq = tid % CQ;
  const int base = blockIdx.z * COLS, col = base + cq * VEC, D = p.D, V = p.V;
  const int t0 = p.cu_seqlens[entry], t1 = p.cu_seqlens[entry + 1];
  const int slot = p.slots[entry];
  if (slot < 0 || slot >= p.n_slots) {
    if (tid == 0) atomicOr(p.status, JV_STATUS_BAD_ROW);
    return;
  }
  if (t0 >= t1) return;
  const bool live = col < V;                           // V is a multiple of VEC
  float* S_g = p.state + (size_t)slot * p.slot_stride + (size_t)h * D * V + (live ? col : 0);
  float S[ROWS][VEC];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const int d = rg + RG * i;
#pragma unroll
    for (int c = 0; c < VEC; ++c) S[i][c] = 0.f;
    if (live && d < D) {
      if constexpr (VEC == 4) {
        const float4 s = *reinterpret_cast<const float4*>(S_g + (size_t)d * V);
        S[i][0] = s.x; S[i][1] = s.y; S[i][2] = s.z; S[i][3] = s.w;
      } else {
        S[i][0] = S_g[(size_t)d * V];
      }
    }
  }
  const bool norm = p.state_n != nullptr && blockIdx.z == 0;
  float* n_g = norm && tid < D ? p.state_n + (size_t)slot * p.slot_stride + (size_t)h * D + tid : nullptr;
  float n_state = n_g != nullptr ? *n_g : 0.f;
  for (int t = t0; t < t1; ++t) {
    const float* src = p.packed + ((size_t)(p.compact ? blockIdx.x : t) * p.heads + h) * NV * D;
    float vv[VEC];
    const T* vsrc = (const T*)p.v + (size_t)t * p.v_stride + p.v_off + (size_t)h * V + (live ? col : 0);
#pragma unroll
    for (int c = 0; c < VEC; ++c) vv[c] = to_f32(vsrc[c]);
    if constexpr (KIND == MAMBA) {
      if (tid < D) {
        const size_t at = (size_t)t * p.bc_stride + (size_t)(h / p.per_group) * D + tid;
        const float B = to_f32(((const T*)p.b)[at]), C = to_f32(((const T*)p.c)[at]);
        const float bias = weight_at(p.dt_bias, p.w_dtype, h), rate = weight_at(p.a_log, p.w_dtype, h);
        const float z = to_f32(((const T*)p.dt_raw)[(size_t)t * p.dt_stride + h]) + bias;
        const float dt = fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)));             // softplus, no clamp
        vec[tid] = C;
        vec[ROWS * RG + tid] = dt * B;
        vec[2 * ROWS * RG + tid] = expf(-expf(rate) * dt);
      }
    } else if constexpr (KIND == GLA) {
      if (tid < D) {
        const size_t e = (size_t)h * D + tid, at = (size_t)t * p.bc_stride + e;
        const float q = to_f32(((const T*)p.b)[at]), k = to_f32(((const T*)p.c)[at]), bias = weight_at(p.a_log, p.w_dtype, e);
        const T* low = (const T*)p.dt_raw + (size_t)t * p.dt_stride;
        float z = 0.f;
#pragma unroll 8
        for (int r = 0; r < p.rank; ++r) z = fmaf(weight_at(p.dt_bias, p.w_dtype, e * p.rank + r), to_f32(low[r]), z);
        vec[tid] = q * p.q_scale;
        vec[ROWS * RG + tid] = k;
        vec[2 * ROWS * RG + tid] = expf(log_sigmoid(z + bias) * p.inv_tau);
      }
    } else if constexpr (KIND == DELTA) {
      const T* row = (const T*)p.b + (size_t)t * p.bc_stride + (size_t)h * D;
      const int half = D > 64 ? 128 : 64;                // the sum of squares in the order of delta_prepare's block
      const size_t e = (size_t)h * D + tid;
      float ss = 0.f, k = 0.f, r = 0.f, za = 0.f, zd = 0.f;
      if (tid < D) {
        k = to_f32(row[tid]);
        r = to_f32(((const T*)p.c)[(size_t)t * p.bc_stride + e]);
        za = to_f32(((const T*)p.dt_raw)[(size_t)t * p.dt_stride + e]) + weight_at(p.dt_bias, p.w_dtype, e);
        zd = to_f32(((const T*)p.zw)[(size_t)t * p.zw_stride + e]) + weight_at(p.a_log, p.w_dtype, e);
      }
      if (tid < half)
        for (int d = tid; d < D; d += half) {
          const float x = to_f32(row[d]);
          ss = fmaf(x, x, ss);
        }
      ss = block_sum(ss, scratch);
      const float inv = 1.f / sqrtf(ss + 1e-6f), c = 0.60653065971263342f;      // e^(-1/2)
      if (tid < D) {
        const float a = 1.f / (1.f + expf(-za)), u = k * inv;
        vec[tid] = r;
        vec[ROWS * RG + tid] = k;
        vec[2 * ROWS * RG + tid] = expf(-c / (1.f + expf(-zd)));
        vec[3 * ROWS * RG + tid] = u;
        vec[4 * ROWS * RG + tid] = a * u;
      }
    } else {
      for (int i = tid; i < NV * D; i += THREADS) vec[(i / D) * (ROWS * RG) + i % D] = src[i];
    }
    __syncthreads();
    float dot[VEC];
    if constexpr (REMOVAL) {
#pragma unroll
      for (int c = 0; c < VEC; ++c) dot[c] = 0.f;
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        const int d = rg + RG * i;
        const float u = d < D ? vec[3 * ROWS * RG + d] : 0.f;
#pragma unroll
        for (int c = 0; c < VEC; ++c) dot[c] = fmaf(u, S[i][c], dot[c]);
      }
#pragma unroll
      for (int c = 0; c < VEC; ++c) part[rg * COLS + cq * VEC + c] = dot[c];
      __syncthreads();
#pragma unroll
      for (int c = 0; c < VEC; ++c) dot[c] = 0.f;
#pragma unroll
      for (int g = 0; g < RG; ++g)
#pragma unroll
        for (int c = 0; c < VEC; ++c) dot[c] += part[g * COLS + cq * VEC + c];
      __syncthreads();
    }
    float o[VEC];
#pragma unroll
    for (int c = 0; c < VEC; ++c) o[c] = 0.f;
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
      const int d = rg + RG * i;
      if (d < D) {
        const float r = vec[d], k = vec[ROWS * RG + d], w = vec[2 * ROWS * RG + d];
        const float b = REMOVAL ? vec[4 * ROWS * RG + d] : 0.f;
#pragma unroll
        for (int c = 0; c < VEC; ++c) {
          float s = fmaf(k, vv[c], w * S[i][c]);
          if constexpr (REMOVAL) s = fmaf(-b, dot[c], s);
          S[i][c] = s;
          o[c] = fmaf(r, s, o[c]);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < VEC; ++c) part[rg * COLS + cq * VEC + c] = o[c];
    if (norm) {                                        // the normaliser: n <- w n + k, and n . r
      float nr = 0.f;
      if (tid < D) {
        n_state = fmaf(vec[2 * ROWS * RG + tid], n_state, vec[ROWS * RG + tid]);
        nr = vec[tid] * n_state;
      }
      nr = block_sum(nr, scratch);
      if (tid == 0) p.nq[((size_t)t * p.heads + h) * p.nq_stride] = nr;
    }
    __syncthreads();
    if (tid < COLS && base + tid < V) {
      float sum = 0.f;
#pragma unroll
      for (int g = 0; g < RG; ++g) sum += part[g * COLS + tid];
      p.out[(size_t)t * p.heads * V + (size_t)h * V + base + tid] = sum;
    }
    if (t + 1 < t1) __syncthreads();                   // vectors and sums are written again
  }
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    const int d = rg + RG * i;
    if (live && d < D) {
      if constexpr (VEC == 4) *reinterpret_cast<float4*>(S_g + (size_t)d * V) = make_float4(S[i][0], S[i][1], S[i][2], S[i][3]);
      else S_g[(size_t)d * V] = S[i][0];
    }
  }
  if (n_g != nullptr) *n_g = n_state;
}

template <int RG, int KIND, typename T>
int launch(const ParamsOf<KIND>& p, bool vec, int entries, cudaStream_t stream) {
  const int cols = THREADS / RG * (vec ? 4 : 1);
  const dim3 grid(entries, p.heads, (p.V + cols - 1) / cols);
  return vec ? jv_launch(state_step_kernel<RG, 4, KIND, T>, grid, dim3(THREADS), 0, stream, p)
             : jv_launch(state_step_kernel<RG, 1, KIND, T>, grid, dim3(THREADS), 0, stream, p);
}

template <int KIND, typename T> int by_size(const ParamsOf<KIND>& p, int entries, cudaStream_t stream) {
  const bool vec = p.V % 4 == 0 && ((uintptr_t)p.state & 15) == 0 && p.slot_stride % 4 == 0;
  if (p.D <= 64) return launch<8, KIND, T>(p, vec, entries, stream);
  if (p.D <= 128) return launch<16, KIND, T>(p, vec, entries, stream);
  return launch<32, KIND, T>(p, vec, entries, stream);
}
}  // namespace

// Arguments as for jv_state_scan, without segments.  work: `entries` pairs (entry, -), or null (all entries); compact (with work,
// entries of one token): packed has a row for every pair, in their order.
JV_EXPORT int jv_state_step(const float* packed, int removal, const void* v, int v_dtype, long long v_stride, int v_off, float* out,
                            float* state, long long slot_stride, const int* cu_seqlens, const int* slots, int n_slots, int entries,
                            int heads, int D, int V, float* state_n, float* nq, int nq_stride, const int* work, int compact,
                            int* status, cudaStream_t stream) {
  if (entries == 0) return JV_OK;
  if ((compact && work == nullptr) || heads < 1 || D < 1 || D > ROWS * 32 || V < 1 || heads > 65535 || (removal && state_n != nullptr)) return JV_ERR_UNSUPPORTED;
  const StepParams p{packed, v, v_stride, v_off, out, state, slot_stride, state_n, nq, nq_stride, cu_seqlens, slots, n_slots, heads, D, V,
                     work, compact, status};
  JV_DISPATCH_DTYPE(v_dtype, T, return removal != 0 ? by_size<REMOVAL_TERM, T>(p, entries, stream) : by_size<PLAIN, T>(p, entries, stream));
  return JV_ERR_UNSUPPORTED;
}

// The same for a state-space layer, from the convolved rows [x | .. ] of `dtype` (B at b_off, C at c_off, [groups][D] each; x first)
// and the raw step sizes; dt_bias, a_log: [heads] of w_dtype.
JV_EXPORT int jv_mamba_step(const void* xbc, int dtype, long long xbc_stride, int b_off, int c_off, const void* dt_raw, long long dt_stride,
                            const void* dt_bias, const void* a_log, int w_dtype, float* out, float* state, long long slot_stride,
                            const int* cu_seqlens, const int* slots, int n_slots, int entries, int heads, int groups, int D, int V,
                            const int* work, int* status, cudaStream_t stream) {
  if (entries == 0) return JV_OK;
  if (heads < 1 || groups < 1 || heads % groups || D < 1 || D > ROWS * 32 || V < 1 || heads > 65535 || w_dtype < 0 || w_dtype > 1)
    return JV_ERR_UNSUPPORTED;
  const size_t size = dtype == 0 ? 4 : 2;
  const FormParams p{{nullptr, xbc, xbc_stride, 0, out, state, slot_stride, nullptr, nullptr, 0, cu_seqlens, slots, n_slots, heads, D, V,
                      work, 0, status},
                     (const char*)xbc + b_off * size, (const char*)xbc + c_off * size, dt_raw, xbc_stride, dt_stride, dt_bias, a_log, w_dtype,
                     heads / groups, 0, 0.f, 0.f, nullptr, 0};
  JV_DISPATCH_DTYPE(dtype, T, return (by_size<MAMBA, T>(p, entries, stream)));
  return JV_ERR_UNSUPPORTED;
}

// The same for gated linear attention, from rows of the projection: q, k and v [heads][..] and `rank` low-rank numbers at their columns;
// w_up: [heads * D, rank], bias: [heads * D] of w_dtype.
JV_EXPORT int jv_gla_step(const void* proj, int dtype, long long stride, int q_off, int k_off, int v_off, int low_off, int rank, const void* w_up,
                          const void* bias, int w_dtype, float inv_tau, float q_scale, float* out, float* state, long long slot_stride,
                          const int* cu_seqlens, const int* slots, int n_slots, int entries, int heads, int D, int V, int* status,
                          cudaStream_t stream) {
  if (entries == 0) return JV_OK;
  if (heads < 1 || D < 1 || D > ROWS * 32 || V < 1 || heads > 65535 || rank < 1 || w_dtype < 0 || w_dtype > 1) return JV_ERR_UNSUPPORTED;
  const size_t size = dtype == 0 ? 4 : 2;
  const char* row = (const char*)proj;
  const FormParams p{{nullptr, proj, stride, v_off, out, state, slot_stride, nullptr, nullptr, 0, cu_seqlens, slots, n_slots, heads, D, V,
                      nullptr, 0, status},
                     row + q_off * size, row + k_off * size, row + low_off * size, stride, stride, w_up, bias, w_dtype, 1, rank, inv_tau,
                     q_scale, nullptr, 0};
  JV_DISPATCH_DTYPE(dtype, T, return (by_size<GLA, T>(p, entries, stream)));
  return JV_ERR_UNSUPPORTED;
}

// The same for the delta rule, from rows of the projection (r, k, v and z_a [heads][D] each at their columns) and of zw; a_bias, w_bias:
// [heads * D] of w_dtype.
JV_EXPORT int jv_delta_step(const void* proj, int dtype, long long stride, int r_off, int k_off, int v_off, int a_off, const void* zw,
                            long long zw_stride, const void* a_bias, const void* w_bias, int w_dtype, float* out, float* state,
                            long long slot_stride, const int* cu_seqlens, const int* slots, int n_slots, int entries, int heads, int D, int V,
                            const int* work, int* status, cudaStream_t stream) {
  if (entries == 0) return JV_OK;
  if (heads < 1 || D < 1 || D > ROWS * 32 || V < 1 || heads > 65535 || w_dtype < 0 || w_dtype > 1) return JV_ERR_UNSUPPORTED;
  const size_t size = dtype == 0 ? 4 : 2;
  const char* row = (const char*)proj;
  const FormParams p{{nullptr, proj, stride, v_off, out, state, slot_stride, nullptr, nullptr, 0, cu_seqlens, slots, n_slots, heads, D, V,
                      work, 0, status},
                     row + k_off * size, row + r_off * size, row + a_off * size, stride, stride, a_bias, w_bias, w_dtype, 1, 0, 0.f, 0.f,
                     zw, zw_stride};
  JV_DISPATCH_DTYPE(dtype, T, return (by_size<DELTA, T>(p, entries, stream)));
  return JV_ERR_UNSUPPORTED;
}
