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
#include "common.cuh"

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

// RG: row groups (D <= ROWS * RG); a thread's rows are rg, rg + RG, ...
template <int RG, int VEC, bool REMOVAL, typename T>
__global__ void __launch_bounds__(THREADS) state_step_kernel(const StepParams p) {
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
    for (int i = tid; i < NV * D; i += THREADS) vec[(i / D) * (ROWS * RG) + i % D] = src[i];
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

template <int RG, typename T>
int dispatch(const StepParams& p, bool removal, bool vec, int entries, cudaStream_t stream) {
  const int cols = THREADS / RG * (vec ? 4 : 1);
  const dim3 grid(entries, p.heads, (p.V + cols - 1) / cols);
  if (vec)
    return removal ? jv_launch(state_step_kernel<RG, 4, true, T>, grid, dim3(THREADS), 0, stream, p)
                   : jv_launch(state_step_kernel<RG, 4, false, T>, grid, dim3(THREADS), 0, stream, p);
  return removal ? jv_launch(state_step_kernel<RG, 1, true, T>, grid, dim3(THREADS), 0, stream, p)
                 : jv_launch(state_step_kernel<RG, 1, false, T>, grid, dim3(THREADS), 0, stream, p);
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
  StepParams p{packed, v, v_stride, v_off, out, state, slot_stride, state_n, nq, nq_stride, cu_seqlens, slots, n_slots, heads, D, V,
               work, compact, status};
  const bool vec = V % 4 == 0 && ((uintptr_t)state & 15) == 0 && slot_stride % 4 == 0;
  JV_DISPATCH_DTYPE(v_dtype, T, {
    if (D <= 64) return dispatch<8, T>(p, removal != 0, vec, entries, stream);
    if (D <= 128) return dispatch<16, T>(p, removal != 0, vec, entries, stream);
    return dispatch<32, T>(p, removal != 0, vec, entries, stream);
  });
  return JV_ERR_UNSUPPORTED;
}
