// Matrix states with ONE decay a head and token, over portions of many tokens, CT tokens at a time on the tensor cores:
//
//     S <- a_t S + g_t k_t v_t^T,   o_t = scale * S^T q_t                     (S [key channel, value channel] in 32-bit)
//
//   state-space mixer    a = exp(-exp(A_log) dt), g = dt = softplus(dt_raw + dt_bias), k = B and q = C of the head's group, v = x
//   matrix memory        a = keep, g = take (jv_memory_gates), and one more column whose value is 1 (the normaliser)
//
// Token by token (recurrent.cu) every state element costs three multiply-adds a token.  With S_0 the state before a chunk
// and L_t = log a_1 + .. + log a_t inside it,
//
//     S_T = exp(L_T) S_0 + D,   D = sum_s k_s (g_s exp(L_T - L_s) v_s)^T                                             (1)
//     o_t = exp(L_t) S_0^T q_t + sum_{s <= t} (q_t . k_s) g_s exp(L_t - L_s) v_s                                     (2)
//
// D hangs on the chunk's own tokens alone, so three kernels do it, and only the middle one, which does next to nothing, goes
// through the tokens in order:
//   chunk_delta_kernel    D of every (chunk, head), all at once
//   chunk_start_kernel    S_0 of every chunk from the one before it, in D's place; the state after the last
//   chunk_output_kernel   the outputs of every (chunk, head), all at once
//
// q, k and v are 16-bit numbers, the operands on the other side are 32-bit: S_0, the weighted scores and the weighted values.
// A 32-bit number is cut into three 16-bit ones (x = hi + mid + lo, eight bits of mantissa each, exactly), so that the three
// products with a 16-bit number are exact and only the sums round.  The tensor core's sums cut where the CUDA cores' round: a sum of
// 16 products starts from zero there (smallest parts first) and is added to the running one on the CUDA cores (one running sum
// in the tensor core: 3.4e-7 relative for 128 channels, this way 0.8e-7, as token by token).  L is summed in 64-bit and kept as two
// floats: L_t - L_s keeps its digits behind a large decay.  The normaliser's sums are made on the CUDA cores.
//
// What bounds it: the two kernels on the tensor cores, their rate of mma.sync (one a 2.2 clocks and multiprocessor at best; 4.8 and 5.7
// here), the middle one its bytes.  4,096 tokens in three entries, 128 heads of 128 x 64: 115, 55 and 259 us; chunks of 32 that a
// block went through in order took 620.  2,048 tokens of 8 heads of 128 x 256 with a normaliser: 19, 9 and 39, where a scan token by token
// in segments took 276; 2,000 tokens of 8 heads of 256 x 512: 58, 18 and 150 (888).  1,200 tokens of 64 heads of 128 x 64: 81 (172).
#include "scan.cuh"
#include <math.h>

namespace {
constexpr int CT = 128;                    // tokens of a chunk
constexpr int VT = 64, LV = VT + 8;        // value columns of a block, padded row (no bank is met twice)
using bf16 = __nv_bfloat16;

struct ChunkParams {
  const bf16 *q, *k, *v;                   // rows of the tokens; the columns of head 0 (group 0)
  long long q_stride, k_stride, v_stride;
  int per_group;                           // heads that share a q and k
  float scale;
  const float* gates;                      // [n, heads, 4] = (keep, take, -, n . q); null: the step sizes below
  const bf16* dt_raw; long long dt_stride;
  const void *dt_bias, *a_log; int w_dtype;
  float* out;                              // [n, heads * V]
  float* state; long long slot_stride;     // S of (slot, head) at state + slot * slot_stride + head * D * V
  float* state_n;                          // the normaliser's state [slots][heads * D], rows slot_stride apart (or null)
  float* nq;                               // its outputs, every fourth float (the gates' last place)
  int h0;                                  // a launch takes as many heads from here on as its grid has rows, the scratch's [heads]
  float* starts;                           // [chunks][heads][D][V]: D of a chunk, then S_0
  float* starts_n;                         // [chunks][heads][D]: the same of the normaliser
  float* whole;                            // [chunks][heads]: exp(L_T)
  const int *cu_seqlens, *slots;
  int n_slots, heads, D, V;
  int portions, n_entries, max_chunks;     // portions > 0: entries of one token are passed by, so many others taken
  int* status;
};

// f = a b + (FIRST ? 0 : f)
template <bool FIRST> __device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if (FIRST)
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
  else
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void add(float (&c)[4], const float (&f)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] += f[i];
}
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], const bf16* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm_t(uint32_t (&r)[4], const bf16* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}

// Two 32-bit numbers as three pairs of 16-bit ones whose sum they are: the leading eight bits of the mantissa, the next
// eight, the rest (what is left over fits eight bits, so every step is exact).
__device__ __forceinline__ void cut3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const uint32_t xb = __float_as_uint(x), yb = __float_as_uint(y);
  hi = __byte_perm(xb, yb, 0x7632);
  const float xr = x - __uint_as_float(xb & 0xffff0000u), yr = y - __uint_as_float(yb & 0xffff0000u);
  const uint32_t xm = __float_as_uint(xr), ym = __float_as_uint(yr);
  mid = __byte_perm(xm, ym, 0x7632);
  const float xl = xr - __uint_as_float(xm & 0xffff0000u), yl = yr - __uint_as_float(ym & 0xffff0000u);
  lo = __byte_perm(__float_as_uint(xl), __float_as_uint(yl), 0x7632);
}

// The chunk that a block works on.
struct Chunk {
  int entry, index, t0, here;              // its number in the entry, its first token, how many tokens it has
};
__device__ __forceinline__ bool find_chunk(const ChunkParams& p, int number, Chunk& c) {
  int n_seg;
  if (!find_segment(p.cu_seqlens, p.n_entries, CT, p.portions, number, c.entry, c.index, n_seg)) return false;
  c.t0 = p.cu_seqlens[c.entry] + c.index * CT;
  c.here = min(CT, p.cu_seqlens[c.entry + 1] - c.t0);
  return c.here > 0;
}

// What a chunk's tokens weigh.
struct alignas(16) Weights {
  float2 L[CT];                              // L_t as a leading and a following number
  float g[CT], from_start[CT], to_end[CT];   // g_s, exp(L_t), g_s exp(L_T - L_s)
  float whole;                               // exp(L_T)
  double part[CT / 32];
};

// By threads 0 .. CT - 1 of the block, a token each; all threads of the block call it.
__device__ __forceinline__ void make_weights(Weights& w, const ChunkParams& p, const Chunk& c, int h) {
  const int s = threadIdx.x, lane = s & 31;
  const bool there = s < c.here;
  float g = 0.f;
  double L = 0.0;
  if (s < CT) {
    const size_t t = c.t0 + min(s, c.here - 1);
    float log_a;
    if (p.gates != nullptr) {
      const float2 both = *reinterpret_cast<const float2*>(p.gates + (t * p.heads + h) * 4);
      g = both.y;
      log_a = logf(both.x);
    } else {
      const float rate = expf(p.w_dtype == 0 ? ((const float*)p.a_log)[h] : to_f32(((const bf16*)p.a_log)[h]));
      const float bias = p.w_dtype == 0 ? ((const float*)p.dt_bias)[h] : to_f32(((const bf16*)p.dt_bias)[h]);
      const float z = to_f32(p.dt_raw[t * p.dt_stride + h]) + bias;
      g = fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)));     // softplus, no clamp
      log_a = -rate * g;
    }
    // below -1e4 a decay is zero in any case, and a sum of them stays a number
    L = there ? (double)(log_a < -1e4f ? -1e4f : log_a) : 0.0;
    if (!there) g = 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double before = __shfl_up_sync(0xffffffffu, L, o);
      if (lane >= o) L += before;
    }
    if (lane == 31) w.part[s >> 5] = L;
  }
  __syncthreads();
  if (s < CT) {
    double end = 0.0;
#pragma unroll
    for (int i = 0; i < CT / 32; ++i) {
      if (i < (s >> 5)) L += w.part[i];
      end += w.part[i];
    }
    w.L[s] = make_float2((float)L, (float)(L - (double)(float)L));
    w.g[s] = g;
    w.from_start[s] = expf((float)L);
    w.to_end[s] = there ? g * expf((float)(end - L)) : 0.f;
    if (s == 0) w.whole = expf((float)end);
  }
}

__device__ __forceinline__ void copy_16(bf16* dst, const bf16* src, bool live) {
  const int n = live ? 16 : 0;                         // 0: zeros are written and nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(n) : "memory");
}
// CT rows of up to `width` elements (zeros past them, and past the tokens that are there) into rows of LD, W of them used.
template <int W, int LD, int THREADS>
__device__ __forceinline__ void copy_rows(bf16* dst, const bf16* src, long long stride, int here, int width) {
  constexpr int PER = W / 8;
  for (int i = threadIdx.x; i < CT * PER; i += THREADS) {
    const int t = i / PER, e = (i - t * PER) * 8;
    const bool live = t < here && e < width;
    copy_16(dst + t * LD + e, src + (live ? t * stride + e : 0), live);
  }
}

// A value that is no number is taken out of the tile and remembered, `bad` [VT] being the first token of a column with one (CT:
// none): the zeros of scores that look ahead would carry it into earlier outputs.
template <int THREADS> __device__ __forceinline__ void take_out(bf16* x, int* bad) {
  for (int i = threadIdx.x; i < CT * (VT / 8); i += THREADS) {
    const int t = i / (VT / 8), e = (i - t * (VT / 8)) * 8;
    const uint4 v = *reinterpret_cast<const uint4*>(x + t * LV + e);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    bool no_number = false;
#pragma unroll
    for (int j = 0; j < 4; ++j) no_number |= (w[j] & 0x7f80u) == 0x7f80u || (w[j] & 0x7f800000u) == 0x7f800000u;
    if (no_number) {
      unsigned short* at = reinterpret_cast<unsigned short*>(x + t * LV + e);
      for (int j = 0; j < 8; ++j)
        if ((at[j] & 0x7f80u) == 0x7f80u) { atomicMin(bad + e + j, t); at[j] = 0; }
    }
  }
}

// ------------------------------------------------------------------------------------------- D of every chunk
constexpr int DELTA_THREADS = 128;         // a warp 16 of the block's value columns

template <int DP> struct DeltaShape {
  static constexpr int DS = DP < 128 ? DP : 128, LD = DS + 8;          // key channels of a block
  static constexpr int SMEM = (CT * LD + CT * LV) * 2 + (int)sizeof(Weights) + VT * 4;
};

template <int DP>
__global__ void __launch_bounds__(DELTA_THREADS) chunk_delta_kernel(const ChunkParams p) {
  using Shape = DeltaShape<DP>;
  constexpr int DS = Shape::DS, LD = Shape::LD, MT = DS / 16;
  extern __shared__ __align__(16) unsigned char raw[];
  Weights& w = *reinterpret_cast<Weights*>(raw);
  bf16* ks = reinterpret_cast<bf16*>(raw + sizeof(Weights));           // [CT][LD]
  bf16* xs = ks + CT * LD;                                              // [CT][LV]
  int* bad = reinterpret_cast<int*>(xs + CT * LV);
  pdl_trigger();
  pdl_wait();
  Chunk c;
  if (!find_chunk(p, blockIdx.x, c)) return;
  const int h = p.h0 + blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gr = lane >> 2, gq = lane & 3, lr = lane & 7, lm = lane >> 3;
  const int d_parts = (p.D + DS - 1) / DS, d0 = blockIdx.z % d_parts * DS, e0 = blockIdx.z / d_parts * VT;
  if (tid < VT) bad[tid] = CT;
  copy_rows<DS, LD, DELTA_THREADS>(ks, p.k + c.t0 * p.k_stride + (h / p.per_group) * p.D + d0, p.k_stride, c.here, p.D - d0);
  copy_rows<VT, LV, DELTA_THREADS>(xs, p.v + c.t0 * p.v_stride + (size_t)h * p.V + e0, p.v_stride, c.here, p.V - e0);
  cp_async_commit();
  make_weights(w, p, c, h);
  cp_async_wait_all();
  __syncthreads();
  take_out<DELTA_THREADS>(xs, bad);
  __syncthreads();
  const size_t at = (size_t)blockIdx.x * gridDim.y + blockIdx.y;
  float acc[MT][2][4];
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
  const int tiles = (c.here + 15) / 16;
  if (e0 + warp * 16 < p.V) {
#pragma unroll 1
    for (int kk = 0; kk < tiles; ++kk) {
      uint32_t raw_b[4], b[2][3][2];
      ldsm_t(raw_b, xs + (kk * 16 + lr + (lm & 1) * 8) * LV + warp * 16 + (lm >> 1) * 8);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const float2 f = *reinterpret_cast<const float2*>(&w.to_end[kk * 16 + u * 8 + gq * 2]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t x = raw_b[2 * j + u];
          cut3(__uint_as_float(x << 16) * f.x, __uint_as_float(x & 0xffff0000u) * f.y, b[j][0][u], b[j][1][u], b[j][2][u]);
        }
      }
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        uint32_t a[4];
        ldsm_t(a, ks + (kk * 16 + lr + (lm >> 1) * 8) * LD + i * 16 + (lm & 1) * 8);
        float f[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j) mma<true>(f[j], a, b[j][2][0], b[j][2][1]);
#pragma unroll
        for (int j = 0; j < 2; ++j) mma<false>(f[j], a, b[j][1][0], b[j][1][1]);
#pragma unroll
        for (int j = 0; j < 2; ++j) mma<false>(f[j], a, b[j][0][0], b[j][0][1]);
#pragma unroll
        for (int j = 0; j < 2; ++j) add(acc[i][j], f[j]);
      }
    }
    float* dst = p.starts + at * p.D * p.V;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int lc = warp * 16 + j * 8 + gq * 2, e = e0 + lc;
      if (e >= p.V) continue;                          // V is a multiple of 8: the pair is there or not
      const bool bad0 = bad[lc] < CT, bad1 = bad[lc + 1] < CT;
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int d = d0 + i * 16 + gr + r * 8;
          if (d < p.D)
            *reinterpret_cast<float2*>(dst + (size_t)d * p.V + e) = make_float2(bad0 ? NAN : acc[i][j][2 * r], bad1 ? NAN : acc[i][j][2 * r + 1]);
        }
    }
  }
  if (e0 == 0) {
    if (d0 == 0 && tid == 0) p.whole[at] = w.whole;
    if (p.state_n != nullptr) {
      for (int d = tid; d < DS && d0 + d < p.D; d += DELTA_THREADS) {
        float n = 0.f;
        for (int s = 0; s < c.here; ++s) n = fmaf(to_f32(ks[s * LD + d]), w.to_end[s], n);
        p.starts_n[at * p.D + d0 + d] = n;
      }
    }
  }
}

// ------------------------------------------------------------------------------- the state before every chunk
constexpr int START_THREADS = 128, START_AHEAD = 4;

// A thread four elements of a head's state (and normaliser); START_AHEAD chunks are asked for at a time.
__global__ void __launch_bounds__(START_THREADS) chunk_start_kernel(const ChunkParams p) {
  pdl_trigger();
  pdl_wait();
  const int entry = entry_of(blockIdx.z, p.portions, p.cu_seqlens, p.n_entries);
  if (entry < 0) return;
  const int h = p.h0 + blockIdx.y, matrix = p.D * p.V / 4, i = blockIdx.x * START_THREADS + threadIdx.x;
  const bool normaliser = i >= matrix;
  if (i >= matrix + (p.state_n != nullptr ? p.D / 4 : 0)) return;
  const int len = p.cu_seqlens[entry + 1] - p.cu_seqlens[entry];
  if (len <= 0) return;
  const int slot = p.slots[entry];
  int g0 = 0;                                          // the number of the entry's first chunk
  for (int e = 0; e < entry; ++e) g0 += segments_of(p.cu_seqlens[e + 1] - p.cu_seqlens[e], CT, p.portions);
  const int chunks = (len + CT - 1) / CT;
  if (slot < 0 || slot >= p.n_slots || g0 + chunks > p.max_chunks) {       // (more portions than were said to be there)
    if (i == 0) atomicOr(p.status, JV_STATUS_BAD_ROW);
    return;
  }
  const int size = normaliser ? p.D : p.D * p.V, e = 4 * (normaliser ? i - matrix : i);
  float* state = (normaliser ? p.state_n : p.state) + (size_t)slot * p.slot_stride + (size_t)h * size + e;
  float* at = (normaliser ? p.starts_n : p.starts) + ((size_t)g0 * gridDim.y + blockIdx.y) * size + e;
  const float* whole = p.whole + (size_t)g0 * gridDim.y + blockIdx.y;
  const size_t step = (size_t)gridDim.y * size;
  float4 S = make_float4(state[0], state[1], state[2], state[3]);
  for (int c0 = 0; c0 < chunks; c0 += START_AHEAD) {
    float4 d[START_AHEAD];
    float a[START_AHEAD];
#pragma unroll
    for (int j = 0; j < START_AHEAD; ++j) {
      const int c = min(c0 + j, chunks - 1);
      d[j] = *reinterpret_cast<const float4*>(at + c * step);
      a[j] = whole[(size_t)c * gridDim.y];
    }
#pragma unroll
    for (int j = 0; j < START_AHEAD; ++j) {
      if (c0 + j >= chunks) break;
      *reinterpret_cast<float4*>(at + (c0 + j) * step) = S;
      S.x = fmaf(a[j], S.x, d[j].x); S.y = fmaf(a[j], S.y, d[j].y); S.z = fmaf(a[j], S.z, d[j].z); S.w = fmaf(a[j], S.w, d[j].w);
    }
  }
  state[0] = S.x; state[1] = S.y; state[2] = S.z; state[3] = S.w;
}

// ------------------------------------------------------------------------------------- the outputs of every chunk
constexpr int OUT_THREADS = 256;           // a warp 16 of the chunk's tokens

template <int DP> struct OutShape {
  static constexpr int LD = DP + 8, DB = DP / 2;       // S_0 passes by in two blocks of channels
  static constexpr bool KEEP = DP <= 128;              // a warp's queries stay in registers, and S_0 passes by where they lay
  static constexpr int ROWS = 2 * CT * LD + CT * LV + (KEEP ? 0 : 3 * DB * LV);
  static constexpr int SMEM = ROWS * 2 + (int)sizeof(Weights) + VT * 4;
  static_assert(!KEEP || 3 * DB * LV <= CT * LD, "a block of S_0 in three parts has to fit q's place");
};

template <int DP>
__global__ void __launch_bounds__(OUT_THREADS, DP <= 128 ? 2 : 1) chunk_output_kernel(const ChunkParams p) {
  using Shape = OutShape<DP>;
  constexpr int LD = Shape::LD, DB = Shape::DB, KT = DP / 16;
  constexpr bool KEEP = Shape::KEEP;
  extern __shared__ __align__(16) unsigned char raw[];
  Weights& w = *reinterpret_cast<Weights*>(raw);
  bf16* qs = reinterpret_cast<bf16*>(raw + sizeof(Weights));           // [CT][LD]
  bf16* ks = qs + CT * LD;                                              // [CT][LD]
  bf16* xs = ks + CT * LD;                                              // [CT][LV]
  bf16* ss = KEEP ? qs : xs + CT * LV;                                  // [3][DB][LV]: a block of S_0
  int* bad = reinterpret_cast<int*>(qs + Shape::ROWS);
  pdl_trigger();
  pdl_wait();
  Chunk c;
  if (!find_chunk(p, blockIdx.x, c)) return;
  const int h = p.h0 + blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gr = lane >> 2, gq = lane & 3, lr = lane & 7, lm = lane >> 3;
  const int e0 = blockIdx.z * VT;
  const size_t at = (size_t)blockIdx.x * gridDim.y + blockIdx.y;
  if (tid < VT) bad[tid] = CT;
  copy_rows<DP, LD, OUT_THREADS>(qs, p.q + c.t0 * p.q_stride + (h / p.per_group) * p.D, p.q_stride, c.here, p.D);
  copy_rows<DP, LD, OUT_THREADS>(ks, p.k + c.t0 * p.k_stride + (h / p.per_group) * p.D, p.k_stride, c.here, p.D);
  copy_rows<VT, LV, OUT_THREADS>(xs, p.v + c.t0 * p.v_stride + (size_t)h * p.V + e0, p.v_stride, c.here, p.V - e0);
  cp_async_commit();
  // a block of S_0: this thread's fours of columns, asked for long before they are used
  constexpr int PER = DB * (VT / 4) / OUT_THREADS > 0 ? DB * (VT / 4) / OUT_THREADS : 1;
  float4 s0[PER];
  auto fetch = [&](int first) {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int j = tid + i * OUT_THREADS, d = first + j / (VT / 4), e = e0 + j % (VT / 4) * 4;
      s0[i] = d < p.D && e < p.V && j < DB * (VT / 4) ? *reinterpret_cast<const float4*>(p.starts + (at * p.D + d) * p.V + e)
                                                       : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  fetch(0);
  make_weights(w, p, c, h);
  cp_async_wait_all();
  __syncthreads();
  take_out<OUT_THREADS>(xs, bad);
  __syncthreads();
  // the warps that share a scheduler take a tile with few earlier tokens and one with many
  const int tm = (warp < 4 ? warp : 11 - warp) * 16, ta = tm + gr, tb = ta + 8;
  const bool at_work = tm < c.here;
  float O[8][4], sum_a = 0.f, sum_b = 0.f;
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) O[j][e] = 0.f;
  const float fa = w.from_start[ta], fb = w.from_start[tb];
  uint32_t qa[KEEP ? KT : 1][4];
  if (KEEP) {
#pragma unroll
    for (int kk = 0; kk < KT; ++kk) ldsm(qa[KEEP ? kk : 0], qs + (tm + lr + (lm & 1) * 8) * LD + kk * 16 + (lm >> 1) * 8);
  }
  const bool counts = p.state_n != nullptr && e0 == 0 && at_work;
  if (counts) {
    // the normaliser: q . n_0 here, the sums of the weighted scores further down
    float na = 0.f, nb = 0.f;
    const float* n0 = p.starts_n + at * p.D;
    for (int d = gq * 2; d < p.D; d += 8) {
      const float2 n = *reinterpret_cast<const float2*>(n0 + d);
      const uint32_t a = *reinterpret_cast<const uint32_t*>(qs + ta * LD + d), b = *reinterpret_cast<const uint32_t*>(qs + tb * LD + d);
      na = fmaf(__uint_as_float(a << 16), n.x, fmaf(__uint_as_float(a & 0xffff0000u), n.y, na));
      nb = fmaf(__uint_as_float(b << 16), n.x, fmaf(__uint_as_float(b & 0xffff0000u), n.y, nb));
    }
    sum_a = fa * na;
    sum_b = fb * nb;
  }
  // What the state before the chunk gives: exp(L_t) q S_0.  First, since all warps have as much of it: behind what the chunk's own tokens
  // give, of which the last warp has eight times the first one's, its barriers made every warp wait for the last (286 us where this order takes 259).
#pragma unroll (KEEP ? 2 : 1)
  for (int first = 0; first < DP; first += DB) {
    if (first >= p.D) break;
    if (KEEP || first > 0) __syncthreads();            // the queries (or the block before) have been read
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int j = tid + i * OUT_THREADS, d = j / (VT / 4), e = j % (VT / 4) * 4;
      if (j < DB * (VT / 4)) {
        uint2 part[3];
        cut3(s0[i].x, s0[i].y, part[0].x, part[1].x, part[2].x);
        cut3(s0[i].z, s0[i].w, part[0].y, part[1].y, part[2].y);
#pragma unroll
        for (int z = 0; z < 3; ++z) *reinterpret_cast<uint2*>(ss + (z * DB + d) * LV + e) = part[z];
      }
    }
    if (first + DB < p.D) fetch(first + DB);
    __syncthreads();
    if (at_work) {
#pragma unroll
      for (int kk = 0; kk < DB / 16; ++kk) {
        uint32_t a[4];
        if (KEEP) {
#pragma unroll
          for (int i = 0; i < 4; ++i) a[i] = qa[KEEP ? first / 16 + kk : 0][i];
        } else {
          ldsm(a, qs + (tm + lr + (lm & 1) * 8) * LD + first + kk * 16 + (lm >> 1) * 8);
        }
#pragma unroll
        for (int j = 0; j < 8; j += 4) {
          float f[4][4];
#pragma unroll
          for (int z = 2; z >= 0; --z) {
            uint32_t b[2][4];
#pragma unroll
            for (int v = 0; v < 2; ++v) ldsm_t(b[v], ss + (z * DB + kk * 16 + lr + (lm & 1) * 8) * LV + (j + 2 * v) * 8 + (lm >> 1) * 8);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              if (z == 2) mma<true>(f[u], a, b[u >> 1][2 * (u & 1)], b[u >> 1][2 * (u & 1) + 1]);
              else mma<false>(f[u], a, b[u >> 1][2 * (u & 1)], b[u >> 1][2 * (u & 1) + 1]);
            }
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) add(O[j + u], f[u]);
        }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) { O[j][0] *= fa; O[j][1] *= fa; O[j][2] *= fb; O[j][3] *= fb; }
  if (!at_work) return;
  // what the chunk's own tokens give
  {
    const float2 La = w.L[ta], Lb = w.L[tb];
#pragma unroll 1
    for (int sn = 0; sn <= tm; sn += 16) {
      float G[2][4] = {};
#pragma unroll
      for (int kk = 0; kk < KT; ++kk) {
        uint32_t b[4];
        if (!KEEP) ldsm(qa[0], qs + (tm + lr + (lm & 1) * 8) * LD + kk * 16 + (lm >> 1) * 8);
        ldsm(b, ks + (sn + lr + (lm >> 1) * 8) * LD + kk * 16 + (lm & 1) * 8);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float f[4];
          mma<true>(f, qa[KEEP ? kk : 0], b[2 * j], b[2 * j + 1]);
          add(G[j], f);
        }
      }
      uint32_t m[3][4];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int s = sn + j * 8 + gq * 2;
        const float4 l = *reinterpret_cast<const float4*>(&w.L[s]);
        const float2 g = *reinterpret_cast<const float2*>(&w.g[s]);
        const float a0 = s <= ta ? G[j][0] * (g.x * expf((La.x - l.x) + (La.y - l.y))) : 0.f;
        const float a1 = s + 1 <= ta ? G[j][1] * (g.y * expf((La.x - l.z) + (La.y - l.w))) : 0.f;
        const float b0 = s <= tb ? G[j][2] * (g.x * expf((Lb.x - l.x) + (Lb.y - l.y))) : 0.f;
        const float b1 = s + 1 <= tb ? G[j][3] * (g.y * expf((Lb.x - l.z) + (Lb.y - l.w))) : 0.f;
        sum_a += a0 + a1;
        sum_b += b0 + b1;
        cut3(a0, a1, m[0][2 * j], m[1][2 * j], m[2][2 * j]);
        cut3(b0, b1, m[0][2 * j + 1], m[1][2 * j + 1], m[2][2 * j + 1]);
      }
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        uint32_t b[2][4];
#pragma unroll
        for (int v = 0; v < 2; ++v) ldsm_t(b[v], xs + (sn + lr + (lm & 1) * 8) * LV + (j + 2 * v) * 8 + (lm >> 1) * 8);
        float f[4][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) mma<true>(f[u], m[2], b[u >> 1][2 * (u & 1)], b[u >> 1][2 * (u & 1) + 1]);
#pragma unroll
        for (int u = 0; u < 4; ++u) mma<false>(f[u], m[1], b[u >> 1][2 * (u & 1)], b[u >> 1][2 * (u & 1) + 1]);
#pragma unroll
        for (int u = 0; u < 4; ++u) mma<false>(f[u], m[0], b[u >> 1][2 * (u & 1)], b[u >> 1][2 * (u & 1) + 1]);
#pragma unroll
        for (int u = 0; u < 4; ++u) add(O[j + u], f[u]);
      }
    }
  }
  if (counts) {
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      sum_a += __shfl_xor_sync(0xffffffffu, sum_a, o);
      sum_b += __shfl_xor_sync(0xffffffffu, sum_b, o);
    }
    if (gq == 0) {
      if (ta < c.here) p.nq[((size_t)(c.t0 + ta) * p.heads + h) * 4] = sum_a * p.scale;
      if (tb < c.here) p.nq[((size_t)(c.t0 + tb) * p.heads + h) * 4] = sum_b * p.scale;
    }
  }
  const size_t orow = (size_t)p.heads * p.V;
  float* o = p.out + (size_t)c.t0 * orow + (size_t)h * p.V + e0;
  const bool pairs = ((uintptr_t)o & 7) == 0;          // a caller's result may start on any number
  auto put = [&](float* dst, float x, float y) {
    if (pairs) {
      *reinterpret_cast<float2*>(dst) = make_float2(x, y);
    } else {
      dst[0] = x;
      dst[1] = y;
    }
  };
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int lc = j * 8 + gq * 2;
    if (e0 + lc >= p.V) continue;
    const int bad0 = bad[lc], bad1 = bad[lc + 1];
    if (ta < c.here) put(o + ta * orow + lc, bad0 <= ta ? NAN : O[j][0] * p.scale, bad1 <= ta ? NAN : O[j][1] * p.scale);
    if (tb < c.here) put(o + tb * orow + lc, bad0 <= tb ? NAN : O[j][2] * p.scale, bad1 <= tb ? NAN : O[j][3] * p.scale);
  }
}

template <int DP>
int launch(ChunkParams p, int entries, int at_once, cudaStream_t stream) {
  static bool done[JV_MAX_DEVICES] = {};
  if (!jv_once_per_device(done, [&] {
        return cudaFuncSetAttribute(chunk_delta_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, DeltaShape<DP>::SMEM) == cudaSuccess &&
               cudaFuncSetAttribute(chunk_output_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, OutShape<DP>::SMEM) == cudaSuccess;
      }))
    return JV_ERR_UNSUPPORTED;
  const int v_parts = (p.V + VT - 1) / VT, d_parts = (p.D + DeltaShape<DP>::DS - 1) / DeltaShape<DP>::DS;
  const int fours = p.D * p.V / 4 + (p.state_n != nullptr ? p.D / 4 : 0);
  if (v_parts * d_parts > 65535 || entries > 65535) return JV_ERR_UNSUPPORTED;
  for (p.h0 = 0; p.h0 < p.heads; p.h0 += at_once) {
    const int heads = p.heads - p.h0 < at_once ? p.heads - p.h0 : at_once;
    int rc = jv_launch(chunk_delta_kernel<DP>, dim3(p.max_chunks, heads, v_parts * d_parts), dim3(DELTA_THREADS), DeltaShape<DP>::SMEM, stream, p);
    if (rc != JV_OK) return rc;
    rc = jv_launch(chunk_start_kernel, dim3((fours + START_THREADS - 1) / START_THREADS, heads, entries), dim3(START_THREADS), 0, stream, p);
    if (rc != JV_OK) return rc;
    rc = jv_launch(chunk_output_kernel<DP>, dim3(p.max_chunks, heads, v_parts), dim3(OUT_THREADS), OutShape<DP>::SMEM, stream, p);
    if (rc != JV_OK) return rc;
  }
  return JV_OK;
}

bool rows_of_16_bytes(const void* p, long long stride) { return ((uintptr_t)p & 15) == 0 && stride % 8 == 0; }
}  // namespace

// q, k, v: the first head's columns in rows of `.._stride` 16-bit elements (head h reads q and k at (h / per_group) * D, v at h * V);
// gates [n, heads, 4] float with nq = gates + 3 and state_n, or null with dt_raw (rows of dt_stride elements, [heads] used),
// dt_bias, a_log [heads] of w_dtype; out [n, heads * V]; state as for jv_state_scan; portions > 0: entries of one token
// are passed by, which leaves this many, with n tokens; scratch: (n / 128 + portions) * at_once * (D * V + D + 1)
// floats, 16-byte aligned, for at_once heads, which are gone through so many at a time.  Taken for D up to 256
// and V, both in steps of 8, with rows on 16-byte boundaries.
JV_EXPORT int jv_chunk_scan(const void* q, long long q_stride, const void* k, long long k_stride, const void* v, long long v_stride,
                            int per_group, float scale, float* gates, const void* dt_raw, long long dt_stride, const void* dt_bias,
                            const void* a_log, int w_dtype, float* out, float* state, long long slot_stride, float* state_n,
                            const int* cu_seqlens, const int* slots, int n_slots, int entries, int heads, int D, int V, int portions,
                            int n, float* scratch, int at_once, int* status, cudaStream_t stream) {
  if (entries == 0 || n == 0) return JV_OK;
  if (D < 8 || D > 256 || D % 8 || V < 8 || V % 8 || per_group < 1 || heads % per_group || heads > 65535 || entries < 0 || n < 0 ||
      !rows_of_16_bytes(q, q_stride) || !rows_of_16_bytes(k, k_stride) || !rows_of_16_bytes(v, v_stride) || w_dtype < 0 || w_dtype > 1 || at_once < 1 ||
      (gates == nullptr && (dt_raw == nullptr || state_n != nullptr)) || ((uintptr_t)gates & 7) || ((uintptr_t)scratch & 15))
    return JV_ERR_UNSUPPORTED;
  if (at_once > heads) at_once = heads;
  const int taken = portions > 0 ? portions : entries, max_chunks = n / CT + taken;
  float* starts_n = scratch + (size_t)max_chunks * at_once * D * V;
  ChunkParams p{(const bf16*)q, (const bf16*)k, (const bf16*)v, q_stride, k_stride, v_stride, per_group, scale, gates,
                (const bf16*)dt_raw, dt_stride, dt_bias, a_log, w_dtype, out, state, slot_stride, state_n,
                gates == nullptr ? nullptr : gates + 3, 0, scratch, starts_n, starts_n + (size_t)max_chunks * at_once * D,
                cu_seqlens, slots, n_slots, heads, D, V, portions, entries, max_chunks, status};
  if (D <= 32) return launch<32>(p, taken, at_once, stream);
  if (D <= 64) return launch<64>(p, taken, at_once, stream);
  if (D <= 128) return launch<128>(p, taken, at_once, stream);
  return launch<256>(p, taken, at_once, stream);
}
