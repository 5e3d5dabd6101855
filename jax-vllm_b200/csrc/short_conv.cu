// A short causal convolution over time on each channel, with the last taps - 1 inputs of every sequence kept as
// state, so that a sequence may be cut into steps anywhere:
//
//   conv_t[c] = sum_j w[c, j] * in_(t - taps + 1 + j)[c]        (the last column weighs the current token; inputs
//                                                                before the sequence's start are zero)
//   out_t[c]  = act(conv_t[c] + bias[c])            act: none or silu
//           or  in_t[c] + conv_t[c]                 `residual`: the convolution is added to what it reads
//
// state[slot, j, c], j < taps - 1, holds the input at the sequence's position (tokens so far) - (taps - 1) + j; a
// fresh slot is zero, which is the zero padding.  All arithmetic is 32-bit, whatever the types of in and out.
//
// A thread owns one channel of one segment of 8 to 32 tokens of one entry and slides a window of taps - 1 registers over
// it (segments are at least taps - 1 long).  Segments are counted per entry, so only an entry's first segment reads the state; the thread of that segment
// is also the ONE writer of the entry's state for its channel: it has the old state in its window before it writes
// the new one (the entry's last taps - 1 inputs, or old state shifted where the entry is shorter), so no other
// thread reads what it overwrites.  Blocks find their (entry, segment) from cu_seqlens; the grid is an upper bound,
// n / (tokens of a segment) + entries, and blocks beyond the last segment leave.
#include "common.cuh"

namespace {
constexpr int THREADS = 128;
constexpr int BATCH = 8;       // inputs a thread asks for before it uses the first

struct ConvParams {
  const void* in; long long in_stride;
  void* out; long long out_stride;
  const void* w; const void* bias;
  float* state; long long state_stride;      // elements between slots
  const int* cu_seqlens; const int* slots;
  int n_entries, n_slots, channels, act, residual;
  int seg_log2;                              // tokens of a segment (a shift: every block goes through the entries)
  int* status;
};

// y <- y * sigmoid(y) = y / d, d = 1 + exp(-y).  The dozen instructions of a division were what a long portion waited for, so results that
// are rounded to 16 bits right away are first formed with 1 / d to 2^-23, which leaves them within four units in the last place of the
// quotient, rounded to 32 bits.  Both round to the same 16-bit number unless a boundary of that rounding (a lower half of 0x8000) is as near;
// where it is within eight, one result in 4,000, or d so large that 1 / d is no normal number, the four of a thread are divided, so that
// every kernel gives the quotient, rounded.  (4,096 tokens of 10,240 channels: 77 us with the division throughout, 44.4 with the reciprocal
// alone, 54.8 so.)
template <typename TO, int N> __device__ __forceinline__ void silu(float (&y)[N]) {
  if constexpr (sizeof(TO) == 2) {
    float q[N], least = y[0];
    uint32_t nearest = 0xffffffffu;                    // two at a time: how far a lower half lies above eight units below the boundary
#pragma unroll
    for (int e = 0; e < N; ++e) {
      float r;
      asm("rcp.approx.ftz.f32 %0, %1;\n" : "=f"(r) : "f"(1.f + expf(-y[e])));
      q[e] = y[e] * r;
      least = fminf(least, y[e]);
    }
    // (a borrow of the first moves the second by one unit, which the eight leave room for)
#pragma unroll
    for (int e = 0; e < N; e += 2)
      nearest = __vminu2(nearest, __byte_perm(__float_as_uint(q[e]), __float_as_uint(q[e + 1 < N ? e + 1 : e]), 0x5410) - 0x7ff87ff8u);
    if ((nearest & 0xffffu) > 16 && nearest >> 16 > 16 && least > -80.f) {
#pragma unroll
      for (int e = 0; e < N; ++e) y[e] = q[e];
      return;
    }
  }
#pragma unroll
  for (int e = 0; e < N; ++e) y[e] = y[e] / (1.f + expf(-y[e]));
}

template <typename TI, typename TO, typename TW, int TAPS>
__global__ void __launch_bounds__(THREADS) short_conv_kernel(const ConvParams p) {
  pdl_trigger();
  pdl_wait();
  // which segment of which entry
  int entry = -1, seg = 0, before = 0;
  for (int e = 0; e < p.n_entries; ++e) {
    const int q = p.cu_seqlens[e + 1] - p.cu_seqlens[e];
    const int segs = (q + (1 << p.seg_log2) - 1) >> p.seg_log2;
    if ((int)blockIdx.x < before + segs) { entry = e; seg = blockIdx.x - before; break; }
    before += segs;
  }
  if (entry < 0) return;
  const int c = blockIdx.y * THREADS + threadIdx.x;
  if (c >= p.channels) return;
  const int t_begin = p.cu_seqlens[entry], q = p.cu_seqlens[entry + 1] - t_begin;
  const int i0 = seg << p.seg_log2, i1 = min(q, i0 + (1 << p.seg_log2));
  constexpr int K = TAPS - 1;
  const int slot = K > 0 ? p.slots[entry] : 0;        // one tap keeps nothing
  if (K > 0 && (slot < 0 || slot >= p.n_slots)) {
    if (threadIdx.x == 0) atomicOr(p.status, JV_STATUS_BAD_ROW);
    return;
  }
  const TI* in = (const TI*)p.in + c;
  TO* out = (TO*)p.out + c;
  float* st = K > 0 ? p.state + (size_t)slot * p.state_stride + c : nullptr;
  float wt[TAPS];
#pragma unroll
  for (int j = 0; j < TAPS; ++j) wt[j] = to_f32(((const TW*)p.w)[(size_t)c * TAPS + j]);
  const float b = p.bias != nullptr ? to_f32(((const TW*)p.bias)[c]) : 0.f;
  float win[K > 0 ? K : 1];          // win[k]: the input at offset i0 - K + k of the entry
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = i0 - K + k;
    win[k] = i >= 0 ? to_f32(in[(size_t)(t_begin + i) * p.in_stride]) : st[(size_t)(K + i) * p.channels];
  }
  if (seg == 0) {
    // the state after this step: the last K inputs of (old state, this entry's tokens)
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int i = q - K + j;
      float v;
      if (i >= 0) {
        v = to_f32(in[(size_t)(t_begin + i) * p.in_stride]);
      } else {
        v = 0.f;
#pragma unroll
        for (int k = 0; k < K; ++k) if (k == K + i) v = win[k];      // old state j + q
      }
      st[(size_t)j * p.channels] = v;
    }
  }
  // BATCH tokens at a time: their loads are under way together (a thread's tokens lie a whole row apart)
  for (int i = i0; i < i1; i += BATCH) {
    float xs[BATCH];
#pragma unroll
    for (int u = 0; u < BATCH; ++u) xs[u] = i + u < i1 ? to_f32(in[(size_t)(t_begin + i + u) * p.in_stride]) : 0.f;
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      if (i + u >= i1) break;
      const float x = xs[u];
      float acc = wt[K] * x;
#pragma unroll
      for (int k = 0; k < K; ++k) acc = fmaf(wt[k], win[k], acc);
#pragma unroll
      for (int k = 0; k + 1 < K; ++k) win[k] = win[k + 1];
      if (K > 0) win[K - 1] = x;
      float y = p.residual ? x + acc : acc + b;
      if (p.act == 1) {
        float one[1] = {y};
        silu<TO>(one);
        y = one[0];
      }
      out[(size_t)(t_begin + i + u) * p.out_stride] = from_f32<TO>(y);
    }
  }
}

// The same with VEC neighbouring channels a thread: 8 bytes (16 in 32-bit) a load where one channel has 2, which is what a portion
// of many tokens is bound by.
constexpr int VEC = 4;

template <typename T> __device__ __forceinline__ void load_raw(uint32_t (&r)[VEC * sizeof(T) / 4], const T* p) {
  if constexpr (sizeof(T) == 4) {
    const uint4 a = *reinterpret_cast<const uint4*>(p);
    r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
  } else {
    const uint2 a = *reinterpret_cast<const uint2*>(p);
    r[0] = a.x; r[1] = a.y;
  }
}
template <typename T> __device__ __forceinline__ float raw_at(const uint32_t (&r)[VEC * sizeof(T) / 4], int v) {
  if constexpr (sizeof(T) == 4) return __uint_as_float(r[v]);
  else return __uint_as_float((v & 1) ? r[v / 2] & 0xffff0000u : r[v / 2] << 16);
}
template <typename T> __device__ __forceinline__ void store_four(T* p, const float (&y)[VEC]) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(y[0], y[1], y[2], y[3]);
  } else {
    const __nv_bfloat162 a = __floats2bfloat162_rn(y[0], y[1]), b = __floats2bfloat162_rn(y[2], y[3]);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  }
}

template <typename TI, typename TO, typename TW, int TAPS>
__global__ void __launch_bounds__(THREADS) short_conv_vec_kernel(const ConvParams p) {
  constexpr int K = TAPS - 1, RAW = VEC * sizeof(TI) / 4, WRAW = VEC * sizeof(TW) / 4;
  static_assert(K > 0, "one tap keeps no state");
  pdl_trigger();
  pdl_wait();
  int entry = -1, seg = 0, before = 0;
  for (int e = 0; e < p.n_entries; ++e) {
    const int q = p.cu_seqlens[e + 1] - p.cu_seqlens[e];
    const int segs = (q + (1 << p.seg_log2) - 1) >> p.seg_log2;
    if ((int)blockIdx.x < before + segs) { entry = e; seg = blockIdx.x - before; break; }
    before += segs;
  }
  if (entry < 0) return;
  const int c = (blockIdx.y * THREADS + threadIdx.x) * VEC;
  if (c >= p.channels) return;
  const int t_begin = p.cu_seqlens[entry], q = p.cu_seqlens[entry + 1] - t_begin;
  const int i0 = seg << p.seg_log2, i1 = min(q, i0 + (1 << p.seg_log2));
  const int slot = p.slots[entry];
  if (slot < 0 || slot >= p.n_slots) {
    if (threadIdx.x == 0) atomicOr(p.status, JV_STATUS_BAD_ROW);
    return;
  }
  const TI* in = (const TI*)p.in + (size_t)t_begin * p.in_stride + c;
  TO* out = (TO*)p.out + (size_t)t_begin * p.out_stride + c;
  float* st = p.state + (size_t)slot * p.state_stride + c;
  uint32_t ahead[BATCH][RAW];
  auto fetch = [&](int i) {
#pragma unroll
    for (int u = 0; u < BATCH; ++u) load_raw<TI>(ahead[u], in + (size_t)min(i + u, i1 - 1) * p.in_stride);
  };
  fetch(i0);
  float wt[TAPS][VEC], bias[VEC] = {}, win[K][VEC];
  {
    uint32_t raw[TAPS][WRAW];                          // TAPS weights of VEC channels, one after another
#pragma unroll
    for (int j = 0; j < TAPS; ++j) load_raw<TW>(raw[j], (const TW*)p.w + (size_t)c * TAPS + j * VEC);
#pragma unroll
    for (int e = 0; e < TAPS * VEC; ++e) wt[e % TAPS][e / TAPS] = raw_at<TW>(raw[e / VEC], e % VEC);
    if (p.bias != nullptr) {
      uint32_t rb[WRAW];
      load_raw<TW>(rb, (const TW*)p.bias + c);
#pragma unroll
      for (int v = 0; v < VEC; ++v) bias[v] = raw_at<TW>(rb, v);
    }
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const int i = i0 - K + k;
    if (i >= 0) {
      uint32_t raw[RAW];
      load_raw<TI>(raw, in + (size_t)i * p.in_stride);
#pragma unroll
      for (int v = 0; v < VEC; ++v) win[k][v] = raw_at<TI>(raw, v);
    } else {
#pragma unroll
      for (int v = 0; v < VEC; ++v) win[k][v] = st[(size_t)(K + i) * p.channels + v];
    }
  }
  if (seg == 0) {
    // the state after this step: the last K inputs of (old state, this entry's tokens)
#pragma unroll
    for (int j = 0; j < K; ++j) {
      const int i = q - K + j;
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        float x = 0.f;
        if (i >= 0) {
          x = to_f32(in[(size_t)i * p.in_stride + v]);
        } else {
#pragma unroll
          for (int k = 0; k < K; ++k) if (k == K + i) x = win[k][v];
        }
        st[(size_t)j * p.channels + v] = x;
      }
    }
  }
  for (int i = i0; i < i1; i += BATCH) {
    uint32_t now[BATCH][RAW];
#pragma unroll
    for (int u = 0; u < BATCH; ++u)
#pragma unroll
      for (int r = 0; r < RAW; ++r) now[u][r] = ahead[u][r];
    if (i + BATCH < i1) fetch(i + BATCH);
#pragma unroll
    for (int u = 0; u < BATCH; ++u) {
      if (i + u >= i1) break;
      float y[VEC];
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        const float x = raw_at<TI>(now[u], v);
        float acc = wt[K][v] * x;
#pragma unroll
        for (int k = 0; k < K; ++k) acc = fmaf(wt[k][v], win[k][v], acc);
#pragma unroll
        for (int k = 0; k + 1 < K; ++k) win[k][v] = win[k + 1][v];
        win[K - 1][v] = x;
        y[v] = p.residual ? x + acc : acc + bias[v];
      }
      if (p.act == 1) silu<TO>(y);
      store_four<TO>(out + (size_t)(i + u) * p.out_stride, y);
    }
  }
}

template <typename TI, typename TO, typename TW>
int launch_taps(const ConvParams& p, int taps, bool vec, dim3 grid, cudaStream_t stream) {
  if (vec) {
    const dim3 wide(grid.x, (p.channels + THREADS * VEC - 1) / (THREADS * VEC));
    switch (taps) {
      case 2: return jv_launch(short_conv_vec_kernel<TI, TO, TW, 2>, wide, dim3(THREADS), 0, stream, p);
      case 3: return jv_launch(short_conv_vec_kernel<TI, TO, TW, 3>, wide, dim3(THREADS), 0, stream, p);
      default: return jv_launch(short_conv_vec_kernel<TI, TO, TW, 4>, wide, dim3(THREADS), 0, stream, p);
    }
  }
  switch (taps) {
    case 1: return jv_launch(short_conv_kernel<TI, TO, TW, 1>, grid, dim3(THREADS), 0, stream, p);
    case 2: return jv_launch(short_conv_kernel<TI, TO, TW, 2>, grid, dim3(THREADS), 0, stream, p);
    case 3: return jv_launch(short_conv_kernel<TI, TO, TW, 3>, grid, dim3(THREADS), 0, stream, p);
    case 4: return jv_launch(short_conv_kernel<TI, TO, TW, 4>, grid, dim3(THREADS), 0, stream, p);
    case 5: return jv_launch(short_conv_kernel<TI, TO, TW, 5>, grid, dim3(THREADS), 0, stream, p);
    case 6: return jv_launch(short_conv_kernel<TI, TO, TW, 6>, grid, dim3(THREADS), 0, stream, p);
    case 7: return jv_launch(short_conv_kernel<TI, TO, TW, 7>, grid, dim3(THREADS), 0, stream, p);
    case 8: return jv_launch(short_conv_kernel<TI, TO, TW, 8>, grid, dim3(THREADS), 0, stream, p);
    default: return JV_ERR_UNSUPPORTED;
  }
}
}  // namespace

JV_EXPORT int jv_short_conv_max_taps() { return 8; }

// in: [n, in_stride] of in_dtype (the first `channels` columns from the pointer); out: [n, out_stride] of out_dtype;
// w: [channels, taps] and bias [channels] (or null) of w_dtype; state: float [n_slots][taps - 1][channels], slots
// `state_stride` elements apart (null only with taps == 1); cu_seqlens [n_entries + 1], slots [n_entries].
// act: 0 none, 1 silu.  residual: out = in + conv (no bias, no activation on the sum unless act says so).
JV_EXPORT int jv_short_conv(const void* in, int in_dtype, long long in_stride, void* out, int out_dtype,
                            long long out_stride, const void* w, const void* bias, int w_dtype, float* state,
                            long long state_stride, const int* cu_seqlens, const int* slots, int n_entries, int n_slots,
                            int n_tokens, int channels, int taps, int act, int residual, int* status,
                            cudaStream_t stream) {
  if (n_tokens == 0 || n_entries == 0 || channels == 0) return JV_OK;
  if (taps < 1 || taps > 8 || act < 0 || act > 1 || (taps > 1 && state == nullptr)) return JV_ERR_UNSUPPORTED;
  ConvParams p;
  p.in = in; p.in_stride = in_stride; p.out = out; p.out_stride = out_stride; p.w = w; p.bias = residual ? nullptr : bias;
  p.state = state; p.state_stride = state_stride; p.cu_seqlens = cu_seqlens; p.slots = slots; p.n_entries = n_entries;
  p.n_slots = n_slots; p.channels = channels; p.act = act; p.residual = residual ? 1 : 0; p.status = status;
  // Four channels a thread where entries have some tokens (or there are 8 M elements), for two to four taps and rows on four-element
  // boundaries; segments as long as the device still fills, since each reads the weights and the taps - 1 inputs before it.  10,240
  // channels, one entry of 130, 700, 4,096 tokens: 5.5, 12.8, 54.8 us, against 9.5, 19.5, 108 a channel a thread (with a silu by the reciprocal
  // alone 4.7, 10.2 and 44.4, segments of 32 throughout 7.4, 14, 45; of 8 4.9, 11, 53).  Entries of one token each a channel a thread: 32 of 2,176
  // channels 5.1 against 7.1.
  auto fours = [](const void* q, long long stride, int dtype) {
    return ((uintptr_t)q & (dtype == 0 ? 15 : 7)) == 0 && stride % VEC == 0;
  };
  const long long size = (long long)n_tokens * channels;
  const bool vec = (size >= (8LL << 20) || (size >= (1LL << 16) && n_tokens >= 8LL * n_entries)) && taps >= 2 && taps <= 4 && channels % VEC == 0 &&
                   fours(in, in_stride, in_dtype) && fours(out, out_stride, out_dtype) && fours(w, 0, w_dtype) &&
                   (bias == nullptr || fours(bias, 0, w_dtype));
  p.seg_log2 = vec && size < (5LL << 20) ? 3 : vec && size < (16LL << 20) ? 4 : 5;
  const dim3 grid((n_tokens >> p.seg_log2) + n_entries, (channels + THREADS - 1) / THREADS);
  JV_DISPATCH_DTYPE(in_dtype, TI, JV_DISPATCH_DTYPE(out_dtype, TO, JV_DISPATCH_DTYPE(w_dtype, TW,
      return launch_taps<TI, TO, TW>(p, taps, vec, grid, stream))));
  return JV_ERR_UNSUPPORTED;
}
