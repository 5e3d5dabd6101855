// The generalized delta rule over portions of several tokens, four tokens at a time (entries of one token run on state_step.cu, a
// scan token by token or in segments is in recurrent.cu).  Per head, with S [key channel, value channel] in 32-bit:
//
//     S <- diag(w_t) S - b_t (u_t^T S) + k_t v_t^T,   o_t = S^T r_t        (both terms of the first read the old S)
//
// Token by token this is a chain: a dot product over the key channels, its sum over the lanes that share a column, an
// update, and again.  But with S_0 the state before a group of four tokens, p_j = u_j^T (old S of token j), and Q_ij =
// w_{i+1} * .. * w_{j-1} element by element,
//
//     p_j = (w_0 .. w_{j-1} u_j)^T S_0  +  sum_{i<j} (u_j . Q_ij k_i) v_i  -  (u_j . Q_ij b_i) p_i
//     o_j = (w_0 .. w_j r_j)^T S_0      +  sum_{i<=j} (r_j . Q_i,j+1 k_i) v_i  -  (r_j . Q_i,j+1 b_i) p_i
//     S_4 = w_0 w_1 w_2 w_3 S_0         +  sum_i (Q_i4 k_i) v_i  -  (Q_i4 b_i) p_i
//
// so all eight dot products of a group read the same S_0 and their sums over the lanes go side by side: one reduction's
// latency a group, not two a token.  Only products of decays appear, never quotients, so a decay of zero is an ordinary number.
// The vectors and the 32 numbers in brackets do not depend on the value columns: group_prepare_kernel makes them once per
// (group, head), fully parallel, and group_scan_kernel reads them through a ring of bulk copies.
//
// What bounds it is that chain's latency (0.5 us a group whatever the number of heads up to two blocks a multiprocessor).
// 2,048 tokens of 32 heads of 64: prepare 40 and scan 197 us, where the token-by-token kernels took 69 and 815; 64 heads: 77 and 260.
#include "mbarrier.cuh"
#include "scan.cuh"

namespace {
constexpr int T4 = 4;                      // tokens of a group
constexpr int VECS = 17;                   // u, r, k, b of the four tokens with their decays, the product of the decays
constexpr int COEF = 64;                   // four 4 x 4 matrices: u.k, u.b, r.k, r.b (zeros where no pair is)

// Sums of 32 numbers a lane over a warp: lane l gets the sum of number l.
__device__ __forceinline__ float warp_sums_32(float (&v)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int half = 16; half > 0; half >>= 1) {
    const bool up = lane & half;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float give = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
    }
  }
  return v[0];
}

// One block per (group of four tokens, head), a thread NCH channels blockDim apart.  packed: [groups, heads, VECS * DP + COEF].
template <int NCH, typename T, typename W>
__global__ void __launch_bounds__(128) group_prepare_kernel(const T* __restrict__ proj, long long stride, int r_off, int k_off,
                                                            int a_off, const T* __restrict__ zw, long long zw_stride,
                                                            const W* __restrict__ a_bias, const W* __restrict__ w_bias,
                                                            const int* __restrict__ cu_seqlens, int n_entries, int portions,
                                                            float* __restrict__ packed, int heads, int D, int DP) {
  __shared__ float norms[4][T4], sums[4][32];
  __shared__ __align__(16) float coef[COEF];
  pdl_trigger();
  pdl_wait();
  int entry, group, n_groups;
  if (!find_segment(cu_seqlens, n_entries, T4, portions, blockIdx.x, entry, group, n_groups)) return;
  const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  const int first = cu_seqlens[entry] + group * T4, tokens = min(T4, cu_seqlens[entry + 1] - first);
  if (tokens <= 0) return;
  // everything that is read, asked for at once; a token or channel that is not there is zero
  float k[NCH][T4], r[NCH][T4], za[NCH][T4], zd[NCH][T4], ab[NCH], wb[NCH], ss[T4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int d = tid + c * blockDim.x, e = h * D + d;
    ab[c] = d < D ? to_f32(a_bias[e]) : 0.f;
    wb[c] = d < D ? to_f32(w_bias[e]) : 0.f;
#pragma unroll
    for (int j = 0; j < T4; ++j) {
      const bool there = j < tokens && d < D;
      const T* row = proj + (size_t)(first + j) * stride + e;
      k[c][j] = there ? to_f32(row[k_off]) : 0.f;
      r[c][j] = there ? to_f32(row[r_off]) : 0.f;
      za[c][j] = there ? to_f32(row[a_off]) : 0.f;
      zd[c][j] = there ? to_f32(zw[(size_t)(first + j) * zw_stride + e]) : 0.f;
    }
  }
#pragma unroll
  for (int c = 0; c < NCH; ++c)
#pragma unroll
    for (int j = 0; j < T4; ++j) ss[j] = fmaf(k[c][j], k[c][j], ss[j]);
#pragma unroll
  for (int j = 0; j < T4; ++j) ss[j] = warp_sum(ss[j]);
  if (lane == 0) {
#pragma unroll
    for (int j = 0; j < T4; ++j) norms[warp][j] = ss[j];
  }
  for (int i = tid; i < COEF; i += blockDim.x) coef[i] = 0.f;
  __syncthreads();
  float inv[T4];
#pragma unroll
  for (int j = 0; j < T4; ++j) {
    float s = 0.f;
    for (int w = 0; w < warps; ++w) s += norms[w][j];
    inv[j] = 1.f / sqrtf(s + 1e-6f);
  }
  const float c0 = 0.60653065971263342f;      // e^(-1/2)
  float* out = packed + ((size_t)blockIdx.x * heads + h) * (VECS * DP + COEF);
  float dots[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) dots[i] = 0.f;
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int d = tid + c * blockDim.x;
    float w[T4], u[T4], b[T4];
#pragma unroll
    for (int j = 0; j < T4; ++j) {             // a token that is not there leaves the state as it is
      const bool there = j < tokens && d < D;
      const float a = 1.f / (1.f + expf(-(za[c][j] + ab[c])));
      w[j] = there ? expf(-c0 / (1.f + expf(-(zd[c][j] + wb[c])))) : 1.f;
      u[j] = k[c][j] * inv[j];
      b[j] = a * u[j];
    }
    float before = 1.f;                        // product of the decays before token j
#pragma unroll
    for (int j = 0; j < T4; ++j) {
      out[j * DP + d] = u[j] * before;
      before *= w[j];
      out[(T4 + j) * DP + d] = r[c][j] * before;
    }
    out[4 * T4 * DP + d] = before;
    // number of a pair: u.k and u.b for i < j, then r.k and r.b for i <= j
#pragma unroll
    for (int i = 0; i < T4; ++i) {
      float kq = k[c][i], bq = b[i];           // times the decays after token i, up to before the reader
#pragma unroll
      for (int j = i; j < T4; ++j) {
        if (j > i) {
          const int q = j * (j - 1) / 2 + i;
          dots[q] = fmaf(u[j], kq, dots[q]);
          dots[6 + q] = fmaf(u[j], bq, dots[6 + q]);
          kq *= w[j];
          bq *= w[j];
        }
        const int q = j * (j + 1) / 2 + i;
        dots[12 + q] = fmaf(r[c][j], kq, dots[12 + q]);
        dots[22 + q] = fmaf(r[c][j], bq, dots[22 + q]);
      }
      out[(2 * T4 + i) * DP + d] = kq;
      out[(3 * T4 + i) * DP + d] = bq;
    }
  }
  sums[warp][lane] = warp_sums_32(dots);
  __syncthreads();
  if (tid < 32) {
    float s = 0.f;
    for (int w = 0; w < warps; ++w) s += sums[w][tid];
    int place;
    if (tid < 12) {
      const int q = tid % 6, j = q < 1 ? 1 : q < 3 ? 2 : 3;
      place = (tid / 6) * 16 + j * 4 + q - j * (j - 1) / 2;
    } else {
      const int q = (tid - 12) % 10, j = q < 1 ? 0 : q < 3 ? 1 : q < 6 ? 2 : 3;
      place = (2 + (tid - 12) / 10) * 16 + j * 4 + q - j * (j + 1) / 2;
    }
    coef[place] = s;
  }
  __syncthreads();
  if (tid < COEF / 4) reinterpret_cast<float4*>(out + VECS * DP)[tid] = reinterpret_cast<const float4*>(coef)[tid];
}

struct GroupScanParams {
  const float* packed;
  const void* v; long long v_stride; int v_off;
  float* out;                              // [n, heads * V]
  float* state; long long slot_stride;     // S of (slot, head) at state + slot * slot_stride + head * D * V
  const int* cu_seqlens; const int* slots;
  int n_slots, heads, D, V;
  int portions, n_entries, max_groups;     // portions > 0: entries of one token are passed by, so many others taken
  int* status;
};

// LANES lanes share a pair of value columns, lane kl the channels 4 LANES i + 4 kl .. + 3 (i < KPT / 4), so that a 16-byte read of eight
// lanes is a run of 128 bytes; a warp takes 64 / LANES columns of one (entry, head), a block twice as many.  Two columns a thread:
// shared memory hands out 128 bytes a clock and each number read should serve more than one multiply-add.
// Eight lanes; 16, which halves what a warp has to do in a group for one more step of every sum over the lanes, where the blocks of eight
// would leave multiprocessors without one and keys have 64 channels or more (32 heads of 64, 2,048 tokens: 258 us with eight, 197 with 16).
// Which of the two hangs on the portions of the step, a portion's sums do not: both add the same numbers in the same order.
// RING_: the stages of the ring.  Six (about 100 KB, two blocks a multiprocessor) carry a block through the latency of its copies;
// where there are more blocks than two a multiprocessor, others do that, and two stages leave room for more of them (32 heads of 64:
// 2,048 tokens in one entry 430 us a layer with six, 598 with two; five entries of 400 313 and 281, eight of 8 tokens 51 and 45).
template <int LANES, int KPT, int RING_> struct GroupScanShape {
  static constexpr int DP = LANES * KPT;
  static constexpr int FLOATS = VECS * DP + COEF;                       // of a group
  static constexpr int GROUPS = DP <= 64 ? 4 : DP <= 128 ? 2 : 1;       // groups of a stage
  static constexpr int RING = RING_, THREADS = 64, COLS = 2 * 64 / LANES;
  static constexpr int VLD = GROUPS * T4 + 4;                           // values of a column in a stage, padded
  static constexpr int STAGE = GROUPS * FLOATS;
  static constexpr int SMEM = (int)sizeof(float) * (RING * STAGE + 2 * COLS * VLD);
};

// (The blocks that its shared memory lets a multiprocessor hold: left to itself the compiler kept to 128 registers and spilled some.)
template <int LANES, int KPT, int RING_, typename T>
__global__ void __launch_bounds__(64, RING_ == 6 ? 2 : LANES * KPT == 32 ? 8 : 4) group_scan_kernel(const GroupScanParams p) {
  using Shape = GroupScanShape<LANES, KPT, RING_>;
  constexpr int DP = Shape::DP, FLOATS = Shape::FLOATS, GROUPS = Shape::GROUPS, RING = Shape::RING, COLS = Shape::COLS;
  constexpr int VLD = Shape::VLD, TOK = GROUPS * T4, Q = KPT / 4, THREADS = Shape::THREADS, RUN = 4 * LANES, WARP_COLS = 64 / LANES;
  constexpr int FINE = LANES / 8;                      // lanes that finish the same output
  // keys of up to 64: a group's vectors are asked for before the group before is finished (there are registers for it)
  constexpr bool AHEAD = Q <= 2;
  extern __shared__ __align__(16) float smem[];
  float* vals = smem + RING * Shape::STAGE;            // [2][COLS][VLD]
  __shared__ uint64_t full[RING];
  pdl_trigger();
  pdl_wait();
  const int entry = entry_of(blockIdx.x, p.portions, p.cu_seqlens, p.n_entries);
  if (entry < 0) return;
  const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int kl = lane % LANES, lcol = warp * WARP_COLS + lane / LANES * 2, base = blockIdx.z * COLS, col = base + lcol;
  const int D = p.D, V = p.V;
  const int t0 = p.cu_seqlens[entry], t1 = p.cu_seqlens[entry + 1];
  const int slot = p.slots[entry];
  if (slot < 0 || slot >= p.n_slots) {
    if (tid == 0) atomicOr(p.status, JV_STATUS_BAD_ROW);
    return;
  }
  if (t0 >= t1) return;
  int g0 = 0;                                          // the number of the entry's first group
  for (int e = 0; e < entry; ++e) g0 += segments_of(p.cu_seqlens[e + 1] - p.cu_seqlens[e], T4, p.portions);
  const int n_groups = (t1 - t0 + T4 - 1) / T4, n_stages = (n_groups + GROUPS - 1) / GROUPS;
  if (g0 + n_groups > p.max_groups) {                  // more portions than were said to be there
    if (tid == 0) atomicOr(p.status, JV_STATUS_BAD_ROW);
    return;
  }
  float* S_g = p.state + (size_t)slot * p.slot_stride + (size_t)h * D * V;
  auto channel = [&](int i) { return (i / 4) * RUN + kl * 4 + (i & 3); };
  const size_t group_stride = (size_t)p.heads * FLOATS;
  const float* src = p.packed + ((size_t)g0 * p.heads + h) * FLOATS;
  // one thread asks for a stage: a bulk copy a group (copies by all threads held up the reads of shared memory behind them)
  auto stage = [&](int s) {
    if (tid != 0 || s >= n_stages) return;
    const int groups = min(GROUPS, n_groups - s * GROUPS);
    mbar_expect_tx(&full[s % RING], groups * FLOATS * 4);
    for (int g = 0; g < groups; ++g)
      bulk_copy(smem + (s % RING) * Shape::STAGE + g * FLOATS, src + (size_t)(s * GROUPS + g) * group_stride, FLOATS * 4, &full[s % RING]);
  };
  // the block's values of a stage: asked for a stage ahead, as they are (a conversion here would wait for them), and put into
  // shared memory when the stage begins
  constexpr int STEP = THREADS / COLS, VPT = (TOK + STEP - 1) / STEP;
  const int vcol = tid % COLS, vtok = tid / COLS;      // tokens vtok + STEP i
  const bool v_live = base + vcol < V;
  const T* vsrc = (const T*)p.v + p.v_off + (size_t)h * V + (v_live ? base + vcol : 0);
  T vr[VPT];
  auto fetch_v = [&](int s) {
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int t = min(t0 + s * TOK + vtok + STEP * i, t1 - 1);
      vr[i] = vsrc[(size_t)t * p.v_stride];
    }
  };
  if (tid == 0) {
    for (int i = 0; i < RING; ++i) mbar_init(&full[i], 1);
    mbar_fence_init();
  }
  __syncthreads();
  for (int s = 0; s < RING - 1; ++s) stage(s);
  fetch_v(0);
  uint64_t S[2][KPT / 2];
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int i = 0; i < KPT / 2; ++i) {
      const int c0 = channel(2 * i), c1 = channel(2 * i + 1);
      S[c][i] = pack2(col + c < V && c0 < D ? S_g[(size_t)c0 * V + col + c] : 0.f,
                      col + c < V && c1 < D ? S_g[(size_t)c1 * V + col + c] : 0.f);
    }
  const int jo = kl / FINE >> 1, co = kl / FINE & 1;   // the token of a group and the column whose output this lane finishes
  const size_t orow = (size_t)p.heads * V;
  float* o_next = p.out + (size_t)t0 * orow + (size_t)h * V + col + co + jo * orow;
  const bool live = col + co < V && kl % FINE == 0;
  ulonglong2 U[T4][Q], R[T4][Q];
  auto load_ur = [&](const float* vec) {
#pragma unroll
    for (int j = 0; j < T4; ++j)
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        U[j][q] = *reinterpret_cast<const ulonglong2*>(vec + j * DP + q * RUN);
        R[j][q] = *reinterpret_cast<const ulonglong2*>(vec + (T4 + j) * DP + q * RUN);
      }
  };
  // A lane of eight holds the channels of two of the 16: they are summed up apart, and then together, as two of the 16 do it.
  constexpr int HELD = LANES == 8 && Q >= 2 ? 2 : 1;
  auto dot = [&](const ulonglong2 (&x)[Q], const uint64_t (&s)[KPT / 2]) {
    float sum[HELD];
#pragma unroll
    for (int k = 0; k < HELD; ++k) {
      uint64_t a = 0;
#pragma unroll
      for (int q = k; q < Q; q += HELD) a = fma2(x[q].y, s[2 * q + 1], fma2(x[q].x, s[2 * q], a));
      float lo, hi;
      unpack2(a, lo, hi);
      sum[k] = lo + hi;
    }
    return HELD == 2 ? sum[0] + sum[HELD - 1] : sum[0];
  };
  for (int s = 0; s < n_stages; ++s) {
    float* vbuf = vals + (s & 1) * COLS * VLD;
#pragma unroll
    for (int i = 0; i < VPT; ++i) {
      const int j = vtok + STEP * i;
      if (j < TOK) vbuf[vcol * VLD + j] = v_live && t0 + s * TOK + j < t1 ? to_f32(vr[i]) : 0.f;
    }
    // the stage has landed; the one before it has been read
    const bool landed = mbar_wait(&full[s % RING], (s / RING) & 1);
    if (!__syncthreads_and(landed)) {
      if (tid == 0) {                                  // the copies already asked for get a bounded time to land
        atomicOr(p.status, JV_STATUS_WAIT_EXPIRED);
        for (int i = s; i < min(s + RING - 1, n_stages); ++i) drain_copies_after_failure(&full[i % RING], (i / RING) & 1);
      }
      __syncthreads();
      return;
    }
    stage(s + RING - 1);
    if (s + 1 < n_stages) fetch_v(s + 1);
    const int groups = min(GROUPS, n_groups - s * GROUPS);
    const float* stage_vecs = smem + (s % RING) * Shape::STAGE + kl * 4;
    if (AHEAD) load_ur(stage_vecs);
    auto do_group = [&](const int g, const bool more) {
      const float* vec = stage_vecs + g * FLOATS;
      const float* cf = smem + (s % RING) * Shape::STAGE + g * FLOATS + VECS * DP;
      if (!AHEAD) load_ur(vec);
      float dp[2][T4], dr[2][T4];
#pragma unroll
      for (int j = 0; j < T4; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) dp[c][j] = dot(U[j], S[c]);
      // while the p's sums travel between the lanes: what needs no p
      auto exchange = [&](int m) {
#pragma unroll
        for (int j = 0; j < T4; ++j)
#pragma unroll
          for (int c = 0; c < 2; ++c) dp[c][j] += __shfl_xor_sync(0xffffffffu, dp[c][j], m);
      };
      if (LANES == 16) exchange(8);
      exchange(4);
      float v[2][T4];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float4 x = *reinterpret_cast<const float4*>(vbuf + (lcol + c) * VLD + g * T4);
        v[c][0] = x.x; v[c][1] = x.y; v[c][2] = x.z; v[c][3] = x.w;
      }
      float fk[T4][T4], fb[T4][T4];
#pragma unroll
      for (int j = 1; j < T4; ++j) {
        const float4 uk = *reinterpret_cast<const float4*>(cf + j * 4), ub = *reinterpret_cast<const float4*>(cf + 16 + j * 4);
        fk[j][0] = uk.x; fk[j][1] = uk.y; fk[j][2] = uk.z;
        fb[j][0] = ub.x; fb[j][1] = ub.y; fb[j][2] = ub.z;
      }
#pragma unroll
      for (int j = 0; j < T4; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) dr[c][j] = dot(R[j], S[c]);
      exchange(2);
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(vec + 4 * T4 * DP + q * RUN);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          S[c][2 * q] = mul2(w.x, S[c][2 * q]);
          S[c][2 * q + 1] = mul2(w.y, S[c][2 * q + 1]);
        }
#pragma unroll
        for (int j = 0; j < T4; ++j) {
          const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(vec + (2 * T4 + j) * DP + q * RUN);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const uint64_t vv = pack2(v[c][j], v[c][j]);
            S[c][2 * q] = fma2(k.x, vv, S[c][2 * q]);
            S[c][2 * q + 1] = fma2(k.y, vv, S[c][2 * q + 1]);
          }
        }
      }
      exchange(1);
      ulonglong2 B[T4][Q];
#pragma unroll
      for (int j = 0; j < T4; ++j)
#pragma unroll
        for (int q = 0; q < Q; ++q) B[j][q] = *reinterpret_cast<const ulonglong2*>(vec + (3 * T4 + j) * DP + q * RUN);
      if (AHEAD && more) load_ur(vec + FLOATS);
      // the p's one after the other
#pragma unroll
      for (int j = 1; j < T4; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
          for (int i = 0; i < j; ++i) dp[c][j] = fmaf(fk[j][i], v[c][i], dp[c][j]);
        }
#pragma unroll
      for (int j = 1; j < T4; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
          for (int i = 0; i < j; ++i) dp[c][j] = fmaf(-fb[j][i], dp[c][i], dp[c][j]);
        }
#pragma unroll
      for (int j = 0; j < T4; ++j)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const uint64_t np = pack2(-dp[c][j], -dp[c][j]);
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            S[c][2 * q] = fma2(B[j][q].x, np, S[c][2 * q]);
            S[c][2 * q + 1] = fma2(B[j][q].y, np, S[c][2 * q + 1]);
          }
        }
      // the outputs: eight sums over eight lanes, a lane hands on those that it does not finish
      const bool up = kl & 4 * FINE, up2 = kl & 2 * FINE, up1 = kl & FINE;
      float e[4], f[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) {                    // (token i / 2 of a half, column i & 1)
        const float lo = dr[i & 1][i >> 1], hi = dr[i & 1][2 + (i >> 1)];
        e[i] = (up ? hi : lo) + __shfl_xor_sync(0xffffffffu, up ? lo : hi, 4 * FINE);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) f[i] = (up2 ? e[2 + i] : e[i]) + __shfl_xor_sync(0xffffffffu, up2 ? e[i] : e[2 + i], 2 * FINE);
      float o = (up1 ? f[1] : f[0]) + __shfl_xor_sync(0xffffffffu, up1 ? f[0] : f[1], FINE);
      if (FINE > 1) o += __shfl_xor_sync(0xffffffffu, o, 1);
      const float4 rk = *reinterpret_cast<const float4*>(cf + 32 + jo * 4), rb = *reinterpret_cast<const float4*>(cf + 48 + jo * 4);
      const float ok[T4] = {rk.x, rk.y, rk.z, rk.w}, ob[T4] = {rb.x, rb.y, rb.z, rb.w};
#pragma unroll
      for (int i = 0; i < T4; ++i) {                   // a later token's infinity stays out of an earlier one's output
        o = fmaf(ok[i], i <= jo ? (up1 ? v[1][i] : v[0][i]) : 0.f, o);
        o = fmaf(-ob[i], i <= jo ? (up1 ? dp[1][i] : dp[0][i]) : 0.f, o);
      }
      if (live && t0 + s * TOK + g * T4 + jo < t1) *o_next = o;
      o_next += T4 * orow;
    };
    if (groups == GROUPS) {                            // a whole stage in one piece: a group's outputs are finished under the next one's sums
#pragma unroll
      for (int g = 0; g < GROUPS; ++g) do_group(g, g + 1 < GROUPS);
    } else {
#pragma unroll 1
      for (int g = 0; g < groups; ++g) do_group(g, g + 1 < groups);
    }
  }
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int i = 0; i < KPT / 2; ++i) {
      const int c0 = channel(2 * i), c1 = channel(2 * i + 1);
      float a, b;
      unpack2(S[c][i], a, b);
      if (col + c < V && c0 < D) S_g[(size_t)c0 * V + col + c] = a;
      if (col + c < V && c1 < D) S_g[(size_t)c1 * V + col + c] = b;
    }
}

template <int LANES, int KPT, int RING, typename T>
int launch_ring(const GroupScanParams& p, int entries, cudaStream_t stream) {
  using Shape = GroupScanShape<LANES, KPT, RING>;
  auto kern = group_scan_kernel<LANES, KPT, RING, T>;
  static bool done[JV_MAX_DEVICES] = {};
  if (!jv_once_per_device(done, [&] {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::SMEM) == cudaSuccess;
      }))
    return JV_ERR_UNSUPPORTED;
  return jv_launch(kern, dim3(entries, p.heads, (p.V + Shape::COLS - 1) / Shape::COLS), dim3(Shape::THREADS), Shape::SMEM, stream, p);
}

template <int KPT, typename T>
int launch_scan(const GroupScanParams& p, int entries, cudaStream_t stream) {
  constexpr int COLS = GroupScanShape<8, KPT, 6>::COLS;
  const long long blocks = (long long)entries * p.heads * ((p.V + COLS - 1) / COLS);
  if constexpr (KPT >= 8) {
    if (blocks <= jv_multiprocessors()) return launch_ring<16, KPT / 2, 6, T>(p, entries, stream);
  }
  return blocks > 2 * jv_multiprocessors() ? launch_ring<8, KPT, 2, T>(p, entries, stream) : launch_ring<8, KPT, 6, T>(p, entries, stream);
}

int padded(int D) { return D <= 32 ? 32 : D <= 64 ? 64 : D <= 128 ? 128 : 256; }
}  // namespace

// Floats of `packed` a (group, head) of keys of D channels.
JV_EXPORT int jv_delta_group_floats(int D) { return VECS * padded(D) + COEF; }

// Both kernels.  proj: [n] rows of `stride` elements of dtype `dtype` holding r, k, the removal gate's pre-activation
// (heads * D each) and the values (heads * V) at the given columns; zw, a_bias, w_bias as for jv_delta_prepare; packed: at least
// (n / 4 + entries) * heads * jv_delta_group_floats(D) floats, 16-byte aligned; state [n_slots] rows of `slot_stride` floats;
// out [n, heads * V].  portions > 0: entries of one token are passed by, which leaves this many, with n tokens.
JV_EXPORT int jv_delta_scan(const void* proj, int dtype, long long stride, int r_off, int k_off, int a_off, int v_off,
                            const void* zw, long long zw_stride, const void* a_bias, const void* w_bias, int w_dtype,
                            float* packed, float* state, long long slot_stride, const int* cu_seqlens, const int* slots,
                            int n_slots, int entries, float* out, int n, int heads, int D, int V, int portions, int* status,
                            cudaStream_t stream) {
  if (entries == 0 || n == 0) return JV_OK;
  if (D < 1 || D > 256 || V < 1 || heads > 65535) return JV_ERR_UNSUPPORTED;
  const int DP = padded(D);
  const dim3 grid(n / T4 + (portions > 0 ? portions : entries), heads);
  int rc = JV_ERR_UNSUPPORTED;
  JV_DISPATCH_DTYPE(dtype, T, JV_DISPATCH_DTYPE(w_dtype, W, rc = jv_launch(
      DP == 256 ? group_prepare_kernel<2, T, W> : group_prepare_kernel<1, T, W>, grid, dim3(DP == 256 ? 128 : DP), 0, stream,
      (const T*)proj, stride, r_off, k_off, a_off, (const T*)zw, zw_stride, (const W*)a_bias, (const W*)w_bias, cu_seqlens, entries,
      portions, packed, heads, D, DP)));
  if (rc != JV_OK) return rc;
  GroupScanParams p{packed, proj, stride, v_off, out, state, slot_stride, cu_seqlens, slots, n_slots, heads, D, V, portions, entries,
                    (int)grid.x, status};
  if (portions > 0) entries = portions;
  JV_DISPATCH_DTYPE(dtype, T, {
    switch (DP) {
      case 32: return launch_scan<4, T>(p, entries, stream);
      case 64: return launch_scan<8, T>(p, entries, stream);
      case 128: return launch_scan<16, T>(p, entries, stream);
      default: return launch_scan<32, T>(p, entries, stream);
    }
  });
  return JV_ERR_UNSUPPORTED;
}
