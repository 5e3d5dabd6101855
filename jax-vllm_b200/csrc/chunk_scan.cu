// Matrix states with ONE decay a head and token, over portions of many tokens, 32 tokens at a time on the tensor cores:
//
//     S <- a_t S + g_t k_t v_t^T,   o_t = scale * S^T q_t                     (S [key channel, value channel] in 32-bit)
//
//   state-space mixer    a = exp(-exp(A_log) dt), g = dt = softplus(dt_raw + dt_bias), k = B and q = C of the head's group, v = x
//   matrix memory        a = keep, g = take (jv_memory_gates), and one more column whose value is 1 (the normaliser)
//
// Token by token (recurrent.cu) every state element costs three multiply-adds a token.  With S_0 the state before a chunk
// and L_t = log a_1 + .. + log a_t inside it,
//
//     o_t = exp(L_t) S_0^T q_t + sum_{s <= t} (q_t . k_s) g_s exp(L_t - L_s) v_s
//     S_T = exp(L_T) S_0 + sum_s k_s (g_s exp(L_T - L_s) v_s)^T
//
// which are four small matrix products.  q, k and v are 16-bit numbers, the operands on the other side are 32-bit: S_0, the
// weighted scores and the weighted values.  A 32-bit number is cut into three 16-bit ones (x = hi + mid + lo, eight bits of
// mantissa each, exactly), so that the three products with a 16-bit number are exact and only the sums round.  The tensor
// core's sums cut where the CUDA cores' round: a sum of 16 products starts from zero there (smallest parts first) and is
// added to the running one on the CUDA cores (one running sum in the tensor core: 3.4e-7 relative for 128 channels, this way 0.8e-7,
// as token by token).  L is summed in 64-bit and kept as two floats: L_t - L_s keeps its digits behind a large decay.
//
// A block is one (entry, head, ET value columns), a warp 16 of the columns: its rows of S^T are the accumulators of the state's
// update and, cut in three in registers, the left operand of the products with q.  The scores are shared by the warps through
// shared memory; one more warp brings the rows of the chunks ahead (bulk copies) and makes their weights.  Nothing but the
// outputs goes to memory between an entry's first token and its last.
//
// What bounds it is the latency of a chunk's phases (3 to 5 us, of which the products are a third), so it pays where many blocks
// run side by side.  4,096 tokens in three entries, 128 heads of 128 x 64: 612 us, 1,476 and 178 for the scan and its preparation
// token by token; 2,048 tokens of 64 such heads: 329 us, 450 and 60.
#include "mbarrier.cuh"
#include "scan.cuh"
#include <math.h>

#include <type_traits>

namespace {
constexpr int TT = 32;                     // tokens of a chunk
constexpr int NBUF = 3;                    // chunks whose rows and weights have a place
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
  const int *cu_seqlens, *slots;
  int n_slots, heads, D, V;
  int portions, n_entries;                 // portions > 0: entries of one token are passed by, so many others taken
  int* status;
};

__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void add(float (&c)[4], const float (&f)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) c[i] += f[i];
}
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], const bf16* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
__device__ __forceinline__ void ldsm_t(uint32_t (&r)[4], const bf16* p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a));
}
// A barrier of the warps at work; true if `ok` is true in all of them.
template <int THREADS> __device__ __forceinline__ bool work_sync(bool ok) {
  int all;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.s32 p, %1, 0;\nbar.red.and.pred q, 1, %2, p;\nselp.s32 %0, 1, 0, q;\n}\n"
               : "=r"(all) : "r"((int)ok), "n"(THREADS) : "memory");
  return all != 0;
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

// D: key channels rounded up (channels past p.D are zeros); ET = 16 * WARPS value columns a block.
template <int D, int WARPS> struct ChunkShape {
  static constexpr int ET = 16 * WARPS, LD = D + 8, LE = ET + 8, LS = TT + 8;      // padded rows: no bank is met twice
  static constexpr int QK = TT * LD, X = TT * LE, M = TT * LS;
  static constexpr int BF16S = NBUF * (2 * QK + X) + 3 * X + 3 * M;
  static constexpr int SMEM = BF16S * 2 + NBUF * (TT * (8 + 3 * 4) + 16) + (ET + 1) * 4;
};

// What a chunk's tokens weigh.
struct Weights {
  float2 L[TT];                              // L_t as a leading and a following number
  float g[TT], from_start[TT], to_end[TT];   // g_s, exp(L_t), g_s exp(L_T - L_s)
  float whole, pad[3];                       // exp(L_T)
};
static_assert(sizeof(Weights) == TT * 20 + 16, "the shared memory's size counts on it");

template <int D, int WARPS>
__global__ void __launch_bounds__(32 * WARPS + 32) chunk_scan_kernel(const ChunkParams p) {
  using Shape = ChunkShape<D, WARPS>;
  constexpr int ET = Shape::ET, LD = Shape::LD, LE = Shape::LE, LS = Shape::LS, KT = D / 16;
  extern __shared__ __align__(16) unsigned char raw[];
  Weights* weights = reinterpret_cast<Weights*>(raw);                            // [NBUF]
  bf16* qs = reinterpret_cast<bf16*>(weights + NBUF);                            // [NBUF][TT][LD]
  bf16* ks = qs + NBUF * Shape::QK;                                              // [NBUF][TT][LD]
  bf16* xs = ks + NBUF * Shape::QK;                                              // [NBUF][TT][LE]
  bf16* xw = xs + NBUF * Shape::X;                                               // [3][TT][LE] weighted values, in three
  bf16* ms = xw + 3 * Shape::X;                                                  // [3][TT][LS] weighted scores [t][s], in three
  int* bad = reinterpret_cast<int*>(ms + 3 * Shape::M);                          // [ET] first token whose value is no number, [ET]: any
  __shared__ uint64_t rows_full[NBUF], weights_full[NBUF], empty[NBUF];
  pdl_trigger();
  pdl_wait();
  const int entry = entry_of(blockIdx.x, p.portions, p.cu_seqlens, p.n_entries);
  if (entry < 0) return;
  const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gr = lane >> 2, gq = lane & 3;             // row and column pair of a fragment
  const int e0 = blockIdx.z * ET;
  const int t0 = p.cu_seqlens[entry], len = p.cu_seqlens[entry + 1] - t0;
  const int slot = p.slots[entry];
  if (slot < 0 || slot >= p.n_slots) {
    if (tid == 0) atomicOr(p.status, JV_STATUS_BAD_ROW);
    return;
  }
  if (len <= 0) return;
  const int chunks = (len + TT - 1) / TT, V = p.V, v_all = V + (p.state_n != nullptr ? 1 : 0);
  const bf16* q_g = p.q + (size_t)t0 * p.q_stride + (h / p.per_group) * p.D;
  const bf16* k_g = p.k + (size_t)t0 * p.k_stride + (h / p.per_group) * p.D;
  const bf16* v_g = p.v + (size_t)t0 * p.v_stride + (size_t)h * V;

  // a copy brings a row: `dk` elements of q and of k, `dx` of v; what lies past them is zero, but for the normaliser's column
  const int dk = p.D, dx = max(0, min(ET, V - e0));
  for (int i = tid; i < (Shape::BF16S * 2) / 16; i += 32 * WARPS + 32) reinterpret_cast<uint4*>(qs)[i] = make_uint4(0, 0, 0, 0);
  for (int i = tid; i <= ET; i += 32 * WARPS + 32) bad[i] = i < ET ? TT : 0;
  if (tid < NBUF) {
    mbar_init(&rows_full[tid], 1);
    mbar_init(&weights_full[tid], 1);
    mbar_init(&empty[tid], WARPS);
    mbar_fence_init();
  }
  __syncthreads();
  if (v_all > V && V >= e0 && V < e0 + ET && tid < NBUF * TT) xs[tid * LE + V - e0] = __float2bfloat16_rn(1.f);
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  __syncthreads();
  auto stage = [&](int c) {                            // chunk c's rows, by one warp
    const int buf = c % NBUF, here = min(TT, len - c * TT);
    if (lane == 0) mbar_expect_tx(&rows_full[buf], here * (2 * dk + dx) * 2);
    __syncwarp();
    if (lane < here) {
      const size_t t = (size_t)c * TT + lane;
      bulk_copy(qs + buf * Shape::QK + lane * LD, q_g + t * p.q_stride, dk * 2, &rows_full[buf]);
      bulk_copy(ks + buf * Shape::QK + lane * LD, k_g + t * p.k_stride, dk * 2, &rows_full[buf]);
      if (dx > 0) bulk_copy(xs + buf * Shape::X + lane * LE, v_g + t * p.v_stride + e0, dx * 2, &rows_full[buf]);
    } else {                                           // past the entry's end
      for (int i = 0; i < D; i += 8) {
        *reinterpret_cast<uint4*>(qs + buf * Shape::QK + lane * LD + i) = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(ks + buf * Shape::QK + lane * LD + i) = make_uint4(0, 0, 0, 0);
      }
      for (int i = 0; i < ET; i += 8) *reinterpret_cast<uint4*>(xs + buf * Shape::X + lane * LE + i) = make_uint4(0, 0, 0, 0);
    }
  };
  // what the decays and steps of a chunk's tokens come from, a lane a token
  float2 in_gates = make_float2(0.f, 0.f);
  unsigned short in_dt = 0;                            // as it is: a conversion where it is asked for would wait for it
  float rate = 0.f, bias = 0.f;
  if (p.gates == nullptr) {
    rate = p.w_dtype == 0 ? ((const float*)p.a_log)[h] : to_f32(((const bf16*)p.a_log)[h]);
    bias = p.w_dtype == 0 ? ((const float*)p.dt_bias)[h] : to_f32(((const bf16*)p.dt_bias)[h]);
    rate = expf(rate);
  }
  auto fetch_gates = [&](int c) {
    const int t = t0 + min(c * TT + lane, len - 1);
    if (p.gates != nullptr) in_gates = *reinterpret_cast<const float2*>(p.gates + ((size_t)t * p.heads + h) * 4);
    else in_dt = *reinterpret_cast<const unsigned short*>(p.dt_raw + (size_t)t * p.dt_stride + h);
  };
  auto make_weights = [&](int c) {                     // one whole warp
    Weights& w = weights[c % NBUF];
    const bool there = c * TT + lane < len;
    float g, log_a;
    if (p.gates != nullptr) {
      g = in_gates.y;
      log_a = logf(in_gates.x);
    } else {
      const float z = __uint_as_float((uint32_t)in_dt << 16) + bias;
      g = fmaxf(z, 0.f) + log1pf(expf(-fabsf(z)));     // softplus, no clamp
      log_a = -rate * g;
    }
    // below -1e4 a decay is zero in any case, and a sum of them stays a number
    double L = there ? (double)(log_a < -1e4f ? -1e4f : log_a) : 0.0;
    if (!there) g = 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double before = __shfl_up_sync(0xffffffffu, L, o);
      if (lane >= o) L += before;
    }
    const double end = __shfl_sync(0xffffffffu, L, 31);
    w.L[lane] = make_float2((float)L, (float)(L - (double)(float)L));
    w.g[lane] = g;
    w.from_start[lane] = expf((float)L);
    w.to_end[lane] = there ? g * expf((float)(end - L)) : 0.f;
    if (lane == 0) w.whole = expf((float)end);
  };

  if (warp == WARPS) {
    // the last warp only supplies: rows up to NBUF chunks ahead, weights as soon as a place is free
    fetch_gates(0);
    bool ok = true;
    int staged = 0;
    for (; staged < min(NBUF, chunks); ++staged) stage(staged);
    for (int c = 0; c < chunks; ++c) {
      if (c >= NBUF) {                                 // the place's last chunk is done with
        ok = __all_sync(0xffffffffu, mbar_wait(&empty[c % NBUF], (c / NBUF - 1) & 1));
        if (!ok) break;
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        stage(c);
        ++staged;
      }
      make_weights(c);
      fetch_gates(c + 1);
      __syncwarp();
      if (lane == 0) mbar_arrive(&weights_full[c % NBUF]);
    }
    if (!ok && lane == 0) atomicOr(p.status, JV_STATUS_WAIT_EXPIRED);
    // whatever became of the others, the copies asked for land (or get a bounded time to) before the block may end
    for (int c = max(0, staged - NBUF); c < staged; ++c) mbar_wait(&rows_full[c % NBUF], (c / NBUF) & 1);
    return;
  }
  // this warp's 16 columns of the state: fragments of S^T [column][channel]
  const int er = e0 + warp * 16 + gr;                  // and er + 8
  float S[2 * KT][4];
#pragma unroll
  for (int j = 0; j < 2 * KT; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = er + (i >> 1) * 8, d = j * 8 + gq * 2 + (i & 1);
      float s = 0.f;
      if (d < p.D) {
        if (e < V) s = p.state[(size_t)slot * p.slot_stride + ((size_t)h * p.D + d) * V + e];
        else if (e < v_all) s = p.state_n[(size_t)slot * p.slot_stride + (size_t)h * p.D + d];
      }
      S[j][i] = s;
    }
  const bool at_work = e0 + warp * 16 < v_all;         // some column of this warp is used

  // where a lane's address of an ldmatrix lies: its row of an 8 x 8 block, and the block
  const int lr = lane & 7, lm = lane >> 3;
  for (int c = 0; c < chunks; ++c) {
    const int buf = c % NBUF, phase = (c / NBUF) & 1;
    const bf16 *q = qs + buf * Shape::QK, *k = ks + buf * Shape::QK;
    bf16* x = xs + buf * Shape::X;
    // the chunk is there, and the warps are done with the scores and weighted values of the one before
    const bool here = mbar_wait(&rows_full[buf], phase) && mbar_wait(&weights_full[buf], phase);
    if (!work_sync<32 * WARPS>(here)) {
      if (tid == 0) atomicOr(p.status, JV_STATUS_WAIT_EXPIRED);
      return;
    }
    const Weights& w = weights[buf];
    // weighted values, in three; a value that is no number is taken out and remembered, since the zeros of scores that
    // look ahead would carry it into earlier outputs
    {
      constexpr int PER = TT * (ET / 2) / (32 * WARPS), STEP = 32 * WARPS / (ET / 2);     // pairs of columns a thread: tokens STEP apart
      const int e = tid % (ET / 2) * 2, s0 = tid / (ET / 2);
      uint32_t both[PER];
      bool no_number = false;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        both[i] = *reinterpret_cast<const uint32_t*>(x + (s0 + i * STEP) * LE + e);
        no_number |= (both[i] & 0x7f80u) == 0x7f80u || (both[i] & 0x7f800000u) == 0x7f800000u;
      }
      if (no_number) {
#pragma unroll 1
        for (int i = 0; i < PER; ++i) {
          const int s = s0 + i * STEP;
          uint32_t v = *reinterpret_cast<const uint32_t*>(x + s * LE + e);
          if ((v & 0x7f80u) == 0x7f80u) { atomicMin(bad + e, s); v &= 0xffff0000u; }
          if ((v & 0x7f800000u) == 0x7f800000u) { atomicMin(bad + e + 1, s); v &= 0xffffu; }
          *reinterpret_cast<uint32_t*>(x + s * LE + e) = v;
        }
        bad[ET] = 1;
#pragma unroll
        for (int i = 0; i < PER; ++i) both[i] = *reinterpret_cast<const uint32_t*>(x + (s0 + i * STEP) * LE + e);
      }
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int s = s0 + i * STEP;
        const float f = w.to_end[s];
        uint32_t hi, mid, lo;
        cut3(__uint_as_float(both[i] << 16) * f, __uint_as_float(both[i] & 0xffff0000u) * f, hi, mid, lo);
        *reinterpret_cast<uint32_t*>(xw + s * LE + e) = hi;
        *reinterpret_cast<uint32_t*>(xw + Shape::X + s * LE + e) = mid;
        *reinterpret_cast<uint32_t*>(xw + 2 * Shape::X + s * LE + e) = lo;
      }
    }
    // Scores q_t . k_s, 16 tokens t by 8 * UNITS tokens s at a time.  Of the four squares of 16 x 16 the one whose s all lie
    // behind its t is left out (its places in shared memory are never read); the two on the diagonal go to a warp each, the
    // halves of the last to the same warps, or to two others.
    auto scores = [&](const int tm, const int sn, auto units) {
      constexpr int UNITS = decltype(units)::value;
      float G[2][4] = {};
#pragma unroll
      for (int kk = 0; kk < KT; ++kk) {
        uint32_t a[4], b[4];
        ldsm(a, q + (tm + lr + (lm & 1) * 8) * LD + kk * 16 + (lm >> 1) * 8);
        ldsm(b, k + (sn + lr + (UNITS == 2 ? (lm >> 1) * 8 : 0)) * LD + kk * 16 + (lm & 1) * 8);
#pragma unroll
        for (int j = 0; j < UNITS; ++j) {
          float f[4] = {};
          mma(f, a, b[2 * j], b[2 * j + 1]);
          add(G[j], f);
        }
      }
#pragma unroll
      for (int j = 0; j < UNITS; ++j)
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
          const int t = tm + gr + (i >> 1) * 8, s = sn + j * 8 + gq * 2;
          const float2 lt = w.L[t], l0 = w.L[s], l1 = w.L[s + 1];
          const float m0 = s <= t ? G[j][i] * (w.g[s] * expf((lt.x - l0.x) + (lt.y - l0.y))) : 0.f;
          const float m1 = s + 1 <= t ? G[j][i + 1] * (w.g[s + 1] * expf((lt.x - l1.x) + (lt.y - l1.y))) : 0.f;
          uint32_t hi, mid, lo;
          cut3(m0, m1, hi, mid, lo);
          *reinterpret_cast<uint32_t*>(ms + t * LS + s) = hi;
          *reinterpret_cast<uint32_t*>(ms + Shape::M + t * LS + s) = mid;
          *reinterpret_cast<uint32_t*>(ms + 2 * Shape::M + t * LS + s) = lo;
        }
    };
    if (warp < 2) scores(warp * 16, warp * 16, std::integral_constant<int, 2>());
    if (WARPS == 2 || warp >= 2) scores(16, (warp & 1) * 8, std::integral_constant<int, 1>());
    work_sync<32 * WARPS>(true);
    if (at_work) {
      // what the state of before gives: S^T q, then exp(L_t) on the tokens
      float O[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) O[j][i] = 0.f;
#pragma unroll
      for (int kk = 0; kk < KT; kk += 2) {
        uint32_t a[2][3][4], b[2][2][4];
        float f[2][4][4] = {};
#pragma unroll
        for (int u = 0; u < 2; ++u) {
#pragma unroll
          for (int j = 0; j < 2; ++j) ldsm(b[u][j], q + (j * 16 + lr + (lm >> 1) * 8) * LD + (kk + u) * 16 + (lm & 1) * 8);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float(&s)[4] = S[2 * (kk + u) + i];
            cut3(s[0], s[1], a[u][0][2 * i], a[u][1][2 * i], a[u][2][2 * i]);
            cut3(s[2], s[3], a[u][0][2 * i + 1], a[u][1][2 * i + 1], a[u][2][2 * i + 1]);
          }
        }
#pragma unroll
        for (int z = 2; z >= 0; --z)
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int j = 0; j < 4; ++j) mma(f[u][j], a[u][z], b[u][j >> 1][(j & 1) * 2], b[u][j >> 1][(j & 1) * 2 + 1]);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i) O[j][i] += f[0][j][i] + f[1][j][i];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = *reinterpret_cast<const float2*>(&w.from_start[j * 8 + gq * 2]);
        O[j][0] *= f.x; O[j][1] *= f.y; O[j][2] *= f.x; O[j][3] *= f.y;
      }
      // what the chunk's own tokens give
#pragma unroll
      for (int kk = 0; kk < TT / 16; ++kk) {
        uint32_t a[4];
        ldsm_t(a, x + (kk * 16 + lr + (lm >> 1) * 8) * LE + warp * 16 + (lm & 1) * 8);
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          if (kk * 16 > j * 8 + 15) continue;          // tokens s that all lie behind these t
          float f[2][4] = {};
#pragma unroll
          for (int z = 2; z >= 0; --z) {
            uint32_t b[4];
            ldsm(b, ms + z * Shape::M + (j * 8 + lr + (lm >> 1) * 8) * LS + kk * 16 + (lm & 1) * 8);
            mma(f[0], a, b[0], b[1]);
            mma(f[1], a, b[2], b[3]);
          }
          add(O[j], f[0]);
          add(O[j + 1], f[1]);
        }
      }
      const bool any_bad = bad[ET] != 0;
      {
        const size_t orow = (size_t)p.heads * V;
        float* o = p.out + ((size_t)t0 + c * TT + gq * 2) * orow + (size_t)h * V + er;
        if (!any_bad && (c + 1) * TT <= len && e0 + warp * 16 + 16 <= V) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            o[0] = O[j][0] * p.scale; o[8] = O[j][2] * p.scale;
            o += orow;
            o[0] = O[j][1] * p.scale; o[8] = O[j][3] * p.scale;
            o += 7 * orow;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int t = j * 8 + gq * 2 + (i & 1), e = er + (i >> 1) * 8;
              if (c * TT + t < len) {
                const float y = any_bad && bad[e - e0] <= t ? NAN : O[j][i] * p.scale;
                if (e < V) o[(size_t)(j * 8 + (i & 1)) * orow + (i >> 1) * 8] = y;
                else if (e < v_all) p.nq[(((size_t)t0 + c * TT + t) * p.heads + h) * 4] = y;
              }
            }
        }
      }
      // the state after the chunk
      const float whole = w.whole;
      uint32_t a[TT / 16][3][4];
#pragma unroll
      for (int kk = 0; kk < TT / 16; ++kk)
#pragma unroll
        for (int z = 0; z < 3; ++z)
          ldsm_t(a[kk][z], xw + z * Shape::X + (kk * 16 + lr + (lm >> 1) * 8) * LE + warp * 16 + (lm & 1) * 8);
#pragma unroll
      for (int j = 0; j < 2 * KT; j += 4) {
        float f[TT / 16][4][4] = {};
        uint32_t b[TT / 16][2][4];
#pragma unroll
        for (int kk = 0; kk < TT / 16; ++kk)
#pragma unroll
          for (int i = 0; i < 2; ++i) ldsm_t(b[kk][i], k + (kk * 16 + lr + (lm & 1) * 8) * LD + (j + 2 * i) * 8 + (lm >> 1) * 8);
#pragma unroll
        for (int z = 2; z >= 0; --z)
#pragma unroll
          for (int kk = 0; kk < TT / 16; ++kk)
#pragma unroll
            for (int i = 0; i < 4; ++i) mma(f[kk][i], a[kk][z], b[kk][i >> 1][(i & 1) * 2], b[kk][i >> 1][(i & 1) * 2 + 1]);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[j + i][e] = fmaf(whole, S[j + i][e], f[0][i][e] + f[1][i][e]);
      }
      if (any_bad) {
#pragma unroll
        for (int i = 0; i < 4; i += 2)
          if (bad[er - e0 + (i >> 1) * 8] < TT) {
#pragma unroll
            for (int j = 0; j < 2 * KT; ++j) S[j][i] = S[j][i + 1] = NAN;
          }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[buf]);           // this warp is done with the chunk's rows and weights
  }
  if (at_work) {
#pragma unroll
    for (int j = 0; j < 2 * KT; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int e = er + (i >> 1) * 8, d = j * 8 + gq * 2 + (i & 1);
        if (d < p.D) {
          if (e < V) p.state[(size_t)slot * p.slot_stride + ((size_t)h * p.D + d) * V + e] = S[j][i];
          else if (e < v_all) p.state_n[(size_t)slot * p.slot_stride + (size_t)h * p.D + d] = S[j][i];
        }
      }
  }
}

template <int D, int WARPS>
int launch(const ChunkParams& p, int entries, cudaStream_t stream) {
  using Shape = ChunkShape<D, WARPS>;
  auto kern = chunk_scan_kernel<D, WARPS>;
  static bool done[JV_MAX_DEVICES] = {};
  if (!jv_once_per_device(done, [&] {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Shape::SMEM) == cudaSuccess;
      }))
    return JV_ERR_UNSUPPORTED;
  const int cols = p.V + (p.state_n != nullptr ? 1 : 0);
  return jv_launch(kern, dim3(entries, p.heads, (cols + Shape::ET - 1) / Shape::ET), dim3(32 * WARPS + 32), Shape::SMEM, stream, p);
}

bool rows_of_16_bytes(const void* p, long long stride) { return ((uintptr_t)p & 15) == 0 && stride % 8 == 0; }
}  // namespace

// q, k, v: the first head's columns in rows of `.._stride` 16-bit elements (head h reads q and k at (h / per_group) * D, v at h * V);
// gates [n, heads, 4] float with nq = gates + 3 and state_n, or null with dt_raw (rows of dt_stride elements, [heads] used),
// dt_bias, a_log [heads] of w_dtype; out [n, heads * V]; state as for jv_state_scan; portions > 0: entries of one token
// are passed by, which leaves this many.  Taken for D up to 128 and V, both in steps of
// 8, with rows on 16-byte boundaries.
JV_EXPORT int jv_chunk_scan(const void* q, long long q_stride, const void* k, long long k_stride, const void* v, long long v_stride,
                            int per_group, float scale, float* gates, const void* dt_raw, long long dt_stride, const void* dt_bias,
                            const void* a_log, int w_dtype, float* out, float* state, long long slot_stride, float* state_n,
                            const int* cu_seqlens, const int* slots, int n_slots, int entries, int heads, int D, int V, int portions,
                            int* status, cudaStream_t stream) {
  if (entries == 0) return JV_OK;
  if (D < 8 || D > 128 || D % 8 || V < 8 || V % 8 || per_group < 1 || heads % per_group || heads > 65535 || entries < 0 ||
      !rows_of_16_bytes(q, q_stride) || !rows_of_16_bytes(k, k_stride) || !rows_of_16_bytes(v, v_stride) || w_dtype < 0 || w_dtype > 1 ||
      (gates == nullptr && (dt_raw == nullptr || state_n != nullptr)) || ((uintptr_t)gates & 7))
    return JV_ERR_UNSUPPORTED;
  ChunkParams p{(const bf16*)q, (const bf16*)k, (const bf16*)v, q_stride, k_stride, v_stride, per_group, scale, gates,
                (const bf16*)dt_raw, dt_stride, dt_bias, a_log, w_dtype, out, state, slot_stride, state_n,
                gates == nullptr ? nullptr : gates + 3, cu_seqlens, slots, n_slots, heads, D, V, portions, entries, status};
  if (portions > 0) entries = portions;
  // four warps share a block's scores; two where that alone leaves multiprocessors without a block
  const long long blocks = (long long)entries * heads * ((V + 63) / 64);
  if (blocks >= 148) {
    if (D <= 32) return launch<32, 4>(p, entries, stream);
    if (D <= 64) return launch<64, 4>(p, entries, stream);
    return launch<128, 4>(p, entries, stream);
  }
  if (D <= 32) return launch<32, 2>(p, entries, stream);
  if (D <= 64) return launch<64, 2>(p, entries, stream);
  return launch<128, 2>(p, entries, stream);
}
