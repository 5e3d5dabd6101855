// Paged causal attention on CUDA cores with 32-bit arithmetic throughout: the kernel of
// the 32-bit path, and the fallback for head sizes that the tensor-core kernels do not
// take.  It serves prompt portions of any length (with earlier context in the cache),
// single decoded tokens, and decoded tokens split along the keys.
//
// Work item = (entry, first token of the tile); grid.y = kv head x head group;
// grid.z = key split (1 unless SPLIT).  The 16 rows of a tile are (token, query head)
// pairs of ONE kv head, so keys and values are read once for all query heads of the
// group: row m -> token q_off + m / heads_per_tile, head kv*G + hg*heads_per_tile +
// m % heads_per_tile.  Keys run over the entry's block table; key j is visible to a
// query at position p iff j <= p and (window == 0 or j > p - window or j < keep: the first `keep` tokens of a sequence may stay
// visible under a window; keys are counted as places in a run, common.cuh, KeyRun).  Softmax is the
// running (max, sum) form; scores, probabilities and the output sum are float.  Key rows (and queries) longer than
// `d_chunk` elements come through shared memory in pieces.
//
// SPLIT: split s covers the places [s*split_size, (s+1)*split_size) of the run of visible
// keys; it writes its unnormalised output sum and (max, sum) to `part_o`/`part_ml`;
// `attn_combine_kernel` merges the splits of a row in ascending order, so the result
// does not depend on what else is in the batch.
#include "mbarrier.cuh"
#include "scan.cuh"
#include <math.h>

namespace {
constexpr int BLOCK_M = 16;
constexpr int BLOCK_N = 32;
constexpr int THREADS = 128;
constexpr int MAX_STAGES = 4;      // chunks of keys whose rows have a place (vector form)

struct AttnParams {
  const void* q; int q_stride;
  void* out; int out_stride;
  float* part_o; float* part_ml;
  const void* k_cache; const void* v_cache;
  const int* block_table; int table_width;
  const int* cu_seqlens; const int* start_pos;
  const int* work;  // [n_work][2] = (entry, q_off)
  int n_q_heads, n_kv_heads, head_dim, v_dim, page_size, num_pages, window;
  float scale;
  int tokens_per_tile, heads_per_tile, n_head_groups, split_size, n_splits;
  int n_v_heads, v_row;      // value heads (group kv reads value head kv % n_v_heads) and elements of a cached value row
  int n_k_heads;             // key heads (group kv reads key head kv % n_k_heads)
  int d_chunk;               // elements of the key rows that are in shared memory at a time
  float out_scale;           // multiplies the heads' outputs
  int keep;                  // positions below this one stay visible under a window
  float score_cap;           // > 0: score <- cap * tanh(score / cap), after the scale
  int sigmoid;               // 1: the weight of a visible key is sigmoid(score + bias[query head]), not normalised over keys
  const float* bias;         // [n_q_heads] or null
  int out_f32;               // 1: `out` is float whatever the type of q and the cache
  const float* head_scale;   // [n_q_heads] or null: multiplies the scaled score of its head (a temperature per head)
  const float* dist_bias;    // [n_q_heads][n_dist] or null: added to the score of a key `pos - j` positions back; distances
  int n_dist;                //   of n_dist - 1 and more share the last row.  Neither `scale` nor `head_scale` touch it.
  const float* sink;         // [n_q_heads] or null (softmax): exp(sink) counts once in the denominator, with no value
  int* status;
};

template <typename T, bool SPLIT>
__global__ void __launch_bounds__(THREADS) attn_simt_kernel(const AttnParams p) {
  extern __shared__ float smem[];
  const int D = p.head_dim, DCH = p.d_chunk;
  const int DV = p.v_dim;                          // leading elements of a value row that are used (<= v_row)
  float* Qs = smem;                                // [BLOCK_M][DCH]
  float* Ks = Qs + BLOCK_M * DCH;                  // [BLOCK_N][DCH+1]
  float* Vs = Ks + BLOCK_N * (DCH + 1);            // [BLOCK_N][DV]
  float* Ss = Vs + BLOCK_N * DV;                   // [BLOCK_M][BLOCK_N]
  float* row_m = Ss + BLOCK_M * BLOCK_N;           // [BLOCK_M]
  float* row_l = row_m + BLOCK_M;                  // [BLOCK_M]
  float* row_alpha = row_l + BLOCK_M;              // [BLOCK_M]
  int* row_pos = (int*)(row_alpha + BLOCK_M);      // [BLOCK_M] absolute position, -1 = unused row

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int entry = p.work[2 * blockIdx.x], q_off = p.work[2 * blockIdx.x + 1];
  const int kv_head = blockIdx.y / p.n_head_groups, hg = blockIdx.y % p.n_head_groups;
  const int G = p.n_q_heads / p.n_kv_heads;
  const int q_begin = p.cu_seqlens[entry];
  const int q_len = p.cu_seqlens[entry + 1] - q_begin;
  const int ctx = p.start_pos[entry];
  const int tokens_here = min(p.tokens_per_tile, q_len - q_off);
  if (tokens_here <= 0) return;

  // visible key range of the tile
  const int pos_first = ctx + q_off, pos_last = ctx + q_off + tokens_here - 1;
  const KeyRun run(first_visible(pos_first, p.window), p.keep);
  int n_lo = 0, n_hi = run.places(pos_last + 1);  // places of the run, the second exclusive
  if (SPLIT) {
    n_lo = blockIdx.z * p.split_size;
    n_hi = min(n_hi, n_lo + p.split_size);
    if (n_lo >= n_hi) return;
  }

  const T* q = (const T*)p.q;
  const T* kc = (const T*)p.k_cache;
  const T* vc = (const T*)p.v_cache;

  // rows: positions and query vectors
  if (tid < BLOCK_M) {
    const int t = tid / p.heads_per_tile, hh = hg * p.heads_per_tile + tid % p.heads_per_tile;
    row_pos[tid] = (t < tokens_here && hh < G) ? ctx + q_off + t : -1;
    row_m[tid] = -INFINITY;
    row_l[tid] = p.sigmoid ? 1.f : 0.f;
    row_alpha[tid] = 1.f;
  }
  auto load_q = [&](int d0, int dn) {                // elements [d0, d0 + dn) of the tile's queries
    for (int idx = tid; idx < BLOCK_M * dn; idx += THREADS) {
      const int m = idx / dn, d = idx - m * dn;
      const int t = m / p.heads_per_tile, hh = hg * p.heads_per_tile + m % p.heads_per_tile;
      float v = 0.f;
      if (t < tokens_here && hh < G)
        v = to_f32(q[(size_t)(q_begin + q_off + t) * p.q_stride + (size_t)(kv_head * G + hh) * D + d0 + d]);
      Qs[m * DCH + d] = v;
    }
  };
  if (D <= DCH) load_q(0, D);                        // whole rows fit: once for all keys

  constexpr int DC = 4;  // output columns per thread: d = tid, tid + THREADS, ...  (v_dim <= 512)
  float acc[BLOCK_M][DC];
#pragma unroll
  for (int m = 0; m < BLOCK_M; ++m)
#pragma unroll
    for (int c = 0; c < DC; ++c) acc[m][c] = 0.f;
  __syncthreads();

  for (int n0 = n_lo; n0 < n_hi; n0 += BLOCK_N) {
    float s[4] = {0.f, 0.f, 0.f, 0.f};               // scores: thread (n = lane, rows warp*4 .. warp*4+3)
    for (int d0 = 0; d0 < D; d0 += DCH) {
      const int dn = min(DCH, D - d0);
      if (d0 > 0) __syncthreads();                     // the piece before has been read
      if (D > DCH) load_q(d0, dn);
      // ---- keys and values of this chunk into shared memory (one warp per key row)
      for (int n = warp; n < BLOCK_N; n += THREADS / 32) {
        const T* krow = nullptr;
        const T* vrow = nullptr;
        if (n0 + n < n_hi) {
          const int j = run.position(n0 + n);
          const int pi = j / p.page_size;
          const int page = pi < p.table_width ? p.block_table[(size_t)entry * p.table_width + pi] : -1;
          if (page < 0 || page >= p.num_pages) {
            if (lane == 0) atomicOr(p.status, JV_STATUS_BAD_PAGE);
          } else {
            const size_t slot = (size_t)page * p.page_size + (j % p.page_size);
            krow = kc + (slot * p.n_k_heads + kv_head % p.n_k_heads) * D + d0;
            vrow = vc + (slot * p.n_v_heads + kv_head % p.n_v_heads) * p.v_row;
          }
        }
        for (int d = lane; d < dn; d += 32) Ks[n * (DCH + 1) + d] = krow ? to_f32(krow[d]) : 0.f;
        if (d0 == 0)
          for (int d = lane; d < DV; d += 32) Vs[n * DV + d] = vrow ? to_f32(vrow[d]) : 0.f;
      }
      __syncthreads();
      const float* kr = Ks + lane * (DCH + 1);
      const float* q0 = Qs + (warp * 4) * DCH;
      for (int d = 0; d < dn; ++d) {
        const float kv = kr[d];
#pragma unroll
        for (int r = 0; r < 4; ++r) s[r] = fmaf(q0[r * DCH + d], kv, s[r]);
      }
    }

    {
      const int j = run.position(n0 + lane);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int m = warp * 4 + r;
        const int pos = row_pos[m];
        const bool vis = pos >= 0 && n0 + lane < n_hi && j <= pos && (j >= first_visible(pos, p.window) || j < p.keep);
        float sc = s[r] * p.scale;
        if (p.head_scale != nullptr || p.dist_bias != nullptr) {
          const int hq = min(hg * p.heads_per_tile + m % p.heads_per_tile, G - 1) + kv_head * G;
          if (p.head_scale != nullptr) sc *= p.head_scale[hq];
          if (p.dist_bias != nullptr && vis) sc += p.dist_bias[(size_t)hq * p.n_dist + min(pos - j, p.n_dist - 1)];
        }
        if (p.score_cap > 0.f) sc = p.score_cap * tanhf(sc / p.score_cap);
        if (p.sigmoid) {
          // ---- weights that do not depend on one another: no maximum, no sum
          const int hh = hg * p.heads_per_tile + m % p.heads_per_tile;
          const float b = (p.bias != nullptr && hh < G) ? p.bias[kv_head * G + hh] : 0.f;
          Ss[m * BLOCK_N + lane] = vis ? 1.f / (1.f + expf(-(sc + b))) : 0.f;
          continue;
        }
        if (!vis) sc = -INFINITY;
        // ---- running softmax for row m (this warp owns the row)
        const float m_old = row_m[m];
        const float m_new = fmaxf(m_old, warp_max(sc));
        float pr = 0.f, alpha = 1.f;
        if (m_new != -INFINITY) {
          pr = vis ? expf(sc - m_new) : 0.f;
          alpha = (m_old == -INFINITY) ? 0.f : expf(m_old - m_new);
        }
        const float psum = warp_sum(pr);
        Ss[m * BLOCK_N + lane] = pr;
        __syncwarp();
        if (lane == 0) {
          row_m[m] = m_new;
          row_l[m] = row_l[m] * alpha + psum;
          row_alpha[m] = alpha;
        }
      }
    }
    __syncthreads();

    // ---- output sum: thread owns columns d = tid + c*THREADS for all rows
#pragma unroll
    for (int c = 0; c < DC; ++c) {
      const int d = tid + c * THREADS;
      if (d < DV) {
#pragma unroll
        for (int m = 0; m < BLOCK_M; ++m) acc[m][c] *= row_alpha[m];
        for (int n = 0; n < BLOCK_N; ++n) {
          const float v = Vs[n * DV + d];
#pragma unroll
          for (int m = 0; m < BLOCK_M; ++m) acc[m][c] = fmaf(Ss[m * BLOCK_N + n], v, acc[m][c]);
        }
      }
    }
    __syncthreads();
  }

  // ---- write
#pragma unroll
  for (int c = 0; c < DC; ++c) {
    const int d = tid + c * THREADS;
    if (d >= DV) continue;
#pragma unroll
    for (int m = 0; m < BLOCK_M; ++m) {
      if (row_pos[m] < 0) continue;
      const int t = m / p.heads_per_tile, hh = hg * p.heads_per_tile + m % p.heads_per_tile;
      const int head = kv_head * G + hh;
      const size_t token = (size_t)(q_begin + q_off + t);
      if (SPLIT) {
        // rows of split launches are single tokens: index by work item
        const size_t slot = ((size_t)blockIdx.x * p.n_q_heads + head) * p.n_splits + blockIdx.z;
        p.part_o[slot * DV + d] = acc[m][c];
        if (d == 0) {
          p.part_ml[slot * 2] = row_m[m];
          p.part_ml[slot * 2 + 1] = row_l[m];
        }
      } else {
        float o = acc[m][c] / row_l[m];
        if (p.sink != nullptr) {          // the sink joins the denominator: rescaled to the larger of the two maxima
          const float sk = p.sink[head], mx = fmaxf(row_m[m], sk);
          const float e = expf(row_m[m] - mx);
          o = acc[m][c] * e / (row_l[m] * e + expf(sk - mx));
        }
        o *= p.out_scale;
        if (p.out_f32) ((float*)p.out)[token * p.out_stride + (size_t)head * DV + d] = o;
        else ((T*)p.out)[token * p.out_stride + (size_t)head * DV + d] = from_f32<T>(o);
      }
    }
  }
}

// The same for float rows of whole vectors: sizes in multiples of four, value sizes of 32 RPT, rows on 16-byte boundaries.  The
// arithmetic is that of the kernel above, term by term; what differs is that nothing waits for one thing at a time.  The places of
// BLOCK_N keys are looked up by a thread each, their rows are copied whole (a bulk copy a row: with cp.async of all threads the reads
// of shared memory behind them wait) `stages` - 1 chunks ahead, and shared memory is read four numbers at a time: four keys'
// elements serve 16 multiply-adds in the scores, and a thread holds RPT rows x 4 columns of the output.
// What bounds it is the latency of a chunk's phases.  203 tokens of 16 heads of 64 on 4: 82 us with the kernel above, 30.5 so.
template <int RPT, bool SPLIT>
__global__ void __launch_bounds__(THREADS) attn_vec_kernel(const AttnParams p, const int stages) {
  extern __shared__ __align__(16) float smem[];
  constexpr int DV = 32 * RPT, VLD = DV + 4, SLD = BLOCK_N + 4;
  const int D = p.head_dim, KLD = D + 4;
  float* Qs = smem;                                // [BLOCK_M][D]
  float* Ks = Qs + BLOCK_M * D;                    // [stages][BLOCK_N][KLD]
  float* Vs = Ks + stages * BLOCK_N * KLD;         // [stages][BLOCK_N][VLD]
  float* Ss = Vs + stages * BLOCK_N * VLD;         // [BLOCK_M][SLD]
  __shared__ float row_l[BLOCK_M], row_m[BLOCK_M], row_alpha[BLOCK_M];
  __shared__ uint64_t full[MAX_STAGES];
  pdl_trigger();
  if (threadIdx.x < MAX_STAGES) mbar_init(&full[threadIdx.x], 2 * BLOCK_N);
  if (threadIdx.x < MAX_STAGES) mbar_fence_init();
  pdl_wait();

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int entry = p.work[2 * blockIdx.x], q_off = p.work[2 * blockIdx.x + 1];
  const int kv_head = blockIdx.y / p.n_head_groups, hg = blockIdx.y % p.n_head_groups;
  const int G = p.n_q_heads / p.n_kv_heads;
  const int q_begin = p.cu_seqlens[entry];
  const int q_len = p.cu_seqlens[entry + 1] - q_begin;
  const int ctx = p.start_pos[entry];
  const int tokens_here = min(p.tokens_per_tile, q_len - q_off);
  if (tokens_here <= 0) return;
  const int pos_first = ctx + q_off, pos_last = ctx + q_off + tokens_here - 1;
  const KeyRun run(first_visible(pos_first, p.window), p.keep);
  int n_lo = 0, n_hi = run.places(pos_last + 1);
  if (SPLIT) {
    n_lo = blockIdx.z * p.split_size;
    n_hi = min(n_hi, n_lo + p.split_size);
    if (n_lo >= n_hi) return;
  }
  const float* q = (const float*)p.q;
  const float* kc = (const float*)p.k_cache + (size_t)(kv_head % p.n_k_heads) * D;
  const float* vc = (const float*)p.v_cache + (size_t)(kv_head % p.n_v_heads) * p.v_row;
  const size_t k_slot = (size_t)p.n_k_heads * D, v_slot = (size_t)p.n_v_heads * p.v_row;
  // where a thread's key of the chunk from place n0 on lies (-1: none there); threads 0 .. BLOCK_N - 1 bring keys, as many more values
  const int mine = tid & (BLOCK_N - 1);
  const bool brings = tid < 2 * BLOCK_N, values = tid >= BLOCK_N;
  auto look_up = [&](int n0) -> long long {
    if (!brings || n0 + mine >= n_hi) return -1;
    const int j = run.position(n0 + mine), pi = j / p.page_size;
    const int page = pi < p.table_width ? p.block_table[(size_t)entry * p.table_width + pi] : -1;
    if (page < 0 || page >= p.num_pages) { atomicOr(p.status, JV_STATUS_BAD_PAGE); return -1; }
    return (long long)page * p.page_size + (j - pi * p.page_size);
  };
  auto bring = [&](long long slot, int stage) {
    if (!brings) return;
    float* dst = values ? Vs + (stage * BLOCK_N + mine) * VLD : Ks + (stage * BLOCK_N + mine) * KLD;
    const int size = values ? DV : D;
    if (slot >= 0) {
      mbar_expect_tx(&full[stage], size * 4);
      bulk_copy(dst, values ? vc + slot * v_slot : kc + slot * k_slot, size * 4, &full[stage]);
    } else {
      for (int d = 0; d < size; d += 4) *reinterpret_cast<float4*>(dst + d) = make_float4(0.f, 0.f, 0.f, 0.f);
      mbar_arrive(&full[stage]);
    }
  };
  const int chunks = (n_hi - n_lo + BLOCK_N - 1) / BLOCK_N;
  __syncthreads();                                 // the barriers are there
  for (int c = 0; c < stages - 1 && c < chunks; ++c) bring(look_up(n_lo + c * BLOCK_N), c);
  long long next = look_up(n_lo + (stages - 1) * BLOCK_N);
  for (int i = tid; i < BLOCK_M * (D / 4); i += THREADS) {
    const int m = i / (D / 4), d = (i - m * (D / 4)) * 4;
    const int t = m / p.heads_per_tile, hh = hg * p.heads_per_tile + m % p.heads_per_tile;
    const bool live = t < tokens_here && hh < G;
    *reinterpret_cast<float4*>(Qs + m * D + d) =
        live ? *reinterpret_cast<const float4*>(q + (size_t)(q_begin + q_off + t) * p.q_stride + (size_t)(kv_head * G + hh) * D + d)
             : make_float4(0.f, 0.f, 0.f, 0.f);
  }

  // what this warp's four rows are; their running maximum and sum lie in every lane
  int pos[4], head[4], seen_from[4];
  float m_run[4], l_run[4], scale[4], bias[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int m = warp * 4 + r, t = m / p.heads_per_tile, hh = hg * p.heads_per_tile + m % p.heads_per_tile;
    pos[r] = t < tokens_here && hh < G ? ctx + q_off + t : -1;
    head[r] = kv_head * G + min(hh, G - 1);
    seen_from[r] = pos[r] >= 0 ? first_visible(pos[r], p.window) : 0;
    m_run[r] = -INFINITY;
    l_run[r] = p.sigmoid ? 1.f : 0.f;
    scale[r] = p.head_scale != nullptr ? p.head_scale[head[r]] : 1.f;
    bias[r] = p.bias != nullptr && hh < G ? p.bias[head[r]] : 0.f;
  }
  const int c4 = tid % (DV / 4) * 4, r0 = tid / (DV / 4) * RPT;      // this thread's columns and rows of the output
  float acc[RPT][4];
#pragma unroll
  for (int i = 0; i < RPT; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;

  for (int c = 0; c < chunks; ++c) {
    const int n0 = n_lo + c * BLOCK_N, buf = c % stages;
    // this chunk's rows have landed (or the block stops), the chunk before is done with
    if (!__syncthreads_and(mbar_wait(&full[buf], (c / stages) & 1))) {
      if (tid == 0) atomicOr(p.status, JV_STATUS_WAIT_EXPIRED);
      for (int e = c; e < min(c + stages - 1, chunks); ++e) drain_copies_after_failure(&full[e % stages], (e / stages) & 1);
      return;
    }
    if (c + stages - 1 < chunks) bring(next, (c + stages - 1) % stages);
    next = look_up(n0 + stages * BLOCK_N);
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    const float* kr = Ks + (buf * BLOCK_N + lane) * KLD;
    const float* q0 = Qs + warp * 4 * D;
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
      const float4 k = *reinterpret_cast<const float4*>(kr + d);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float4 x = *reinterpret_cast<const float4*>(q0 + r * D + d);
        s[r] = fmaf(x.x, k.x, s[r]); s[r] = fmaf(x.y, k.y, s[r]); s[r] = fmaf(x.z, k.z, s[r]); s[r] = fmaf(x.w, k.w, s[r]);
      }
    }
    const int j = run.position(n0 + lane);
    bool vis[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      vis[r] = pos[r] >= 0 && n0 + lane < n_hi && j <= pos[r] && (j >= seen_from[r] || j < p.keep);
      float sc = s[r] * p.scale;
      if (p.head_scale != nullptr) sc *= scale[r];
      if (p.dist_bias != nullptr && vis[r]) sc += p.dist_bias[(size_t)head[r] * p.n_dist + min(pos[r] - j, p.n_dist - 1)];
      if (p.score_cap > 0.f) sc = p.score_cap * tanhf(sc / p.score_cap);
      s[r] = sc;
    }
    if (p.sigmoid) {
#pragma unroll
      for (int r = 0; r < 4; ++r) Ss[(warp * 4 + r) * SLD + lane] = vis[r] ? 1.f / (1.f + expf(-(s[r] + bias[r]))) : 0.f;
      if (lane < 4) row_alpha[warp * 4 + lane] = 1.f;
    } else {
      float top[4], sum[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) top[r] = vis[r] ? s[r] : -INFINITY;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < 4; ++r) top[r] = fmaxf(top[r], __shfl_xor_sync(0xffffffffu, top[r], o));
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float m_new = fmaxf(m_run[r], top[r]);
        float pr = 0.f, alpha = 1.f;
        if (m_new != -INFINITY) {
          pr = vis[r] ? expf(s[r] - m_new) : 0.f;
          alpha = m_run[r] == -INFINITY ? 0.f : expf(m_run[r] - m_new);
        }
        Ss[(warp * 4 + r) * SLD + lane] = pr;
        sum[r] = pr;
        l_run[r] *= alpha;
        m_run[r] = m_new;
        if (lane == 0) row_alpha[warp * 4 + r] = alpha;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < 4; ++r) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], o);
#pragma unroll
      for (int r = 0; r < 4; ++r) l_run[r] += sum[r];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const float a = row_alpha[r0 + i];
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[i][c] *= a;
    }
    const float* vr = Vs + buf * BLOCK_N * VLD + c4;
#pragma unroll 2
    for (int n = 0; n < BLOCK_N; n += 4) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = *reinterpret_cast<const float4*>(vr + (n + u) * VLD);
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const float4 w = *reinterpret_cast<const float4*>(Ss + (r0 + i) * SLD + n);
        const float wu[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          acc[i][0] = fmaf(wu[u], v[u].x, acc[i][0]); acc[i][1] = fmaf(wu[u], v[u].y, acc[i][1]);
          acc[i][2] = fmaf(wu[u], v[u].z, acc[i][2]); acc[i][3] = fmaf(wu[u], v[u].w, acc[i][3]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
    if (lane == r) { row_m[warp * 4 + r] = m_run[r]; row_l[warp * 4 + r] = l_run[r]; }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < RPT; ++i) {
    const int m = r0 + i, t = m / p.heads_per_tile, hh = hg * p.heads_per_tile + m % p.heads_per_tile;
    if (t >= tokens_here || hh >= G) continue;
    const int head_of = kv_head * G + hh;
    if (SPLIT) {
      const size_t slot = ((size_t)blockIdx.x * p.n_q_heads + head_of) * p.n_splits + blockIdx.z;
      *reinterpret_cast<float4*>(p.part_o + slot * DV + c4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      if (c4 == 0) { p.part_ml[slot * 2] = row_m[m]; p.part_ml[slot * 2 + 1] = row_l[m]; }
      continue;
    }
    float* out = (float*)p.out + (size_t)(q_begin + q_off + t) * p.out_stride + (size_t)head_of * DV + c4;
    float e = 1.f, l = row_l[m];
    if (p.sink != nullptr) {                       // the sink joins the denominator: rescaled to the larger of the two maxima
      const float sk = p.sink[head_of], mx = fmaxf(row_m[m], sk);
      e = expf(row_m[m] - mx);
      l = l * e + expf(sk - mx);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) out[c] = (p.sink != nullptr ? acc[i][c] * e / l : acc[i][c] / l) * p.out_scale;
  }
}

// Merges the key splits of single-token rows.  grid = (n_work, n_q_heads).
template <typename T>
__global__ void attn_combine_kernel(const AttnParams p) {
  const int x = blockIdx.x, head = blockIdx.y;
  const int entry = p.work[2 * x];
  const int D = p.v_dim;
  const int pos = p.start_pos[entry];
  const KeyRun run(first_visible(pos, p.window), p.keep);
  constexpr int s_first = 0;
  int s_last = (run.places(pos + 1) - 1) / p.split_size;  // inclusive
  if (s_last >= p.n_splits) {  // the launch has too few splits for this length
    if (threadIdx.x == 0) atomicOr(p.status, JV_STATUS_BAD_ROW);
    s_last = p.n_splits - 1;
  }
  const size_t base = ((size_t)x * p.n_q_heads + head) * p.n_splits;
  if (p.sigmoid) {            // un-normalised weights: the splits' sums are added, in ascending order
    const size_t tok = (size_t)p.cu_seqlens[entry];
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
      float o = 0.f;
      for (int s = s_first; s <= s_last; ++s) o += p.part_o[(base + s) * D + d];
      o *= p.out_scale;
      if (p.out_f32) ((float*)p.out)[tok * p.out_stride + (size_t)head * D + d] = o;
      else ((T*)p.out)[tok * p.out_stride + (size_t)head * D + d] = from_f32<T>(o);
    }
    return;
  }
  float m_all = p.sink != nullptr ? p.sink[head] : -INFINITY;
  for (int s = s_first; s <= s_last; ++s) m_all = fmaxf(m_all, p.part_ml[(base + s) * 2]);
  float l_all = p.sink != nullptr ? expf(p.sink[head] - m_all) : 0.f;
  for (int s = s_first; s <= s_last; ++s)
    l_all += expf(p.part_ml[(base + s) * 2] - m_all) * p.part_ml[(base + s) * 2 + 1];
  const size_t token = (size_t)p.cu_seqlens[entry];
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    float o = 0.f;
    for (int s = s_first; s <= s_last; ++s)
      o += expf(p.part_ml[(base + s) * 2] - m_all) * p.part_o[(base + s) * D + d];
    const float r = o / l_all * p.out_scale;
    if (p.out_f32) ((float*)p.out)[token * p.out_stride + (size_t)head * D + d] = r;
    else ((T*)p.out)[token * p.out_stride + (size_t)head * D + d] = from_f32<T>(r);
  }
}

constexpr size_t MAX_SMEM = 227 * 1024;      // the largest size that is taken

size_t smem_bytes(int D, int DV) {
  return sizeof(float) * ((size_t)BLOCK_M * D + (size_t)BLOCK_N * (D + 1) + (size_t)BLOCK_N * DV +
                          BLOCK_M * BLOCK_N + 3 * BLOCK_M) + sizeof(int) * BLOCK_M;
}
// Shared memory of the vector form, and its stages: as many as fit, up to MAX_STAGES.
size_t vec_smem(int D, int DV, int stages) {
  return sizeof(float) * ((size_t)BLOCK_M * D + stages * BLOCK_N * (size_t)(D + 4 + DV + 4) + BLOCK_M * (BLOCK_N + 4));
}
int vec_stages(int D, int DV) {
  int stages = MAX_STAGES;
  while (stages > 2 && vec_smem(D, DV, stages) > (stages > 3 ? 100 * 1024 : MAX_SMEM - 2048)) --stages;
  return stages;
}
// Whether the vector form takes the case.
bool vec_takes(const AttnParams& p, int dtype) {
  const auto whole = [](const void* x) { return ((uintptr_t)x & 15) == 0; };
  return dtype == 0 && p.head_dim % 4 == 0 && (p.v_dim == 32 || p.v_dim == 64 || p.v_dim == 128 || p.v_dim == 256 || p.v_dim == 512) &&
         p.v_row % 4 == 0 && p.q_stride % 4 == 0 && whole(p.q) && whole(p.k_cache) && whole(p.v_cache) && whole(p.part_o) &&
         vec_smem(p.head_dim, p.v_dim, 2) <= MAX_SMEM - 2048;
}

template <int RPT, bool SPLIT>
int launch_vec(const AttnParams& p, dim3 grid, cudaStream_t stream) {
  auto kern = attn_vec_kernel<RPT, SPLIT>;
  static bool ready[JV_MAX_DEVICES];
  if (!jv_once_per_device(ready, [&] {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SMEM - 2048) == cudaSuccess;
      }))
    return JV_ERR_UNSUPPORTED;
  const int stages = vec_stages(p.head_dim, 32 * RPT);
  return jv_launch(kern, grid, dim3(THREADS), vec_smem(p.head_dim, 32 * RPT, stages), stream, p, stages);
}
template <bool SPLIT>
int launch_vec(const AttnParams& p, dim3 grid, cudaStream_t stream) {
  switch (p.v_dim) {
    case 32: return launch_vec<1, SPLIT>(p, grid, stream);
    case 64: return launch_vec<2, SPLIT>(p, grid, stream);
    case 128: return launch_vec<4, SPLIT>(p, grid, stream);
    case 256: return launch_vec<8, SPLIT>(p, grid, stream);
    default: return launch_vec<16, SPLIT>(p, grid, stream);
  }
}
}  // namespace

// Rows of a tile that hold tokens: 16 / heads_per_tile, with heads_per_tile = min(G, 16).
JV_EXPORT int jv_attn_simt_tokens_per_tile(int n_q_heads, int n_kv_heads) {
  const int G = n_q_heads / n_kv_heads;
  const int hpt = G < BLOCK_M ? G : BLOCK_M;
  return BLOCK_M / hpt;
}

// q: rows of `q_stride` elements (head h of token n at q[n*q_stride + h*D]); out: [n, out_stride];
// k_cache/v_cache: [num_pages, page_size, n_kv_heads, head_dim]; block_table: [entries, table_width];
// cu_seqlens: [entries+1]; start_pos: [entries] (tokens cached before this step); work:
// [n_work, 2] int32 (entry, first token of the tile within the entry's new tokens).
// v_dim: how many leading elements of a value row are used (0: all head_dim); out and part_o then have v_dim
// elements per head.  A cache whose values are the leading part of its keys passes the same tensor twice.
// jv_attn_simt_ex: keys and values of different sizes and head counts, capped scores, sigmoid weights, float output
// a temperature per head, a bias by distance, a sink in the softmax's denominator, fewer key heads than groups, an output
// scale
// (see AttnParams); jv_attn_simt is the plain softmax form with values shaped like the keys.
// n_splits == 0: every work item attends to its whole visible range and writes `out`.
// n_splits > 0: work items are single tokens; part_o [n_work*Hq*n_splits*D] and part_ml
// [n_work*Hq*n_splits*2] floats are scratch; a second launch merges into `out`.
JV_EXPORT int jv_attn_simt_ex(const void* q, int q_stride, void* out, int out_stride, int dtype,
                              float* part_o, float* part_ml, const void* k_cache, const void* v_cache,
                              const int* block_table, int table_width, const int* cu_seqlens,
                              const int* start_pos, const int* work, int n_work, int n_q_heads,
                              int n_kv_heads, int head_dim, int page_size, int num_pages, int window,
                              float scale, int split_size, int n_splits, int v_dim, int n_v_heads, int v_row,
                              float score_cap, int sigmoid, const float* bias, int out_f32, const float* head_scale,
                              const float* dist_bias, int n_dist, const float* sink, int n_k_heads, float out_scale,
                              int keep, int* status, cudaStream_t stream) {
  if (n_work == 0) return JV_OK;
  if ((dist_bias != nullptr && n_dist < 1) || (sink != nullptr && sigmoid)) return JV_ERR_UNSUPPORTED;
  if (v_row <= 0) v_row = head_dim;
  if (n_v_heads <= 0) n_v_heads = n_kv_heads;
  if (v_dim <= 0) v_dim = v_row;
  if (n_k_heads <= 0) n_k_heads = n_kv_heads;
  // whole key rows where they fit in shared memory beside the values, else pieces of 256 elements
  const int d_chunk = smem_bytes(head_dim, v_dim) <= 200 * 1024 ? head_dim : 256;
  if (head_dim < 1 || v_dim > v_row || v_dim > 512 || smem_bytes(d_chunk, v_dim) > MAX_SMEM || n_kv_heads < 1 ||
      n_q_heads % n_kv_heads != 0)
    return JV_ERR_UNSUPPORTED;
  AttnParams p;
  p.n_v_heads = n_v_heads; p.v_row = v_row; p.score_cap = score_cap; p.sigmoid = sigmoid ? 1 : 0; p.bias = bias;
  p.out_f32 = out_f32 ? 1 : 0; p.n_k_heads = n_k_heads; p.d_chunk = d_chunk; p.out_scale = out_scale;
  p.keep = window > 0 ? keep : 0;
  p.head_scale = head_scale; p.dist_bias = dist_bias; p.n_dist = n_dist; p.sink = sink;
  p.q = q; p.q_stride = q_stride; p.out = out; p.out_stride = out_stride;
  p.part_o = part_o; p.part_ml = part_ml; p.k_cache = k_cache; p.v_cache = v_cache;
  p.block_table = block_table; p.table_width = table_width; p.cu_seqlens = cu_seqlens;
  p.start_pos = start_pos; p.work = work; p.n_q_heads = n_q_heads; p.n_kv_heads = n_kv_heads;
  p.head_dim = head_dim; p.v_dim = v_dim; p.page_size = page_size; p.num_pages = num_pages; p.window = window;
  p.scale = scale; p.status = status;
  const int G = n_q_heads / n_kv_heads;
  p.heads_per_tile = G < BLOCK_M ? G : BLOCK_M;
  p.tokens_per_tile = n_splits > 0 ? 1 : BLOCK_M / p.heads_per_tile;
  p.n_head_groups = (G + p.heads_per_tile - 1) / p.heads_per_tile;
  p.split_size = split_size > 0 ? split_size : 1;
  p.n_splits = n_splits;
  const size_t smem = smem_bytes(d_chunk, v_dim);
  dim3 grid(n_work, n_kv_heads * p.n_head_groups, n_splits > 0 ? n_splits : 1);
  int rc = JV_OK;
  if (vec_takes(p, dtype)) {
    if (n_splits == 0) return launch_vec<false>(p, grid, stream);
    rc = launch_vec<true>(p, grid, stream);
    if (rc != JV_OK) return rc;
    attn_combine_kernel<float><<<dim3(n_work, n_q_heads), 64, 0, stream>>>(p);
    return jv_check_launch();
  }
  JV_DISPATCH_DTYPE(dtype, T, {
    if (n_splits > 0) {
      auto kern = attn_simt_kernel<T, true>;
      static bool ready[JV_MAX_DEVICES];
      if (!jv_once_per_device(ready, [&] {
            return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SMEM) == cudaSuccess;
          }))
        return JV_ERR_UNSUPPORTED;
      kern<<<grid, THREADS, smem, stream>>>(p);
      rc = jv_check_launch();
      if (rc == JV_OK) {
        attn_combine_kernel<T><<<dim3(n_work, n_q_heads), 64, 0, stream>>>(p);
        rc = jv_check_launch();
      }
    } else {
      auto kern = attn_simt_kernel<T, false>;
      static bool ready[JV_MAX_DEVICES];
      if (!jv_once_per_device(ready, [&] {
            return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SMEM) == cudaSuccess;
          }))
        return JV_ERR_UNSUPPORTED;
      kern<<<grid, THREADS, smem, stream>>>(p);
      rc = jv_check_launch();
    }
  });
  return rc;
}

JV_EXPORT int jv_attn_simt(const void* q, int q_stride, void* out, int out_stride, int dtype,
                           float* part_o, float* part_ml, const void* k_cache, const void* v_cache,
                           const int* block_table, int table_width, const int* cu_seqlens,
                           const int* start_pos, const int* work, int n_work, int n_q_heads,
                           int n_kv_heads, int head_dim, int page_size, int num_pages, int window,
                           float scale, int split_size, int n_splits, int v_dim, int* status,
                           cudaStream_t stream) {
  if (v_dim > head_dim) return JV_ERR_UNSUPPORTED;
  return jv_attn_simt_ex(q, q_stride, out, out_stride, dtype, part_o, part_ml, k_cache, v_cache, block_table,
                         table_width, cu_seqlens, start_pos, work, n_work, n_q_heads, n_kv_heads, head_dim, page_size,
                         num_pages, window, scale, split_size, n_splits, v_dim, n_kv_heads, head_dim, 0.f, 0, nullptr,
                         0, nullptr, nullptr, 0, nullptr, n_kv_heads, 1.f, 0, status, stream);
}
