// Paged causal attention of prompt portions over a latent cache on the 5th-generation tensor cores: ONE key/value head whose key
// is the whole cache row [dk] and whose value is the row's first dv elements, shared by all query heads (the mathematics of
// attn_latent_mma.cu, which keeps decoding, short portions and the sizes that this kernel does not take).
//
// Persistent blocks; work item = up to 128 rows = (token, query head) pairs x 256 of the value's columns (O of 128 x 256 and two
// tiles of scores fill tensor memory, so dv = 512 is two items that form the same scores).  Per tile of 128 keys:
//
//   queries    all of an item's (up to nine tiles of [128 rows][64 elements]) stay in shared memory
//   ring       16 KB stages [128 keys][64 elements] in the order in which the tensor cores take them: the key tiles of the next
//              128 keys, then the value tiles of these (the first elements of the same rows, copied a second time: to keep them
//              from the scores on would leave no stages for the next keys)
//   weights    lie where their scores lay: each of a row's two softmax threads reads its 64 columns and writes over them the 64
//              weights in bfloat16 and what that rounding took off, which meets the values in eight more steps.  (With the
//              rounded weights alone the error against 64 bits was up to 0.6 % above that of attn_latent_mma.cu, whose shorter
//              chunks round fewer of the largest weights.)
//   warp 0     producer;  warp 1  issues the products, and clears the value rows that no row of the item sees;  warps 2..9
//              softmax, two threads a row
//
// Bound by the turns of the ring: 13 stages for 128 keys of rows of 576 (213 KB), each a copy, its products and two barriers, for
// 5,500 clocks of products; the products are issued by one elected thread, which took 13 % off against `lane == 0`.  2,048 tokens
// of 16 heads, rows of 576, values of 512, a window of 1,024: 371 us with attn_latent_mma.cu, 179 here; 8,192 tokens without a
// window 6,570 and 2,808.
// Every wait on a barrier is bounded by a clock deadline and reports to the status word.
//
// Restrictions: bfloat16, dk up to 576 and dv up to 512 in multiples of 8, up to 128 query heads, page size a power of two from 8
// to 128.
#include "tcgen05.cuh"

#include <math.h>

namespace {

constexpr int ROWS = 128, BN = 128;
constexpr int STAGE_BYTES = 128 * 64 * 2;       // 128 rows of 64 bfloat16
constexpr int MAX_PIECES = 9;                   // tiles of a query or key row
constexpr int VALUE_TILES = 4;                  // tiles of 64 value columns in an item
constexpr int COLUMNS = VALUE_TILES * 64;
constexpr int TILES = 14;                       // of shared memory: an item's queries and the ring
constexpr int MAX_STAGES = TILES - 1;
constexpr int THREADS = 320;                    // producer warp, mma warp, 8 softmax warps
constexpr int SOFTMAX_THREADS = 256;
constexpr int TMEM_COLS = 512;                  // S0, then P0 in it: [0,128)  S1, P1: [128,256)  O: [256,512)
constexpr int TMEM_O = 256;
constexpr int MAX_LISTED = 16;                  // rounds whose item a block looks up once, for all roles
constexpr float LOG2E = 1.4426950408889634f;
constexpr uint32_t IDESC_PV0 = IDESC_PV & ~(0x3Fu << 17);      // without the number of columns

struct Params {
  __nv_bfloat16* out; int out_stride;
  const int* block_table; int table_width;
  const int* cu_seqlens; const int* start_pos; const int* work;
  int n_work, n_heads, dk, dv, pieces, stages, column_parts, page_size, num_pages, tokens_per_tile;
  int mask;                    // as one number (common.cuh, first_visible)
  float scale_log2;
  const float* sink;           // [n_heads] or null: exp(sink) counts once in the denominator
  int* status;
};

struct Shared {
  uint64_t q_full, q_free, full[MAX_STAGES], empty[MAX_STAGES];
  uint64_t s_full[2], p_full[2], o_done[2];
  uint64_t o_free;              // the softmax threads have read an item's output: the next item's may be written
  uint64_t drain;               // used only after a wait ran out
  uint32_t tmem_base;
  int failed;                   // a role gave up on a wait
  int armed_q, armed[MAX_STAGES];      // parity of the phase the producer armed last; -1: never
  int4 items[MAX_LISTED];       // the block's first items: entry, first row, first position, (part of the columns << 16 | tokens)
  float xch[2][128];            // a row's two softmax threads exchange their maxima (and at the end their sums)
};

struct Item {
  int entry, part, q_first;         // request of the batch, part of the value's columns, first row of the tile among all tokens
  int tokens_here, pos_first;       // tokens in the tile, position of the first
  int j_lo, j_hi;                   // keys [j_lo, j_hi) are visible to some row
  int t_lo, n_tiles;                // first key tile, key tiles
  int turn;                         // the tile that the item begins with

  // The j-th tile that the item takes.  Items begin at different tiles: starting all at the first one, they would ask the
  // L2 for the same few lines at the same time.  The order hangs on the item's position alone, not on the rest of the batch.
  __device__ __forceinline__ int tile(int j) const { return t_lo + (j + turn < n_tiles ? j + turn : j + turn - n_tiles); }
};

__global__ void __launch_bounds__(THREADS, 1) attn_latent_tcgen05_kernel(const __grid_constant__ CUtensorMap q_map,
                                                                         const __grid_constant__ CUtensorMap k_map,
                                                                         const Params p) {
  pdl_trigger();
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* q_s = base;                                   // [pieces][128 rows][128 B]
  unsigned char* r_s = q_s + p.pieces * STAGE_BYTES;           // [stages][128 keys][128 B]
  Shared* sh = reinterpret_cast<Shared*>(base + TILES * STAGE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int H = p.n_heads, stages = p.stages;
  const int n_items = p.n_work * p.column_parts, n_blocks = gridDim.x;
  pdl_wait();                           // queries, keys and values are the work of the kernels before this one

  // The items of this block: in round r the blocks take the items r G .. r G + G - 1 of the list ordered longest first (the
  // work list is in ascending order of a tile's first token, so from its end), in the order of their numbers in even rounds
  // and against it in odd ones.
  auto item_of_round = [&](int r) -> int {
    const int L = r * n_blocks + ((r & 1) ? n_blocks - 1 - (int)blockIdx.x : (int)blockIdx.x);
    return L < n_items ? L : -1;
  };
  const int n_rounds = (n_items + n_blocks - 1) / n_blocks;
  auto look_up = [&](int r) -> int4 {
    const int L = item_of_round(r);
    if (L < 0) return make_int4(0, 0, 0, 0);
    const int w = p.n_work - 1 - L / p.column_parts, part = L % p.column_parts;
    const int entry = p.work[2 * w], q_off = p.work[2 * w + 1];
    const int q_begin = p.cu_seqlens[entry];
    const int tokens = max(0, min(p.tokens_per_tile, p.cu_seqlens[entry + 1] - q_begin - q_off));
    return make_int4(entry, q_begin + q_off, p.start_pos[entry] + q_off, part << 16 | tokens);
  };
  auto load_item = [&](int r) -> Item {
    const int4 v = r < MAX_LISTED ? sh->items[r] : look_up(r);
    Item it;
    it.entry = v.x;
    it.q_first = v.y;
    it.pos_first = v.z;
    it.part = v.w >> 16;
    it.tokens_here = v.w & 0xffff;
    it.j_lo = first_visible(it.pos_first, p.mask);
    it.j_hi = it.pos_first + it.tokens_here;
    it.t_lo = it.j_lo / BN;
    it.n_tiles = it.tokens_here > 0 ? (it.j_hi + BN - 1) / BN - it.t_lo : 0;
    it.turn = it.n_tiles > 0 ? it.pos_first / p.tokens_per_tile % it.n_tiles : 0;
    return it;
  };
  // the first item with tiles from round r on; r becomes its round
  auto next_item = [&](int& r, Item& out) -> bool {
    for (; r < n_rounds; ++r) {
      out = load_item(r);
      if (out.n_tiles > 0) return true;
    }
    return false;
  };
  auto value_tiles = [&](const Item& it) -> int { return min(VALUE_TILES, (p.dv - it.part * COLUMNS + 63) / 64); };

  if (threadIdx.x == 0) {
    mbar_init(&sh->q_full, 1); mbar_init(&sh->q_free, 1); sh->armed_q = -1;
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sh->s_full[b], 1); mbar_init(&sh->p_full[b], SOFTMAX_THREADS); mbar_init(&sh->o_done[b], 1);
    }
    for (int s = 0; s < stages; ++s) { mbar_init(&sh->full[s], 1); mbar_init(&sh->empty[s], 1); sh->armed[s] = -1; }
    mbar_init(&sh->o_free, SOFTMAX_THREADS);
    mbar_init(&sh->drain, 1);
    sh->failed = 0;
    mbar_fence_init();
  }
  for (int r = threadIdx.x; r < min(n_rounds, MAX_LISTED); r += THREADS) sh->items[r] = look_up(r);
  __syncthreads();
  // the producer starts at once; the others wait until the second warp has its tensor memory
  if (warp >= 1) {
    if (warp == 1) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sh->tmem_base)), "r"(TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    TC_FENCE_BEFORE();
    asm volatile("bar.sync 6, 288;\n" ::: "memory");
    TC_FENCE_AFTER();
  }
  const uint32_t tmem = warp >= 1 ? sh->tmem_base : 0u;
  const uint32_t tmem_o = tmem + TMEM_O;

  if (warp == 0) {
    // ---------------------------------------------------------------- producer
    const int P = p.page_size, pages_per_tile = BN / P;
    const int q_bytes = 128 * H * p.tokens_per_tile;            // of one piece: a box of 64 d x heads x tokens
    bool ok = true;
    // page ids of a tile: lane i reads the i-th (a tile has at most 16 pages); NOT_NEEDED, or what the table says (-1: none)
    constexpr int NOT_NEEDED = -2;
    auto tile_pages = [&](const Item& it, int j) -> int {
      const int pi = it.tile(j) * pages_per_tile + lane;
      if (lane >= pages_per_tile || pi * P >= it.j_hi || (pi + 1) * P <= it.j_lo) return NOT_NEEDED;
      return pi < p.table_width ? p.block_table[(size_t)it.entry * p.table_width + pi] : -1;
    };
    int s_at = 0, s_ph = 0;             // the next stage and the parity of its phase
    // `count` stages with the rows that the lanes' pages hold of elements 64 first ..; a lane copies its own page's.  The
    // announcement need not come before the copies: the phase cannot complete before lane 0 has arrived.
    auto put_rows = [&](int first, int count, int pages, int n_pages) {
      for (int c = first; c < first + count; ++c) {
        ok = __all_sync(0xffffffffu, mbar_wait(&sh->empty[s_at], s_ph ^ 1)) && ok;
        if (ok) {
          uint64_t* bar = &sh->full[s_at];
          if (lane == 0) { sh->armed[s_at] = s_ph; mbar_expect_tx(bar, n_pages * P * 128); }
          if (pages >= 0) tma_load_3d(r_s + s_at * STAGE_BYTES + lane * P * 128, &k_map, c * 64, 0, pages, bar);
        }
        if (++s_at == stages) { s_at = 0; s_ph ^= 1; }
      }
    };
    auto put_queries = [&](const Item& it, int n) {
      if (ok && elect_one()) {
        ok = mbar_wait(&sh->q_free, (n & 1) ^ 1);
        if (ok) {
          sh->armed_q = n & 1;
          mbar_expect_tx(&sh->q_full, p.pieces * q_bytes);
          for (int c = 0; c < p.pieces; ++c) tma_load_3d(q_s + c * STAGE_BYTES, &q_map, c * 64, 0, it.q_first, &sh->q_full);
        }
      }
      ok = __all_sync(0xffffffffu, ok);
    };
    auto put_keys = [&](int pages, int n_pages) { put_rows(0, p.pieces, pages, n_pages); };
    auto put_values = [&](const Item& it, int pages, int n_pages) {
      put_rows(it.part * VALUE_TILES, value_tiles(it), pages, n_pages);
    };
    // what the table says -> pages to copy from (-1: none), with a report of those that should be there
    auto usable = [&](int said, int& n_pages) -> int {
      const bool there = said >= 0 && said < p.num_pages;
      if (said != NOT_NEEDED && !there) atomicOr(p.status, JV_STATUS_BAD_PAGE);
      n_pages = __popc(__ballot_sync(0xffffffffu, there));
      return there ? said : -1;
    };
    // the tiles of all items as one sequence; a tile's page ids are asked for two tiles before they are used
    struct At { Item it; int r, n, j; bool valid; };
    auto after = [&](const At& x) -> At {
      At y = x;
      if (!x.valid) return y;
      if (++y.j < x.it.n_tiles) return y;
      y.j = 0;
      ++y.n;
      ++y.r;
      y.valid = next_item(y.r, y.it);
      return y;
    };
    At cur;
    cur.r = cur.n = cur.j = 0;
    cur.valid = next_item(cur.r, cur.it);
    At nxt = after(cur);
    int n_pages = 0, n_pages_next = 0;
    int pages = usable(cur.valid ? tile_pages(cur.it, 0) : NOT_NEEDED, n_pages);
    int said_next = nxt.valid ? tile_pages(nxt.it, nxt.j) : NOT_NEEDED;
    if (cur.valid) {
      put_queries(cur.it, 0);
      put_keys(pages, n_pages);
    }
    while (cur.valid && ok) {
      const At next2 = after(nxt);
      const int said_next2 = next2.valid ? tile_pages(next2.it, next2.j) : NOT_NEEDED;
      const bool values_first = !nxt.valid || nxt.n != cur.n;   // an item's last values go before the next item's keys
      const int pages_next = usable(said_next, n_pages_next);
      if (values_first) put_values(cur.it, pages, n_pages);
      if (nxt.valid) {
        if (nxt.n != cur.n) put_queries(nxt.it, nxt.n);
        put_keys(pages_next, n_pages_next);
      }
      if (!values_first) put_values(cur.it, pages, n_pages);
      cur = nxt;
      nxt = next2;
      pages = pages_next;
      n_pages = n_pages_next;
      said_next = said_next2;
    }
    if (!ok && lane == 0) { atomicOr(p.status, JV_STATUS_WAIT_EXPIRED); sh->failed = 1; }
  } else if (warp == 1) {
    // -------------------------------------------------------------- mma issuer
    // The whole warp walks through the tiles; one thread takes a tile's stages of keys and issues the products.
    const uint64_t q_desc = desc_k_major(smem_u32(q_s)), k_desc = desc_k_major(smem_u32(r_s));
    const uint64_t v_desc = desc_mn_major(smem_u32(r_s), STAGE_BYTES);
    int s_at = 0, s_ph = 0;             // the next stage and the parity of its phase
    auto advance = [&](int count) {
      s_at += count;
      while (s_at >= stages) { s_at -= stages; s_ph ^= 1; }
    };
    auto wait = [&](uint64_t* bar, int parity) -> bool { return __all_sync(0xffffffffu, mbar_wait(bar, parity)); };
    auto issue_qk = [&](int n, int j, int n_tiles, int gt) -> bool {        // S[gt % 2] = sum_c Q_c K_c^T
      bool fine = true;
      if (elect_one()) {
        // the scores go where the weights of the tile before last lay: its product has to be complete
        if (gt >= 2) fine = mbar_wait(&sh->o_done[gt & 1], ((gt - 2) >> 1) & 1);
        if (j == 0 && fine) fine = mbar_wait(&sh->q_full, n & 1);
        const uint32_t tmem_s = tmem + (gt & 1) * 128;
        int s = s_at, ph = s_ph;
        for (int c = 0; c < p.pieces && fine; ++c) {
          fine = mbar_wait(&sh->full[s], ph);
          if (!fine) break;
          TC_FENCE_AFTER();
          const uint64_t q0 = q_desc + (uint64_t)((c * STAGE_BYTES) >> 4), k0 = k_desc + (uint64_t)((s * STAGE_BYTES) >> 4);
          // what lies past dk in the last piece is zero on both sides
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma(tmem_s, q0 + 2 * kk, k0 + 2 * kk, IDESC_QK, (c | kk) != 0);
          umma_commit(&sh->empty[s]);
          if (++s == stages) { s = 0; ph ^= 1; }
        }
        if (fine) {
          if (j == n_tiles - 1) umma_commit(&sh->q_free);       // the item's queries have been used for the last time
          umma_commit(&sh->s_full[gt & 1]);
        }
      }
      advance(p.pieces);
      return __all_sync(0xffffffffu, fine);
    };
    bool ok = true;
    int r = 0, n = 0, gt = 0;
    Item it, nx;
    bool have = next_item(r, it);
    if (have) ok = issue_qk(0, 0, it.n_tiles, 0);
    while (have && ok) {
      int rn = r + 1;
      const bool more = next_item(rn, nx);
      const int tiles = value_tiles(it);
      for (int j = 0; j < it.n_tiles && ok; ++j, ++gt) {
        const bool last = j + 1 == it.n_tiles;
        // the next scores while this tile's softmax runs (the next item's wait for its queries, which take this one's place)
        if (!last) ok = issue_qk(n, j + 1, it.n_tiles, gt + 1);
        if (!ok) break;
        const int key0 = it.tile(j) * BN, from = max(0, it.j_lo - key0), to = min(BN, it.j_hi - key0);   // rows with keys
        const int s0 = s_at;
        for (int c = 0; c < tiles && ok; ++c) {
          const int s = s_at;
          ok = wait(&sh->full[s], s_ph);
          advance(1);
          if (ok && (from > 0 || to < BN)) {
            // the value rows that no row of the item sees become zero (they may hold anything, and their weights are zero)
            for (int i = lane; i < BN * 8; i += 32)
              if (i / 8 < from || i / 8 >= to) *reinterpret_cast<uint4*>(r_s + s * STAGE_BYTES + i * 16) = make_uint4(0, 0, 0, 0);
            PROXY_FENCE();                                        // visible to the tensor core
            __syncwarp();
          }
        }
        if (!ok) break;
        if (!wait(&sh->p_full[gt & 1], (gt >> 1) & 1)) { ok = false; break; }
        // an item's first product overwrites the output of the item before it, which its softmax threads must have read
        if (j == 0 && n > 0 && !wait(&sh->o_free, (n - 1) & 1)) { ok = false; break; }
        if (elect_one()) {
          TC_FENCE_AFTER();
          // O += P V : 8 steps of 16 keys with the weights, 8 with what their rounding took off; P from tensor memory (8 columns
          // a step, the second 64 keys from column 64 on), two 8-row groups down V.  Value tiles in stages that follow one another go into one product (a product of 64 columns
          // takes as long as one of 128): two products where the ring begins anew between them
          const uint32_t tmem_p = tmem + (gt & 1) * 128;
          int c = 0;
          while (c < tiles) {
            const int s = s0 + c < stages ? s0 + c : s0 + c - stages, run = min(tiles - c, stages - s);
            const uint64_t v0 = v_desc + (uint64_t)((s * STAGE_BYTES) >> 4);
            const uint32_t idesc = IDESC_PV0 | ((uint32_t)(run * 64 >> 3) << 17);
#pragma unroll
            for (int kk = 0; kk < 16; ++kk)
              umma_a_tmem(tmem_o + c * 64, tmem_p + ((kk >> 2) & 1) * 64 + (kk >> 3) * 32 + (kk & 3) * 8, v0 + (kk & 7) * (2048 / 16), idesc,
                          (j | kk) != 0);
            for (int i = 0; i < run; ++i) umma_commit(&sh->empty[s + i]);
            c += run;
          }
          umma_commit(&sh->o_done[gt & 1]);
        }
        __syncwarp();
        if (ok && last && more) ok = issue_qk(n + 1, 0, nx.n_tiles, gt + 1);
      }
      it = nx;
      r = rn;
      have = more;
      ++n;
    }
    if (!ok && lane == 0) { atomicOr(p.status, JV_STATUS_WAIT_EXPIRED); sh->failed = 1; }
  } else {
    // ----------------------------------------------------------------- softmax
    // Two threads per row: warps 2..5 take the first 64 keys of a tile (and the first 128 columns of O), warps 6..9 the
    // other 64.  A warp reads the 32 TMEM lanes of its number modulo 4.
    const int quad = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row = quad * 32 + lane;                           // this thread's row of the tile
    const int t = row / H, head = row % H;
    const uint32_t lane_addr = (uint32_t)(quad * 32) << 16;
    const float sc = p.scale_log2;
    constexpr float LAZY = 8.f;
    bool ok = true;
    int gt = 0, r_next = 0;
    Item upcoming;
    bool more = next_item(r_next, upcoming);
    while (more) {
      const Item it = upcoming;
      ++r_next;
      more = next_item(r_next, upcoming);       // asked for while the current item runs
      const bool row_ok = t < it.tokens_here;
      const int pos = row_ok ? it.pos_first + t : -1;
      const int seen_from = row_ok ? first_visible(pos, p.mask) : 0;
      // m_ref is the reference that the exponentials are taken against.  It follows the true maximum lazily: only when the
      // maximum has grown by more than 2^8 (in the exponent) is O rescaled.
      float m_ref = -INFINITY, l_run = 0.f;
      const int last_from = first_visible(it.j_hi - 1, p.mask);   // the first key that the item's last token sees
      // A wait that runs out makes `ok` false for the whole warp; the loops then only keep their appointments at the named
      // barriers (so that nobody is left waiting there) and do no further work.
      for (int j = 0; j < it.n_tiles; ++j, ++gt) {
        if (ok) ok = mbar_wait(&sh->s_full[gt & 1], (gt >> 1) & 1);
        ok = __all_sync(0xffffffffu, ok);
        const uint32_t s_addr = tmem + lane_addr + (gt & 1) * 128 + half * 64;
        const int jt = it.tile(j);
        const int key0 = jt * BN + half * 64;                    // first key of this thread's 64
        const bool need_mask = jt * BN + BN - 1 > it.pos_first || jt * BN < last_from;   // block-uniform
        uint32_t sr[2][32];
        float my_max = -INFINITY;
        if (ok) {
          TC_FENCE_AFTER();
          tmem_ld32_issue(s_addr, sr[0]);
          tmem_ld32_issue(s_addr + 32, sr[1]);
          tmem_ld_wait();
          if (need_mask) {
            const int last = pos - key0, from = seen_from - key0;   // of this thread's 64 keys those from `from` to `last` count
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (c * 32 + i > last || c * 32 + i < from) sr[c][i] = __float_as_uint(-INFINITY);
          }
          float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 32; i += 2)
              mx[(i >> 1) & 3] = max3(mx[(i >> 1) & 3], __uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1]));
          my_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        }
        // the reference moves only if some score of the tile has outgrown it; only then do a row's two threads exchange maxima
        const bool outgrown = ok && my_max != -INFINITY && (m_ref == -INFINITY || (my_max - m_ref) * sc > LAZY);
        float alpha = 1.f;
        if (pair_barrier_or(quad, outgrown)) {
          sh->xch[half][row] = my_max;
          pair_barrier(quad);
          const float m_tile = fmaxf(sh->xch[0][row], sh->xch[1][row]);
          pair_barrier(quad);                                    // both have read before a later tile writes
          if (ok && m_tile != -INFINITY && (m_ref == -INFINITY || (m_tile - m_ref) * sc > LAZY)) {
            alpha = (m_ref == -INFINITY) ? 0.f : fast_exp2((m_ref - m_tile) * sc);
            m_ref = m_tile;
          }
        }
        const float m_scaled = (m_ref == -INFINITY) ? 0.f : m_ref * sc;
        // O is rescaled only if some row of this warp moved its reference; the previous P V must be complete then
        if (ok && j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
          ok = __all_sync(0xffffffffu, mbar_wait(&sh->o_done[(gt - 1) & 1], ((gt - 1) >> 1) & 1));
          if (ok) {
            TC_FENCE_AFTER();
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              float v[32];
              tmem_ld32(tmem_o + lane_addr + half * 128 + c * 32, v);
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] *= alpha;
              tmem_st32(tmem_o + lane_addr + half * 128 + c * 32, v);
            }
          }
        }
        if (!ok) continue;
        // weights: pairs of scores in packed 32-bit arithmetic, as bfloat16 pairs into 32 columns, and what the rounding
        // took off into 32 more
        {
          const uint64_t scale2 = pack2(sc, sc), neg_m2 = pack2(-m_scaled, -m_scaled);
          uint64_t sum2[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
          uint32_t pw[32], rest[32];
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int i = 0; i < 32; i += 2) {
              const uint64_t x2 = fma2(pack2(__uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1])), scale2, neg_m2);
              float x0, x1;
              unpack2(x2, x0, x1);
              const float p0 = fast_exp2(x0), p1 = fast_exp2(x1);
              sum2[(i >> 1) & 1] = add2(sum2[(i >> 1) & 1], pack2(p0, p1));
              const __nv_bfloat162 h2 = __floats2bfloat162_rn(p0, p1);
              const uint32_t bits = *reinterpret_cast<const uint32_t*>(&h2);
              pw[c * 16 + (i >> 1)] = bits;
              const __nv_bfloat162 l2 = __floats2bfloat162_rn(p0 - __uint_as_float(bits << 16), p1 - __uint_as_float(bits & 0xffff0000u));
              rest[c * 16 + (i >> 1)] = *reinterpret_cast<const uint32_t*>(&l2);
            }
          float sum[4];
          unpack2(sum2[0], sum[0], sum[1]);
          unpack2(sum2[1], sum[2], sum[3]);
          tmem_st32_bits(s_addr, pw);                            // over this thread's own scores
          tmem_st32_bits(s_addr + 32, rest);
          l_run = l_run * alpha + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
        }
        TC_FENCE_BEFORE();                                       // P is in tensor memory before the arrival
        mbar_arrive(&sh->p_full[gt & 1]);
      }
      // ---- the item's output: O / sum, each thread its 128 columns; the row's sum is the two threads' together
      const int g_last = gt - 1;
      sh->xch[half][row] = l_run;
      pair_barrier(quad);
      const float l_row = sh->xch[0][row] + sh->xch[1][row];
      pair_barrier(quad);                                        // both have read before the next item's first tile writes
      const bool got = ok && mbar_wait(&sh->o_done[g_last & 1], (g_last >> 1) & 1);
      float inv = row_ok ? 1.f / l_row : 0.f;
      if (p.sink != nullptr && row_ok && m_ref != -INFINITY) {
        // the sink joins the denominator: the row's sum stands against the reference m_ref * sc (an exponent of two)
        const float sk = p.sink[head] * LOG2E, mr = m_ref * sc, mx = fmaxf(mr, sk);
        const float e = fast_exp2(mr - mx);
        inv = e / (l_row * e + fast_exp2(sk - mx));
      }
      const int col0 = it.part * COLUMNS + half * 128;
      __nv_bfloat16* dst = p.out + (size_t)(it.q_first + t) * p.out_stride + (size_t)head * p.dv + col0;
      if (__all_sync(0xffffffffu, got)) {
        TC_FENCE_AFTER();
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          if (col0 + c * 32 >= p.dv) break;                      // the same for the whole warp
          float v[32];
          tmem_ld32(tmem_o + lane_addr + half * 128 + c * 32, v);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            uint4 pk;
            __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
            for (int e = 0; e < 4; ++e) h2[e] = __floats2bfloat162_rn(v[q * 8 + 2 * e] * inv, v[q * 8 + 2 * e + 1] * inv);
            if (row_ok && col0 + c * 32 + q * 8 < p.dv) *reinterpret_cast<uint4*>(dst + c * 32 + q * 8) = pk;
          }
        }
        TC_FENCE_BEFORE();
        mbar_arrive(&sh->o_free);                                // this thread has read its part of the output
      } else {
        ok = false;
      }
    }
    if (!ok && lane == 0) { atomicOr(p.status, JV_STATUS_WAIT_EXPIRED); sh->failed = 1; }
  }

  TC_FENCE_BEFORE();
  __syncthreads();
  if (sh->failed) {
    // a wait ran out: products already issued may still write tensor memory and copies already asked for still land in this
    // block's shared memory; both get a bounded time to finish before tensor memory is freed and the block ends
    if (warp == 1 && elect_one()) drain_products_after_failure(&sh->drain);
    if (warp == 0 && lane == 0) {
      if (sh->armed_q >= 0) drain_copies_after_failure(&sh->q_full, sh->armed_q);
      for (int s = 0; s < stages; ++s)
        if (sh->armed[s] >= 0) drain_copies_after_failure(&sh->full[s], sh->armed[s]);
    }
    __syncthreads();
  }
  if (warp == 1) {
    TC_FENCE_AFTER();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

constexpr size_t SMEM = (size_t)STAGE_BYTES * TILES + sizeof(Shared) + 1024;
static_assert(SMEM <= 227 * 1024, "shared memory");
}  // namespace

JV_EXPORT int jv_attn_latent_tcgen05_supports(int n_heads, int dk, int dv, int page_size) {
  return n_heads >= 1 && n_heads <= ROWS && dk >= 8 && dk % 8 == 0 && dk <= 64 * MAX_PIECES && dv >= 8 && dv % 8 == 0 && dv <= dk &&
         dv <= 2 * COLUMNS && page_size >= 8 && page_size <= BN && (page_size & (page_size - 1)) == 0;
}

// q: [n_tokens, q_stride] bfloat16, head h of a token at column h * dk; out: [n_tokens, out_stride], head h at h * dv; cache:
// [num_pages, page_size, dk]; work: [n_work, 2] (entry, first token of the tile), tiles of 128 / n_heads tokens, in ascending order
// of work; mask as one number; sink: [n_heads] floats or null.
JV_EXPORT int jv_attn_latent_tcgen05(const void* q, int q_stride, int n_tokens, void* out, int out_stride, const void* cache,
                                     const int* block_table, int table_width, const int* cu_seqlens, const int* start_pos,
                                     const int* work, int n_work, int n_heads, int dk, int dv, int page_size, int num_pages,
                                     float scale, int mask, const float* sink, int* status, cudaStream_t stream) {
  if (n_work == 0) return JV_OK;
  if (!jv_attn_latent_tcgen05_supports(n_heads, dk, dv, page_size) || (q_stride % 8) || (out_stride % 8) || ((uintptr_t)q % 16) ||
      ((uintptr_t)out % 16) || ((uintptr_t)cache % 16))
    return JV_ERR_UNSUPPORTED;
  auto fn = encode_fn();
  if (fn == nullptr) return JV_ERR_UNSUPPORTED;
  const int tokens = ROWS / n_heads;
  CUtensorMap q_map, k_map;
  const cuuint32_t es[3] = {1, 1, 1};
  {
    // queries: (d, head, token); a box is 64 d x heads x (128 / heads) tokens, up to 128 rows, head fastest.  What lies past
    // dk (in the last piece) and past the last token is filled with zeros
    const cuuint64_t dims[3] = {(cuuint64_t)dk, (cuuint64_t)n_heads, (cuuint64_t)n_tokens};
    const cuuint64_t strides[2] = {(cuuint64_t)dk * 2, (cuuint64_t)q_stride * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)n_heads, (cuuint32_t)tokens};
    if (fn(&q_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return JV_ERR_UNSUPPORTED;
  }
  {
    // cache: (d, slot, page); a box is 64 d of a page's rows
    const cuuint64_t dims[3] = {(cuuint64_t)dk, (cuuint64_t)page_size, (cuuint64_t)num_pages};
    const cuuint64_t strides[2] = {(cuuint64_t)dk * 2, (cuuint64_t)page_size * dk * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)page_size, 1};
    if (fn(&k_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(cache), dims, strides, box, es,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return JV_ERR_UNSUPPORTED;
  }
  Params p;
  p.out = (__nv_bfloat16*)out; p.out_stride = out_stride; p.block_table = block_table; p.table_width = table_width;
  p.cu_seqlens = cu_seqlens; p.start_pos = start_pos; p.work = work; p.n_work = n_work; p.n_heads = n_heads; p.dk = dk; p.dv = dv;
  p.pieces = (dk + 63) / 64; p.stages = TILES - p.pieces; p.column_parts = (dv + COLUMNS - 1) / COLUMNS;
  p.page_size = page_size; p.num_pages = num_pages; p.tokens_per_tile = tokens; p.mask = mask; p.scale_log2 = scale * LOG2E;
  p.sink = sink; p.status = status;
  static bool ready[JV_MAX_DEVICES];
  if (!jv_once_per_device(ready, [&] {
        return cudaFuncSetAttribute(attn_latent_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM) == cudaSuccess;
      }))
    return JV_ERR_UNSUPPORTED;
  // persistent blocks: one per multiprocessor (or per item, if there are fewer)
  static int sm_count[JV_MAX_DEVICES];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= JV_MAX_DEVICES) return JV_ERR_UNSUPPORTED;
  if (sm_count[dev] == 0 &&
      (cudaDeviceGetAttribute(&sm_count[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sm_count[dev] <= 0))
    sm_count[dev] = 148;
  const long long items = (long long)n_work * p.column_parts;
  const int blocks = items < sm_count[dev] ? (int)items : sm_count[dev];
  return jv_launch(attn_latent_tcgen05_kernel, dim3(blocks), dim3(THREADS), SMEM, stream, q_map, k_map, p);
}
