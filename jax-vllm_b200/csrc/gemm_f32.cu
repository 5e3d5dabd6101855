// C[M, N] = A[M, K] * W[N, K]^T in 32-bit on the 5th-generation tensor cores: the matrix product of the 32-bit path, also used where a
// result must leave in 32-bit (logits) from 16-bit operands; batched, and grouped for routed experts.
//
// A 32-bit number is the sum of three 16-bit ones (x = hi + mid + lo, each the nearest to what is left; exactly), and a product of two
// is hi hi + (hi mid + mid hi) + (hi lo + mid mid + lo hi) but for 2^-25 of it: six products of 16-bit numbers, each exact in the tensor
// core.  Its sums cut where the CUDA cores' round, so they stay short: a sum of CHUNK = 32 k's starts from zero in tensor memory,
// smallest parts first, and is added to the running one, which registers hold, on the CUDA cores.
// (Against 64-bit sums, random operands, K = 1,024 to 2,816: relative error 0.9e-7 to 1.2e-7, where 32-bit multiply-adds in segments of
// 128 k's made 2.1e-7; with sums of 64 k's in tensor memory it was 3.2e-7.)
// 16-bit operands are one part.
// (A bfloat16 reaches as far down as a float: where all of a row lies below 2^-110 its third parts become too small for one, then the second.
// Relative error of rows of 7.7e-34 0.9e-7, of 2.4e-35 1.1e-6, of 1e-36 2.7e-5; such numbers beside larger ones lose nothing that counts.)
//
// The rows of W are the 128-row operand (a strip of 128 columns of C), the rows of A the narrow one, up to 128 of them: few rows
// waste nothing, and an element's sum is the same whatever M is.  (k is cut into up to six parts by N and K alone, so that strips times
// parts about fill the device.  Every part is summed with k ascending; the blocks of a tile's parts are a cluster, leave their sums in
// shared memory and add up each some of the tile, in ascending order.  By a kernel of their own, from memory, that took 5 us a product of 203 rows, 2.2 of one.
// With up to 16 rows, which wait for latency alone, a block pushes its sums to those that add them up, without a barrier between.)
//
// A block is one (strip, tile of rows, part), a pipeline of warps.  One brings 32 k's of the operands' rows with TMA, RAW chunks ahead.
// Two groups of four cut them, a chunk each in turn.  The parts of W go to tensor memory, a thread a row: through shared memory their
// stores and the tensor cores' reading them for each part of A again were half of a chunk's traffic for few rows.  The parts of A go to
// shared memory (up to 16 rows: two warps of their own cut them) in 8 x 16 byte blocks as the tensor cores read them without a swizzle
// (eight rows of a block follow one another, so that a warp's stores are 512 bytes in a row).  One warp issues the products into one of the accumulators, and eight more (four where
// the rows of A are few) add another to their registers, a thread a row of W and half of the rows of A.  What each warp does of a chunk
// is a chain of latencies longer than the products, so every role is a warp of its own (128 columns of
// 148 multiprocessors each, clocks a chunk: 128 rows 2,030 with eight warps that brought, cut and eight that issued and added, 1,260 so;
// 16 rows 1,440 and 1,010, of which the products are 400).  Per chunk a cutting warp takes 250 to 310 clocks for the 32 k's of W, 130 for
// eight rows of A, and some 200 for its waits.
// Rows that TMA cannot address (not on 16-byte boundaries) are loaded by the warps that cut them.
// Every wait on a barrier is bounded by a clock deadline and reports to the status word.
//
// An output that is no number (an infinity among the operands, whose parts are none, or a sum past the largest) is formed again on
// the CUDA cores.
//
// Measured, model of width 1,024, two layers, 32-bit: 203 tokens, eight products 0.68 ms with 8 x 8 outputs a thread in multiply-adds on
// the CUDA cores and 0.147 so (400 tokens 0.277), the head (one row, 32,000 columns) 26 and 29.6 us.  A product of one row takes
// 0.5 to 2 us longer than multiply-adds did (N = 1,024 4.8 us against 4.3, 4,256 7.9 against 5.8; 16 rows 5.3 against 13.0 and 8.6 against 13.8),
// which a sum that is the same whatever M is has to bear; it was 1.5 to 3 us before few rows had their A cut and their sums pushed as above.
// Grouped, 16 experts of 2,048 x 1,024 and 1,024 x 512, both products: 4 tokens of two choices 224 us on the CUDA cores and 37 so,
// 200 tokens 280 and 105.
#include "tcgen05.cuh"

namespace {
constexpr int BM = 128, CHUNK = 32, MAX_ROWS = 128;     // rows of A of a block
constexpr int CUTTERS = 8, GROUP = CUTTERS / 2;        // warps that cut, of a group of them
constexpr int GROUP_BYTES = 8 * CHUNK * 2;             // eight rows of a chunk in one 16-bit part: four blocks of 8 rows x 16 bytes
constexpr int LEAST_PART = 64, MAX_PARTS = 6;          // k's of a part; the parts of a tile are one cluster
constexpr int GROUPED_AT_ONCE = 4;                     // tiles of experts that k's parts are cut for (how many there are, hangs on the tokens)
constexpr int MAX_RAW = 6, MAX_STAGES = 4, MAX_ACCS = 4;

struct Params {
  const void* A; const void* W; void* C;
  int lda, ldw, ldc, M, N, K;
  size_t a_batch, w_batch, c_batch;                    // independent products: grid.y of them, operands this far apart
  int a_vec, w_vec;                                    // four elements a load along k
  int strips, parts, part_k, row_tile;                 // row_tile: rows of A of a block, a multiple of 16
  int w_fixed;                                         // no kernel before this one writes W: it is asked for before they have finished
  int* status;
  // grouped (routed experts): the expert of every tile of rows of A (-1: nothing to do), the token of every row (-1: nobody's, left alone)
  const int *tile_expert, *row_token;
  int gelu;
};

struct Shared {
  uint64_t w_full[MAX_RAW], a_full[MAX_RAW], raw_empty[MAX_RAW];      // chunks as they are in memory: rows of W, of A, free places
  uint64_t full[MAX_STAGES], empty[MAX_STAGES], acc_full[MAX_ACCS], acc_empty[MAX_ACCS];       // chunks in parts; their sums
  uint64_t pushed;                                     // what the blocks of the cluster add up of this block's share (few rows)
  uint64_t drain;                                      // used only after a wait ran out
  uint32_t tmem_base;
  int failed;
};

// Descriptor of a K-major operand without a swizzle: blocks of 8 rows x 16 bytes, the next 16 bytes of k 128 bytes further, the next
// eight rows GROUP_BYTES.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(GROUP_BYTES >> 4) << 32) | ((uint64_t)1 << 46);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&a)[4], const uint32_t (&b)[4]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n"
               ::"r"(taddr), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]) : "memory");
}
// Every thread of every block of the cluster; what they wrote before is seen by all after.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// The same in two halves and without a word about what was written: this block reads no other any more (or may be written to) ... and is
// read by none (and may write to others).
__device__ __forceinline__ void cluster_leave() { asm volatile("barrier.cluster.arrive.relaxed.aligned;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_left() { asm volatile("barrier.cluster.wait.aligned;\n" ::: "memory"); }
// 16 bytes of block `rank` of the cluster, at its address of what this block has at `addr`.
__device__ __forceinline__ float4 cluster_load(uint32_t addr, int rank) {
  float4 v;
  asm volatile("{\n.reg .b32 a;\nmapa.shared::cluster.u32 a, %4, %5;\nld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [a];\n}\n"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr), "r"(rank) : "memory");
  return v;
}
// x into block `rank` of the cluster, at its address of what this block has at `addr`; its barrier at `bar` counts the four bytes.
__device__ __forceinline__ void cluster_push(uint32_t addr, uint64_t* bar, float x, int rank) {
  asm volatile("{\n.reg .b32 a, b;\nmapa.shared::cluster.u32 a, %0, %3;\nmapa.shared::cluster.u32 b, %1, %3;\n"
               "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [a], %2, [b];\n}\n"
               ::"r"(addr), "r"(smem_u32(bar)), "r"(__float_as_uint(x)), "r"(rank) : "memory");
}
// As mbar_wait, for what the other blocks have pushed.
__device__ __forceinline__ bool wait_pushed(uint64_t* bar) {
  const long long deadline = clock64() + JV_WAIT_CYCLES;
  uint32_t done;
  do {
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(smem_u32(bar)) : "memory");
  } while (!done && clock64() < deadline);
  return done != 0;
}
__device__ __forceinline__ uint32_t pack_bf16(float x, float y) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// What a lane has of a row: eight consecutive k's, as they are in memory; zeros past k_end or for a row that is not there.
template <typename T> struct Eight;
template <> struct Eight<float> {
  static constexpr int PARTS = 3;
  float v[8];
  __device__ __forceinline__ void load(const float* __restrict__ row, bool live, int k, int k_end, bool vec) {
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      if (live && vec && k + h + 4 <= k_end) {
        const float4 x = __ldg(reinterpret_cast<const float4*>(row + k + h));
        v[h] = x.x; v[h + 1] = x.y; v[h + 2] = x.z; v[h + 3] = x.w;
      } else {
#pragma unroll
        for (int i = h; i < h + 4; ++i) v[i] = live && k + i < k_end ? __ldg(row + k + i) : 0.f;
      }
    }
  }
  // from a tile of rows of 128 bytes as TMA leaves it (128-byte swizzle)
  static constexpr int ROW_BYTES = CHUNK * 4;
  static constexpr CUtensorMapDataType MAP_TYPE = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  static constexpr CUtensorMapSwizzle MAP_SWIZZLE = CU_TENSOR_MAP_SWIZZLE_128B;
  __device__ __forceinline__ void read(const unsigned char* tile, int row, int kb) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4 x = *reinterpret_cast<const float4*>(tile + row * ROW_BYTES + (((2 * kb + h) ^ (row & 7)) << 4));
      v[4 * h] = x.x; v[4 * h + 1] = x.y; v[4 * h + 2] = x.z; v[4 * h + 3] = x.w;
    }
  }
  __device__ __forceinline__ void cut(uint32_t (&part)[3][4]) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float x = v[2 * i], y = v[2 * i + 1];
      const uint32_t hi = part[0][i] = pack_bf16(x, y);
      x -= __uint_as_float(hi << 16);
      y -= __uint_as_float(hi & 0xffff0000u);
      const uint32_t mid = part[1][i] = pack_bf16(x, y);
      part[2][i] = pack_bf16(x - __uint_as_float(mid << 16), y - __uint_as_float(mid & 0xffff0000u));
    }
  }
};
template <> struct Eight<__nv_bfloat16> {
  static constexpr int PARTS = 1;
  uint2 v[2];
  __device__ __forceinline__ void load(const __nv_bfloat16* __restrict__ row, bool live, int k, int k_end, bool vec) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (live && vec && k + 4 * h + 4 <= k_end) {
        v[h] = __ldg(reinterpret_cast<const uint2*>(row + k + 4 * h));
      } else {
        const unsigned short* r = reinterpret_cast<const unsigned short*>(row);
        uint32_t e[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) e[i] = live && k + 4 * h + i < k_end ? __ldg(r + k + 4 * h + i) : 0u;
        v[h] = make_uint2(e[0] | e[1] << 16, e[2] | e[3] << 16);
      }
    }
  }
  static constexpr int ROW_BYTES = CHUNK * 2;
  static constexpr CUtensorMapDataType MAP_TYPE = CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  static constexpr CUtensorMapSwizzle MAP_SWIZZLE = CU_TENSOR_MAP_SWIZZLE_64B;
  __device__ __forceinline__ void read(const unsigned char* tile, int row, int kb) {
    const uint4 x = *reinterpret_cast<const uint4*>(tile + row * ROW_BYTES + ((kb ^ ((row >> 1) & 3)) << 4));
    v[0] = make_uint2(x.x, x.y); v[1] = make_uint2(x.z, x.w);
  }
  __device__ __forceinline__ void cut(uint32_t (&part)[1][4]) const {
    part[0][0] = v[0].x; part[0][1] = v[0].y; part[0][2] = v[1].x; part[0][3] = v[1].y;
  }
};

// An output element on the CUDA cores.
template <typename TA, typename TW>
__device__ __noinline__ float plain_sum(const TA* __restrict__ a, const TW* __restrict__ w, int K) {
  float s = 0.f;
  for (int k = 0; k < K; ++k) s = fmaf(to_f32(a[k]), to_f32(w[k]), s);
  return s;
}
__device__ __forceinline__ bool is_number(float x) { return fabsf(x) <= 3.402823466e38f; }

template <bool TMA, int NB, typename TA, typename TW> struct Shape {
  static constexpr int PA = Eight<TA>::PARTS, PW = Eight<TW>::PARTS;
  static constexpr int ADDERS = NB <= 16 ? 4 : 8, A_CUTTERS = TMA && NB <= 16 ? NB / 8 : 0;      // (few rows: warps of their own cut A)
  static constexpr int ISSUER = CUTTERS + ADDERS + A_CUTTERS, BRINGER = ISSUER + 1, THREADS = 32 * (BRINGER + 1);
  static constexpr int ACCS = NB <= 64 ? 4 : 2, STAGES = 4;       // accumulators, chunks in parts
  static constexpr int A_PART = NB / 8 * GROUP_BYTES, STAGE = PA * A_PART;
  static constexpr int W_RAW = BM * Eight<TW>::ROW_BYTES, A_RAW = (NB * Eight<TA>::ROW_BYTES + 1023) / 1024 * 1024;
  static constexpr int RAW = !TMA ? 1 : NB <= 16 ? 5 : NB <= 64 ? 6 : 4, RAW_STAGE = W_RAW + A_RAW;
  // Few rows: the parts' sums of the columns that a block adds up are pushed to it, behind the ring, which it may still be using.
  static constexpr bool PUSH = TMA && NB <= 16;
  static constexpr int RING = (TMA ? RAW * RAW_STAGE : 0) + STAGES * STAGE, SUMS = 2 * NB * BM * 4 + MAX_PARTS * 16;     // the block's sums, and of all parts those that it adds up, lie over the ring
  static constexpr int HERE = PUSH ? (BM / 4 + MAX_PARTS - 1) * NB * 16 : 0;
  static constexpr int SMEM = (PUSH ? RING + HERE : RING > SUMS ? RING : SUMS) + (int)sizeof(Shared) + 1024;
  static_assert(!PUSH || 2 * (SMEM + 1024) <= 228 * 1024, "two blocks a multiprocessor");
  static constexpr int A_GROUPS = (NB / 8 + GROUP - 1) / GROUP;   // of eight rows that a warp cuts
  // tensor memory: accumulators of NB columns, then stages of 16 columns (two k's each) a part of W
  static constexpr int TMEM_COLS = NB <= 16 ? 256 : 512, W_COLS = 16 * PW;
  static_assert(ACCS * NB + STAGES * W_COLS <= TMEM_COLS, "tensor memory");
};

// A place in a ring of N and the parity of its phase.
template <int N> struct Place {
  int i = 0, phase = 0;
  __device__ __forceinline__ void next() {
    if (++i == N) { i = 0; phase ^= 1; }
  }
};

// NB: rows of A that a block has room for
template <bool TMA, int NB, typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(Shape<TMA, NB, TA, TW>::THREADS, NB <= 16 ? 2 : 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map, const Params p) {
  using S = Shape<TMA, NB, TA, TW>;
  constexpr int PA = S::PA, PW = S::PW, ACCS = S::ACCS, STAGES = S::STAGES, RAW = S::RAW;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* raw = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);     // [RAW][W rows, A rows]
  unsigned char* stages = raw + (TMA ? RAW * S::RAW_STAGE : 0);
  float* sums = reinterpret_cast<float*>(raw);         // [row of A][row of W], once all is summed
  Shared* sh = reinterpret_cast<Shared*>(raw + (S::PUSH ? S::RING + S::HERE : S::RING > S::SUMS ? S::RING : S::SUMS));
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  // the parts of one tile are a cluster
  const int m_tiles = (p.M + p.row_tile - 1) / p.row_tile;
  const int part = blockIdx.x % p.parts, m0 = blockIdx.x / p.parts % m_tiles * p.row_tile, n0 = blockIdx.x / p.parts / m_tiles * BM;
  const int rows = min(p.row_tile, p.M - m0), rows16 = (rows + 15) / 16 * 16;
  const int k0 = part * p.part_k, k_end = min(p.K, k0 + p.part_k), chunks = (k_end - k0 + CHUNK - 1) / CHUNK;
  // PUSH: this block adds up `quads` fours of the tile's columns (the last block fewer), from `quad0` on; its room is [part][row][quads]
  const int quads = (BM / 4 + p.parts - 1) / p.parts, quad0 = part * quads, my_quads = max(0, min(quads, BM / 4 - quad0));
  float* here = reinterpret_cast<float*>(raw + S::RING);
  const TA* A = (const TA*)p.A + blockIdx.y * p.a_batch + (size_t)m0 * p.lda;
  int wb = blockIdx.y;                                 // which of the matrices W
  if (p.tile_expert != nullptr) {                      // found out by the kernels before this one; the same for the whole cluster
    pdl_wait();
    wb = p.tile_expert[m0 / p.row_tile];
    if (wb < 0) return;
  }
  const TW* W = (const TW*)p.W + wb * p.w_batch + (size_t)n0 * p.ldw;
  const int early = TMA ? min(RAW, chunks) : 0;
  auto bring_w = [&](int c, int s) {
    mbar_expect_tx(&sh->w_full[s], BM * Eight<TW>::ROW_BYTES);
    tma_load_3d(raw + s * S::RAW_STAGE, &w_map, k0 + c * CHUNK, n0, wb, &sh->w_full[s]);
  };
  if (TMA && threadIdx.x == 0) {
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(&w_map) : "memory");
    asm volatile("prefetch.tensormap [%0];\n" ::"l"(&a_map) : "memory");
  }
  if (warp == S::BRINGER) {
    constexpr int CUT = GROUP + S::A_CUTTERS;          // warps that cut a chunk
    for (int i = lane; i < MAX_RAW; i += 32) { mbar_init(&sh->w_full[i], 1); mbar_init(&sh->a_full[i], 1); mbar_init(&sh->raw_empty[i], CUT); }
    for (int i = lane - MAX_RAW; i >= 0 && i < MAX_STAGES; i += 32) { mbar_init(&sh->full[i], CUT); mbar_init(&sh->empty[i], 1); }
    for (int i = lane - MAX_RAW - MAX_STAGES; i >= 0 && i < MAX_ACCS; i += 32) { mbar_init(&sh->acc_full[i], 1); mbar_init(&sh->acc_empty[i], S::ADDERS); }
    if (lane == 31) {
      mbar_init(&sh->drain, 1);
      sh->failed = 0;
      if (S::PUSH) {
        mbar_init(&sh->pushed, 1);
        mbar_fence_init();
        if (p.parts > 1) mbar_expect_tx(&sh->pushed, p.parts * rows * my_quads * 16);
      }
    }
    mbar_fence_init();
    __syncwarp();
    if (p.w_fixed && elect_one())
      for (int c = 0; c < early; ++c) bring_w(c, c);
    __syncwarp();
  }
  if (warp == S::ISSUER) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sh->tmem_base)), "n"(S::TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  TC_FENCE_BEFORE();
  __syncthreads();
  TC_FENCE_AFTER();
  // The others may push: the barrier's set-up is fenced above.  (With a release of everything before, which waits for the copies under
  // way, the arrival took 1,900 clocks.)
  if (S::PUSH && p.parts > 1) cluster_leave();
  pdl_trigger();                                       // not before this block has its tensor memory
  const uint32_t tmem = __shfl_sync(0xffffffffu, sh->tmem_base, 0), tmem_w = tmem + ACCS * NB;
  int brought = 0;                                     // chunks that have been asked for, in the thread that does it
  bool ok = true;

  if (warp == S::BRINGER) {
    // ------------------------------------------------------------- rows as they are: zeros past K, N and M
    if (TMA && elect_one()) {
      auto bring_a = [&](int c, int s) {
        mbar_expect_tx(&sh->a_full[s], p.row_tile * Eight<TA>::ROW_BYTES);
        tma_load_3d(raw + s * S::RAW_STAGE + S::W_RAW, &a_map, k0 + c * CHUNK, m0, blockIdx.y, &sh->a_full[s]);
      };
      pdl_wait();
      for (int c = 0; c < early; ++c) {
        if (!p.w_fixed) bring_w(c, c);
        bring_a(c, c);
      }
      brought = early;
      Place<RAW> to;
      for (; brought < chunks; ++brought, to.next()) {
        if (!(ok = mbar_wait(&sh->raw_empty[to.i], to.phase))) break;
        bring_w(brought, to.i);
        bring_a(brought, to.i);
      }
    }
  } else if (warp == S::ISSUER) {
    // ------------------------------------------------------------- products
    // (the whole warp takes every turn and one elected thread issues)
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(rows16 >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    const uint64_t a_desc = smem_desc(smem_u32(stages));
    Place<STAGES> at;
    Place<ACCS> into;
    for (int c = 0; c < chunks; ++c) {
      ok = __all_sync(0xffffffffu, mbar_wait(&sh->acc_empty[into.i], into.phase ^ 1) && mbar_wait(&sh->full[at.i], at.phase));
      if (!ok) break;
      TC_FENCE_AFTER();
      const uint64_t a = a_desc + (uint64_t)((at.i * S::STAGE) >> 4);
      const uint32_t w = tmem_w + at.i * S::W_COLS, d = tmem + into.i * NB;
      constexpr int MOST = PW + PA - 2 < 2 ? PW + PA - 2 : 2;
      if (elect_one()) {
        bool zero = true;
#pragma unroll
        for (int sum = MOST; sum >= 0; --sum)                       // parts x of W and y of A with x + y = sum
#pragma unroll
          for (int kk = 0; kk < CHUNK / 16; ++kk)                   // 16 k's are two blocks of 16 bytes: 256 bytes on
#pragma unroll
            for (int x = 0; x < PW; ++x) {
              const int y = sum - x;
              if (y < 0 || y >= PA) continue;
              umma_a_tmem(d, w + x * 16 + kk * 8, a + ((y * S::A_PART + kk * 256) >> 4), idesc, zero ? 0u : 1u);
              zero = false;
            }
        umma_commit(&sh->empty[at.i]);
        umma_commit(&sh->acc_full[into.i]);
      }
      __syncwarp();
      at.next();
      into.next();
    }
  } else if (warp < CUTTERS) {
    // ------------------------------------------------------------- rows into parts
    const int r = lane & 7, kb = lane >> 3, quad = warp & 3;        // of A: a row and which eight k's; the 32 rows of W
    const int w_rows = min(BM, p.N - n0), w_row = quad * 32 + lane;
    Place<STAGES> to;
    Place<RAW> from;
    if (!TMA) pdl_wait();
    if (warp >= GROUP) { to.next(); from.next(); }                  // the second four warps start with the second chunk
    for (int c = warp / GROUP; c < chunks; c += 2) {
      ok = mbar_wait(&sh->empty[to.i], to.phase ^ 1);
      if (TMA && ok) ok = mbar_wait(&sh->w_full[from.i], from.phase);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      TC_FENCE_AFTER();
      const unsigned char* src = raw + from.i * S::RAW_STAGE;
      const int k = k0 + c * CHUNK;
      const uint32_t to_w = tmem_w + ((uint32_t)(quad * 32) << 16) + to.i * S::W_COLS;
#pragma unroll
      for (int half = 0; half < 2; ++half) {           // W: a thread a row
        uint32_t part[2][PW][4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          Eight<TW> v;
          if constexpr (TMA) v.read(src, w_row, 2 * half + h);
          else v.load(W + (size_t)(w_row < w_rows ? w_row : 0) * p.ldw, w_row < w_rows, k + 16 * half + 8 * h, k_end, p.w_vec != 0);
          v.cut(part[h]);
        }
#pragma unroll
        for (int x = 0; x < PW; ++x) tmem_st8(to_w + 16 * x + 8 * half, part[0][x], part[1][x]);
      }
      if (TMA && S::A_CUTTERS == 0 && !(ok = __all_sync(0xffffffffu, mbar_wait(&sh->a_full[from.i], from.phase)))) break;
      unsigned char* dst = stages + to.i * S::STAGE + kb * 128 + r * 16;
#pragma unroll
      for (int i = 0; i < (S::A_CUTTERS == 0 ? S::A_GROUPS : 0); ++i) {          // A: eight rows at a time, 32 bytes a lane (16 of 16-bit numbers)
        const int g = quad + i * GROUP, row = g * 8 + r;
        if (g * 8 >= rows16) break;
        Eight<TA> v;
        uint32_t part[PA][4];
        if constexpr (TMA) v.read(src + S::W_RAW, row, kb);
        else v.load(A + (size_t)(row < rows ? row : 0) * p.lda, row < rows, k + kb * 8, k_end, p.a_vec != 0);
        v.cut(part);
#pragma unroll
        for (int x = 0; x < PA; ++x)
          *reinterpret_cast<uint4*>(dst + g * GROUP_BYTES + x * S::A_PART) = make_uint4(part[x][0], part[x][1], part[x][2], part[x][3]);
      }
      asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
      TC_FENCE_BEFORE();
      PROXY_FENCE();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&sh->full[to.i]);
        if (TMA) mbar_arrive(&sh->raw_empty[from.i]);
      }
      to.next(); to.next();
      from.next(); from.next();
    }
  } else if (warp >= CUTTERS + S::ADDERS) {
    // ------------------------------------------------------------- few rows of A into parts, eight a warp
    const int g = warp - CUTTERS - S::ADDERS, r = lane & 7, kb = lane >> 3;
    Place<STAGES> to;
    Place<RAW> from;
    for (int c = 0; c < chunks; ++c, to.next(), from.next()) {
      ok = __all_sync(0xffffffffu, mbar_wait(&sh->empty[to.i], to.phase ^ 1) && mbar_wait(&sh->a_full[from.i], from.phase));
      if (!ok) break;
      if (g * 8 < rows16) {
        Eight<TA> v;
        uint32_t part[PA][4];
        v.read(raw + from.i * S::RAW_STAGE + S::W_RAW, g * 8 + r, kb);
        v.cut(part);
#pragma unroll
        for (int x = 0; x < PA; ++x)
          *reinterpret_cast<uint4*>(stages + to.i * S::STAGE + kb * 128 + r * 16 + g * GROUP_BYTES + x * S::A_PART) =
              make_uint4(part[x][0], part[x][1], part[x][2], part[x][3]);
      }
      PROXY_FENCE();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&sh->full[to.i]);
        mbar_arrive(&sh->raw_empty[from.i]);
      }
    }
  } else {
    // ------------------------------------------------------------- sums
    constexpr int HALF = NB <= 16 ? 16 : NB / 2;
    const int adder = warp - CUTTERS, quad = warp & 3, h0 = (rows16 / 16 + 1) / 2 * 16;     // the second four warps take the rows from h0 on
    const int first = adder < 4 ? 0 : h0, mine = S::ADDERS == 4 ? rows16 : adder < 4 ? min(h0, rows16) : rows16 - h0;
    float acc[HALF];                                   // this thread's sums: row n of W, rows of A from `first` on
#pragma unroll
    for (int i = 0; i < HALF; ++i) acc[i] = 0.f;
    Place<ACCS> out;
    for (int c = 0; c < chunks; ++c, out.next()) {
      ok = __all_sync(0xffffffffu, mbar_wait(&sh->acc_full[out.i], out.phase));
      if (!ok) break;
      TC_FENCE_AFTER();
      const uint32_t taddr = tmem + ((uint32_t)(quad * 32) << 16) + out.i * NB + first;
#pragma unroll
      for (int j = 0; j < HALF; j += 16) {
        if (j >= mine) break;
        uint32_t v[16];
        tmem_ld16(taddr + j, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[j + i] += __uint_as_float(v[i]);
      }
      TC_FENCE_BEFORE();
      warp_arrive(&sh->acc_empty[out.i], lane);
    }
    if constexpr (S::PUSH) {
      const int n = quad * 32 + lane, to = (n >> 2) / quads;
      const uint32_t addr = smem_u32(here + ((part * rows) * quads + (n >> 2) - to * quads) * 4 + (n & 3));
      if (p.parts > 1) cluster_left();
#pragma unroll
      for (int i = 0; i < HALF; ++i) {
        if (i >= rows) break;
        if (p.parts > 1) cluster_push(addr + i * quads * 16, &sh->pushed, acc[i], to);
        else here[i * quads * 4 + n] = acc[i];
      }
    } else {
      // every product of this block is done, and with them every read of the ring
#pragma unroll
      for (int i = 0; i < HALF; ++i)
        if (i < mine) sums[(first + i) * BM + quad * 32 + lane] = acc[i];
    }
  }
  if (S::PUSH && p.parts > 1 && (warp < CUTTERS || warp >= CUTTERS + S::ADDERS)) {
    __syncwarp();
    cluster_left();
  }
  // (a wait that one elected thread made alone counts too, whichever it is)
  if (__any_sync(0xffffffffu, !ok) && lane == 0) { atomicOr(p.status, JV_STATUS_WAIT_EXPIRED); sh->failed = 1; }
  TC_FENCE_BEFORE();
  __syncthreads();
  if (sh->failed) {                                    // products and copies under way get a bounded time to finish
    if (warp == S::ISSUER && elect_one()) drain_products_after_failure(&sh->drain);
    if (TMA && warp == S::BRINGER && brought > 0)
      for (int c = max(0, brought - RAW); c < brought; ++c) {
        drain_copies_after_failure(&sh->w_full[c % RAW], (c / RAW) & 1);
        drain_copies_after_failure(&sh->a_full[c % RAW], (c / RAW) & 1);
      }
    __syncthreads();
  }
  if (warp == S::ISSUER) {
    TC_FENCE_AFTER();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(S::TMEM_COLS) : "memory");
  }
  // ------------------------------------------------------------- the parts' sums, added up in their order: each block some of the tile
  const int share = (rows * (BM / 4) + p.parts - 1) / p.parts, t0 = part * share;     // of four numbers
  const int n_mine = S::PUSH ? rows * my_quads : min(share, rows * (BM / 4) - t0);
  const float4* ours = S::PUSH ? reinterpret_cast<const float4*>(here) : reinterpret_cast<const float4*>(sums) + t0;
  int stride = S::PUSH ? rows * quads : 0;
  if (S::PUSH && p.parts > 1) {
    // (Read from the others behind a barrier of the cluster they took 1,800 clocks.)
    if (!__syncthreads_and(wait_pushed(&sh->pushed))) {
      if (threadIdx.x == 0) atomicOr(p.status, JV_STATUS_WAIT_EXPIRED);
      cluster_sync();                                  // what others have pushed, or may yet push, finds this block there
    }
  } else if (!S::PUSH && p.parts > 1) {
    __syncwarp();
    cluster_sync();
    // they come here first, each block's from its own part on: read in their order, by all blocks alike, they took 4,600 clocks of 112 rows
    float4* all = reinterpret_cast<float4*>(sums) + NB * (BM / 4);
    for (int u = threadIdx.x; u < p.parts * share; u += S::THREADS) {
      const int turn = u / share, e = u - turn * share, q = turn + part < p.parts ? turn + part : turn + part - p.parts;
      if (e < n_mine) all[q * share + e] = cluster_load(smem_u32(ours + e), q);
    }
    __syncthreads();
    cluster_leave();
    ours = all;
    stride = share;
  }
  pdl_wait();                                          // nothing is written before the kernels before this one are done
  const bool vec = sizeof(TC) == 4 && (((uintptr_t)p.C | (p.ldc * sizeof(TC)) | (p.c_batch * sizeof(TC))) & 15) == 0;
  TC* C = (TC*)p.C + blockIdx.y * p.c_batch + (size_t)m0 * p.ldc + n0;
  for (int e = threadIdx.x; e < n_mine; e += S::THREADS) {
    int m = (t0 + e) / (BM / 4), n = (t0 + e) % (BM / 4) * 4, at = e;
    if (S::PUSH) {
      m = e / my_quads;
      n = (quad0 + e - m * my_quads) * 4;
      at = m * quads + e - m * my_quads;
    }
    if (n0 + n >= p.N || (p.row_token != nullptr && p.row_token[m0 + m] < 0)) continue;
    float y[4] = {0.f, 0.f, 0.f, 0.f};
    for (int q = 0; q < p.parts; ++q) {
      const float4 v = ours[q * stride + at];
      y[0] += v.x; y[1] += v.y; y[2] += v.z; y[3] += v.w;
    }
    TC* dst = C + (size_t)m * p.ldc + n;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (n0 + n + i < p.N && !is_number(y[i])) y[i] = plain_sum(A + (size_t)m * p.lda, W + (size_t)(n + i) * p.ldw, p.K);
    if (p.gelu) {
#pragma unroll
      for (int i = 0; i < 4; ++i) y[i] = 0.5f * y[i] * (1.f + erff(y[i] * 0.70710678118654752f));
    }
    if constexpr (sizeof(TC) == 4)
      if (vec && n0 + n + 4 <= p.N) {
        *reinterpret_cast<float4*>(dst) = make_float4(y[0], y[1], y[2], y[3]);
        continue;
      }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (n0 + n + i < p.N) dst[i] = from_f32<TC>(y[i]);
  }
  if (!S::PUSH && p.parts > 1) {                       // the others may still read this block's sums
    __syncwarp();
    cluster_left();
  }
}

// [batch][rows][k] as TMA sees it, boxes of `box` rows of a chunk.
template <typename T> bool make_map(CUtensorMap* map, const void* base, int k, int rows, int ld, size_t batch_stride, int batch, int box) {
  auto fn = encode_fn();
  if (fn == nullptr) return false;
  const cuuint64_t size = sizeof(T);
  const cuuint64_t dims[3] = {(cuuint64_t)k, (cuuint64_t)rows, (cuuint64_t)batch};
  const cuuint64_t strides[2] = {(cuuint64_t)ld * size, batch > 1 ? (cuuint64_t)batch_stride * size : (cuuint64_t)ld * size};
  const cuuint32_t boxes[3] = {(cuuint32_t)CHUNK, (cuuint32_t)box, 1};
  const cuuint32_t es[3] = {1, 1, 1};
  return fn(map, Eight<T>::MAP_TYPE, 3, const_cast<void*>(base), dims, strides, boxes, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            Eight<T>::MAP_SWIZZLE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
template <typename T> bool addressable(const void* base, int ld, size_t batch_stride, int batch) {
  constexpr int whole = 16 / sizeof(T);
  return ((uintptr_t)base & 15) == 0 && ld > 0 && ld % whole == 0 && (batch <= 1 || (batch_stride % whole == 0 && batch_stride > 0));
}

// jv_launch with clusters of `cluster` blocks along x (at most eight, and a divisor of the grid's x).
template <typename... KArgs, typename... Args>
int launch_clusters(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, int cluster, cudaStream_t stream,
                    Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int n = 0;
  if (cluster > 1) {
    attr[n].id = cudaLaunchAttributeClusterDimension;
    attr[n].val.clusterDim.x = (unsigned)cluster;
    attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
    ++n;
  }
  if (jv_pdl_enabled()) {
    attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  cfg.attrs = attr;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...) == cudaSuccess ? JV_OK : JV_ERR_LAUNCH;
}

template <bool TMA, int NB, typename TA, typename TW, typename TC>
int launch(const CUtensorMap& w_map, const CUtensorMap& a_map, const Params& p, int batch, cudaStream_t stream) {
  auto kern = gemm_f32_kernel<TMA, NB, TA, TW, TC>;
  constexpr int smem = Shape<TMA, NB, TA, TW>::SMEM;
  static_assert(smem <= 227 * 1024, "shared memory");
  static bool done[JV_MAX_DEVICES] = {};
  if (!jv_once_per_device(done, [&] {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess;
      }))
    return JV_ERR_UNSUPPORTED;
  const long long blocks = (long long)p.strips * p.parts * ((p.M + p.row_tile - 1) / p.row_tile);
  if (blocks > 0x7fffffff) return JV_ERR_UNSUPPORTED;
  return launch_clusters(kern, dim3((unsigned)blocks, batch), dim3(Shape<TMA, NB, TA, TW>::THREADS), smem, p.parts, stream, w_map, a_map, p);
}

template <typename TA, typename TW, typename TC>
int dispatch(Params p, int batch, int matrices, cudaStream_t stream) {
  CUtensorMap w_map = {}, a_map = {};
  const bool grouped = p.tile_expert != nullptr;
  auto tile_of = [&](int most) {
    if (grouped) return p.row_tile;
    const int tiles = (p.M + most - 1) / most;
    return ((p.M + tiles - 1) / tiles + 15) / 16 * 16;
  };
  p.row_tile = tile_of(MAX_ROWS);
  if (p.K < 1 || !addressable<TA>(p.A, p.lda, p.a_batch, batch) || !addressable<TW>(p.W, p.ldw, p.w_batch, matrices) ||
      !make_map<TW>(&w_map, p.W, p.K, p.N, p.ldw, p.w_batch, matrices, BM) ||
      !make_map<TA>(&a_map, p.A, p.K, p.M, p.lda, p.a_batch, batch, p.row_tile)) {
    p.row_tile = tile_of(64);
    return launch<false, 64, TA, TW, TC>(w_map, a_map, p, batch, stream);
  }
  if (p.row_tile <= 16) return launch<true, 16, TA, TW, TC>(w_map, a_map, p, batch, stream);
  if (p.row_tile <= 64) return launch<true, 64, TA, TW, TC>(w_map, a_map, p, batch, stream);
  return launch<true, 128, TA, TW, TC>(w_map, a_map, p, batch, stream);
}

// k's of a part, by N, K and the batch alone, never by the rows.  Strips times parts about fill the device, and so that two tiles of rows
// (129 to 256) still run at once, up to 16 strips: clusters of five or six blocks, one a multiprocessor, fill 130 of a B200's, clusters
// of eight 120, and eight strips of two tiles are 128.  (Model of width 1,024, 203 rows: 192 us of products with up to eight parts, 147 so;
// 100 rows 102 and 110; one row: no difference.)
int part_of_k(int N, int K, int batch) {
  const long long strips = (long long)((N + BM - 1) / BM) * batch;
  const long long room = jv_multiprocessors() * 9 / 10, two_tiles = room / (2 * strips);
  const long long parts = two_tiles >= 4 ? (two_tiles < MAX_PARTS ? two_tiles : MAX_PARTS) : room / strips < MAX_PARTS ? room / strips : MAX_PARTS;
  if (parts <= 1) return (K + CHUNK - 1) / CHUNK * CHUNK;
  const int even = (int)((K + parts - 1) / parts + CHUNK - 1) / CHUNK * CHUNK;
  return even < LEAST_PART ? LEAST_PART : even;
}

// four elements a load along k: every row (of every product of a batch) starts on such a boundary
bool rows_aligned(const void* p, int size, int ld, size_t batch_stride, int batch) {
  return ((uintptr_t)p & (4 * size - 1)) == 0 && ld % 4 == 0 && (batch <= 1 || batch_stride % 4 == 0);
}

int run(const void* A, int a_dtype, int lda, size_t a_batch, const void* W, int w_dtype, int ldw, size_t w_batch, void* C,
        int c_dtype, int ldc, size_t c_batch, int M, int N, int K, int batch, int w_fixed, int* status, cudaStream_t stream) {
  Params p{A, W, C, lda, ldw, ldc, M, N, K, a_batch, w_batch, c_batch, 0, 0, (N + BM - 1) / BM, 1, 0, 0, w_fixed, status, nullptr, nullptr, 0};
  p.part_k = part_of_k(N, K, batch);
  p.parts = K > 0 ? (K + p.part_k - 1) / p.part_k : 1;
  p.a_vec = rows_aligned(A, a_dtype == 0 ? 4 : 2, lda, a_batch, batch);
  p.w_vec = rows_aligned(W, w_dtype == 0 ? 4 : 2, ldw, w_batch, batch);
  JV_DISPATCH_DTYPE(a_dtype, TA, JV_DISPATCH_DTYPE(w_dtype, TW, JV_DISPATCH_DTYPE(c_dtype, TC,
      return (dispatch<TA, TW, TC>(p, batch, batch, stream)))));
  return JV_ERR_UNSUPPORTED;
}
}  // namespace

// A: [M, K] rows of lda elements; W: [N, K] rows of ldw elements; C: [M, N] rows of ldc.  w_fixed: none of the kernels launched before
// this one writes W, which is then read before they have finished.
JV_EXPORT int jv_gemm_f32(const void* A, int a_dtype, int lda, const void* W, int w_dtype, int ldw, void* C, int c_dtype, int ldc,
                          int M, int N, int K, int w_fixed, int* status, cudaStream_t stream) {
  if (M == 0 || N == 0) return JV_OK;
  return run(A, a_dtype, lda, 0, W, w_dtype, ldw, 0, C, c_dtype, ldc, 0, M, N, K, 1, w_fixed, status, stream);
}

// Routed experts: rows of A and C in tiles of `tile` (16 or 64), tile t of expert tile_expert[t] (-1: nothing to do) with the weight
// W + expert * w_expert; rows whose row_token is -1 are left alone.  gelu: the exact gelu of the result.
JV_EXPORT int jv_gemm_f32_grouped(const void* A, int a_dtype, int lda, const void* W, int w_dtype, int ldw, long long w_expert, int experts,
                                  void* C, int c_dtype, int ldc, int tiles, int tile, const int* tile_expert, const int* row_token,
                                  int N, int K, int gelu, int* status, cudaStream_t stream) {
  if (tiles == 0 || N == 0) return JV_OK;
  if ((tile != 16 && tile != 64) || experts < 1 || tiles > 0x7fffffff / 64) return JV_ERR_UNSUPPORTED;
  Params p{A, W, C, lda, ldw, ldc, tiles * tile, N, K, 0, (size_t)w_expert, 0, 0, 0, (N + BM - 1) / BM, 1, 0, tile, 0, status,
           tile_expert, row_token, gelu};
  p.part_k = part_of_k(N, K, GROUPED_AT_ONCE);
  p.parts = K > 0 ? (K + p.part_k - 1) / p.part_k : 1;
  p.a_vec = rows_aligned(A, a_dtype == 0 ? 4 : 2, lda, 0, 1);
  p.w_vec = rows_aligned(W, w_dtype == 0 ? 4 : 2, ldw, (size_t)w_expert, experts);
  JV_DISPATCH_DTYPE(a_dtype, TA, JV_DISPATCH_DTYPE(w_dtype, TW, JV_DISPATCH_DTYPE(c_dtype, TC,
      return (dispatch<TA, TW, TC>(p, 1, experts, stream)))));
  return JV_ERR_UNSUPPORTED;
}

// `batch` products of the same sizes in one launch: product b reads A + b*a_batch, W + b*w_batch and writes
// C + b*c_batch (strides in elements; rows of one product may lie between rows of another).
JV_EXPORT int jv_gemm_f32_batched(const void* A, int a_dtype, int lda, long long a_batch, const void* W, int w_dtype, int ldw,
                                  long long w_batch, void* C, int c_dtype, int ldc, long long c_batch, int M, int N, int K,
                                  int batch, int w_fixed, int* status, cudaStream_t stream) {
  if (M == 0 || N == 0 || batch == 0) return JV_OK;
  if (batch > 65535) return JV_ERR_UNSUPPORTED;
  return run(A, a_dtype, lda, (size_t)a_batch, W, w_dtype, ldw, (size_t)w_batch, C, c_dtype, ldc, (size_t)c_batch, M, N, K, batch,
             w_fixed, status, stream);
}
