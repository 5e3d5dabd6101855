// C[M, N] = A[M, K] * W[N, K]^T on CUDA cores, accumulating in 32-bit with FFMA: the
// matrix product of the 32-bit path (no reduced-precision tensor mode), also used where
// a result must leave in 32-bit (logits) from 16-bit operands.
//
// Every output element is the same sum whatever M and N are, so a row's result does not depend on which other rows are
// in the batch: k is cut into segments of SEG, a segment is summed with k ascending, and the segments' sums are added in
// ascending order.  Which threads take which segment is then free, and that is what both kernels use to fill the device:
//
//   rows_kernel   up to 16 rows (decode steps), bound by the bytes of W: a warp takes 32 columns (a lane each) and one
//                 segment at a time, W comes through a ring of three cp.async stages a warp; the eight warps of a block take
//                 eight segments of the same columns and add their sums through shared memory.
//   tile_kernel   64 x 64 tiles, a group of 64 threads with 8 x 8 outputs a thread in packed pairs of columns (a warp's reads of
//                 shared memory cost a clock a number and lane, whoever else reads the same: 16 of them for 32 packed
//                 multiply-adds), the next 16 k under way in registers; G = 1, 2 or 4 groups a block take segments in turn
//                 where tiles alone leave multiprocessors idle.
//
// Measured on a model of width 1,024 (two layers, 203 tokens, 32-bit): its products take 0.68 ms, 1.98 ms with 64 x 64 tiles of
// 4 x 4 outputs a thread, four-byte loads and no split of k (which a decode step of four rows also ran on: 0.47 against 0.09 ms).
// The first two products of a layer (64 and 96 tiles on 148 multiprocessors) run at 40 % of the multiply-adds of the
// multiprocessors that have a tile.
#include "common.cuh"

namespace {
constexpr int SEG = 128;                 // k's whose sum is one chain
constexpr int BM = 64, BN = 64, BK = 16;
constexpr int GROUP = 64;                // threads of a group
constexpr int STAGE = BK * BM;           // floats of one operand's stage, [k][row ^ swizzle]
constexpr int GROUP_FLOATS = 4 * STAGE;  // two stages of A and of W; also holds a group's sums of one segment (64 x 64)
static_assert(GROUP_FLOATS >= BM * BN, "a segment's sums have to fit the stages");

struct GemmParams {
  const void* A; const void* W; void* C;
  int lda, ldw, ldc, M, N, K;
  size_t a_batch, w_batch, c_batch;      // a batch of independent products: grid.z of them, operands this far apart
  int a_vec, w_vec;                      // four elements a load along k
};

// 4 consecutive k's of a row as floats; zeros past `k_end` or for a row that is not there
template <typename T>
__device__ __forceinline__ float4 load4(const T* __restrict__ row, bool live, int k, int k_end, bool vec) {
  if (live && vec && k + 4 <= k_end) {
    if constexpr (sizeof(T) == 4) {
      return *reinterpret_cast<const float4*>(row + k);
    } else {
      const uint2 a = *reinterpret_cast<const uint2*>(row + k);
      return make_float4(__uint_as_float(a.x << 16), __uint_as_float(a.x & 0xffff0000u), __uint_as_float(a.y << 16),
                         __uint_as_float(a.y & 0xffff0000u));
    }
  }
  float v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = live && k + i < k_end ? to_f32(row[k + i]) : 0.f;
  return make_float4(v[0], v[1], v[2], v[3]);
}

__device__ __forceinline__ void group_sync(int group) { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(GROUP) : "memory"); }

template <int G, typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(G* GROUP) tile_kernel(const GemmParams p) {
  extern __shared__ __align__(16) float smem[];
  pdl_trigger();
  pdl_wait();
  const TA* A = (const TA*)p.A + blockIdx.z * p.a_batch;
  const TW* W = (const TW*)p.W + blockIdx.z * p.w_batch;
  TC* C = (TC*)p.C + blockIdx.z * p.c_batch;
  const int group = threadIdx.x / GROUP, tid = threadIdx.x % GROUP;
  float* mine = smem + group * GROUP_FLOATS;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tx = tid & 7, ty = tid >> 3;               // this thread's outputs: rows ty * 8 .., columns tx * 8 ..
  // what it loads of a stage: 4 k's of rows lrow, lrow + 16, .. of either operand (four lanes a row's 64 bytes)
  const int lrow = tid >> 2, lq = tid & 3;
  const int n_seg = (p.K + SEG - 1) / SEG;
  uint64_t total[8][4];                                // rows x pairs of columns
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) total[i][j] = 0;       // a pair of zeros
  float4 av[4], wv[4];
  auto fetch = [&](int k, int k_end) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = lrow + 16 * i;
      const bool a_live = m0 + r < p.M, w_live = n0 + r < p.N;
      av[i] = load4<TA>(A + (size_t)(a_live ? m0 + r : 0) * p.lda, a_live, k + lq * 4, k_end, p.a_vec);
      wv[i] = load4<TW>(W + (size_t)(w_live ? n0 + r : 0) * p.ldw, w_live, k + lq * 4, k_end, p.w_vec);
    }
  };
  // a row's place is turned by its quarter of the stage's k's, so that the four lanes of a row meet no bank twice
  auto put = [&](int buf) {
    float* as = mine + buf * 2 * STAGE + lq * 4 * BM;
    float* ws = as + STAGE;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = (lrow + 16 * i) ^ (lq << 3);
      as[r] = av[i].x; as[BM + r] = av[i].y; as[2 * BM + r] = av[i].z; as[3 * BM + r] = av[i].w;
      ws[r] = wv[i].x; ws[BM + r] = wv[i].y; ws[2 * BM + r] = wv[i].z; ws[3 * BM + r] = wv[i].w;
    }
  };
  for (int first = 0; first < n_seg; first += G) {     // a round: one segment a group
    const int seg = first + group;
    uint64_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    if (seg < n_seg) {
      const int k0 = seg * SEG, k_end = min(p.K, k0 + SEG);
      fetch(k0, k_end);
      put(0);
      group_sync(group);
      int buf = 0;
      for (int k = k0; k < k_end; k += BK, buf ^= 1) {
        const bool more = k + BK < k_end;
        if (more) fetch(k + BK, k_end);
        const float* as = mine + buf * 2 * STAGE;
        const float* ws = as + STAGE;
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
          const int turn = kk >> 2;
          const float4 a0 = *reinterpret_cast<const float4*>(as + kk * BM + ((ty ^ turn) << 3));
          const float4 a1 = *reinterpret_cast<const float4*>(as + kk * BM + ((ty ^ turn) << 3) + 4);
          const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(ws + kk * BM + ((tx ^ turn) << 3));
          const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(ws + kk * BM + ((tx ^ turn) << 3) + 4);
          const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
          const uint64_t w[4] = {w0.x, w0.y, w1.x, w1.y};
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint64_t aa = pack2(a[i], a[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fma2(aa, w[j], acc[i][j]);
          }
        }
        if (more) put(buf ^ 1);                        // last read before the sync that ended the stage before
        group_sync(group);
      }
    }
    if constexpr (G == 1) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) total[i][j] = first == 0 ? acc[i][j] : add2(total[i][j], acc[i][j]);
    } else {
      // the other groups' sums go through their own stages, and the first group adds them in the segments' order
      if (group > 0 && seg < n_seg) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) *reinterpret_cast<uint64_t*>(mine + ((i * 4 + j) * GROUP + tid) * 2) = acc[i][j];
      }
      __syncthreads();
      if (group == 0) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint64_t t = first == 0 ? acc[i][j] : add2(total[i][j], acc[i][j]);
#pragma unroll
            for (int g = 1; g < G; ++g)
              if (first + g < n_seg) t = add2(t, *reinterpret_cast<const uint64_t*>(smem + g * GROUP_FLOATS + ((i * 4 + j) * GROUP + tid) * 2));
            total[i][j] = t;
          }
      }
      __syncthreads();
    }
  }
  if (group > 0) return;
  const bool vec_c = sizeof(TC) == 4 && ((uintptr_t)C & 15) == 0 && (p.ldc & 3) == 0 && n0 + tx * 8 + 8 <= p.N;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + ty * 8 + i;
    if (m >= p.M) continue;
    TC* row = C + (size_t)m * p.ldc + n0 + tx * 8;
    float c[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) unpack2(total[i][j], c[2 * j], c[2 * j + 1]);
    if (vec_c) {
      reinterpret_cast<float4*>(row)[0] = make_float4(c[0], c[1], c[2], c[3]);
      reinterpret_cast<float4*>(row)[1] = make_float4(c[4], c[5], c[6], c[7]);
      continue;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (n0 + tx * 8 + j < p.N) row[j] = from_f32<TC>(c[j]);
  }
}

// ------------------------------------------------------------------------------------------------- few rows
constexpr int ROWS_WARPS = 8, ROWS_COLS = 32, KC = 32, RING = 3, WLD = KC + 4;

template <int MR> struct RowsShape {
  static constexpr int STAGE_FLOATS = ROWS_COLS * WLD + KC * MR;
  static constexpr int SMEM = (int)sizeof(float) * (ROWS_WARPS * RING * STAGE_FLOATS + ROWS_WARPS * MR * ROWS_COLS);
};

__device__ __forceinline__ void copy_16(float* dst, const void* src, bool live) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = live ? 16 : 0;                         // 0: zeros are written and nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copy_4(float* dst, const void* src, bool live) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = live ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

// MR: rows that the lanes keep sums of (M <= MR; rows past M are zeros)
template <int MR, typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(ROWS_WARPS * 32) rows_kernel(const GemmParams p) {
  extern __shared__ __align__(16) float smem[];
  pdl_trigger();
  pdl_wait();
  const TA* A = (const TA*)p.A + blockIdx.z * p.a_batch;
  const TW* W = (const TW*)p.W + blockIdx.z * p.w_batch;
  TC* C = (TC*)p.C + blockIdx.z * p.c_batch;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n0 = blockIdx.x * ROWS_COLS;
  constexpr int SF = RowsShape<MR>::STAGE_FLOATS;
  float* ring = smem + warp * RING * SF;
  float* parts = smem + ROWS_WARPS * RING * SF;        // [warp][row][column]
  const int n_seg = (p.K + SEG - 1) / SEG;
  // this warp's chunks: KC k's each, those of its segments warp, warp + 8, ... one after the other
  constexpr int PER_SEG = SEG / KC;
  const int my_segs = warp < n_seg ? (n_seg - warp - 1) / ROWS_WARPS + 1 : 0;
  const int chunks = my_segs * PER_SEG;
  auto chunk_k = [&](int c) { return ((c / PER_SEG) * ROWS_WARPS + warp) * SEG + (c % PER_SEG) * KC; };
  auto stage = [&](int c) {
    if (c < chunks) {
      const int k = chunk_k(c);
      float* ws = ring + (c % RING) * SF;
      float* xs = ws + ROWS_COLS * WLD;
      if (sizeof(TW) == 4 && p.w_vec) {                // eight lanes a row of 32 floats
#pragma unroll
        for (int i = 0; i < ROWS_COLS / 4; ++i) {
          const int r = i * 4 + (lane >> 3), kk = k + (lane & 7) * 4;
          const bool live = n0 + r < p.N && kk < p.K;  // a row's length is a multiple of four here
          copy_16(ws + r * WLD + (lane & 7) * 4, W + (live ? (size_t)(n0 + r) * p.ldw + kk : 0), live);
        }
      } else {
#pragma unroll 4
        for (int i = 0; i < ROWS_COLS; ++i) {
          const bool live = n0 + i < p.N && k + lane < p.K;
          ws[i * WLD + lane] = live ? to_f32(W[(size_t)(n0 + i) * p.ldw + k + lane]) : 0.f;
        }
      }
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        const bool live = m < p.M && k + lane < p.K;
        const TA* x = A + (live ? (size_t)m * p.lda + k + lane : 0);
        if constexpr (sizeof(TA) == 4) copy_4(xs + lane * MR + m, x, live);
        else xs[lane * MR + m] = live ? to_f32(*x) : 0.f;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int c = 0; c < RING - 1; ++c) stage(c);
  constexpr int PAIRS = MR > 1 ? MR / 2 : 1;
  uint64_t acc[PAIRS];                                 // pairs of rows (one row: the low half)
  const int rounds = (n_seg + ROWS_WARPS - 1) / ROWS_WARPS;
  constexpr int OUTS = (MR * ROWS_COLS + 255) / 256;
  float sum[OUTS];
#pragma unroll
  for (int i = 0; i < OUTS; ++i) sum[i] = 0.f;
  for (int round = 0; round < rounds; ++round) {
    const int seg = round * ROWS_WARPS + warp;
    if (seg < n_seg) {
#pragma unroll
      for (int i = 0; i < PAIRS; ++i) acc[i] = 0;
      for (int cc = 0; cc < PER_SEG; ++cc) {
        const int c = round * PER_SEG + cc;
        __syncwarp();                                  // the slot that is filled next has been read
        stage(c + RING - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(RING - 1) : "memory");
        __syncwarp();
        const float* ws = ring + (c % RING) * SF + lane * WLD;
        const float* xs = ring + (c % RING) * SF + ROWS_COLS * WLD;
#pragma unroll
        for (int kk = 0; kk < KC; kk += 4) {
          const float4 w4 = *reinterpret_cast<const float4*>(ws + kk);
          const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float* x = xs + (kk + t) * MR;
            if constexpr (MR == 1) {
              float lo, hi;
              unpack2(acc[0], lo, hi);
              acc[0] = pack2(fmaf(x[0], w[t], lo), 0.f);
            } else {
              const uint64_t ww = pack2(w[t], w[t]);
#pragma unroll
              for (int i = 0; i < PAIRS; ++i) acc[i] = fma2(*reinterpret_cast<const uint64_t*>(x + 2 * i), ww, acc[i]);
            }
          }
        }
      }
#pragma unroll
      for (int i = 0; i < PAIRS; ++i) {
        float lo, hi;
        unpack2(acc[i], lo, hi);
        parts[(warp * MR + 2 * i) * ROWS_COLS + lane] = lo;
        if (MR > 1) parts[(warp * MR + 2 * i + 1) * ROWS_COLS + lane] = hi;
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < OUTS; ++i) {
      const int o = threadIdx.x + i * 256;
      if (o < MR * ROWS_COLS) {
        for (int w = 0; w < ROWS_WARPS && round * ROWS_WARPS + w < n_seg; ++w) {
          const float v = parts[w * MR * ROWS_COLS + o];
          sum[i] = round == 0 && w == 0 ? v : sum[i] + v;
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < OUTS; ++i) {
    const int o = threadIdx.x + i * 256, m = o / ROWS_COLS, n = n0 + o % ROWS_COLS;
    if (m < p.M && m < MR && n < p.N) C[(size_t)m * p.ldc + n] = from_f32<TC>(sum[i]);
  }
}

template <int MR, typename TA, typename TW, typename TC>
int launch_rows(const GemmParams& p, int batch, cudaStream_t stream) {
  auto kern = rows_kernel<MR, TA, TW, TC>;
  static bool done[JV_MAX_DEVICES] = {};
  if (!jv_once_per_device(done, [&] {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, RowsShape<MR>::SMEM) == cudaSuccess;
      }))
    return JV_ERR_UNSUPPORTED;
  return jv_launch(kern, dim3((p.N + ROWS_COLS - 1) / ROWS_COLS, 1, batch), dim3(ROWS_WARPS * 32), RowsShape<MR>::SMEM, stream, p);
}

template <int G, typename TA, typename TW, typename TC>
int launch_tiles(const GemmParams& p, int batch, cudaStream_t stream) {
  auto kern = tile_kernel<G, TA, TW, TC>;
  constexpr int smem = (int)sizeof(float) * G * GROUP_FLOATS;
  static bool done[JV_MAX_DEVICES] = {};
  if (!jv_once_per_device(done, [&] {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess;
      }))
    return JV_ERR_UNSUPPORTED;
  return jv_launch(kern, dim3((p.N + BN - 1) / BN, (p.M + BM - 1) / BM, batch), dim3(G * GROUP), smem, stream, p);
}

// Up to 16 rows are bound by the bytes of W, more by the multiply-adds.  One group a block once there are four tiles a
// multiprocessor (eight warps); fewer tiles share theirs out by segments.
template <typename TA, typename TW, typename TC>
int dispatch(const GemmParams& p, int batch, cudaStream_t stream) {
  if (p.M <= 1) return launch_rows<1, TA, TW, TC>(p, batch, stream);
  if (p.M <= 2) return launch_rows<2, TA, TW, TC>(p, batch, stream);
  if (p.M <= 4) return launch_rows<4, TA, TW, TC>(p, batch, stream);
  if (p.M <= 8) return launch_rows<8, TA, TW, TC>(p, batch, stream);
  if (p.M <= 16) return launch_rows<16, TA, TW, TC>(p, batch, stream);
  const long long tiles = (long long)((p.N + BN - 1) / BN) * ((p.M + BM - 1) / BM) * batch;
  const int sms = jv_multiprocessors(), n_seg = (p.K + SEG - 1) / SEG;
  if (n_seg >= 4 && tiles <= sms) return launch_tiles<4, TA, TW, TC>(p, batch, stream);
  if (n_seg >= 2 && tiles <= 3 * sms) return launch_tiles<2, TA, TW, TC>(p, batch, stream);
  return launch_tiles<1, TA, TW, TC>(p, batch, stream);
}

// four elements a load along k: every row (of every product of a batch) starts on such a boundary
bool rows_aligned(const void* p, int size, int ld, size_t batch_stride, int batch) {
  return ((uintptr_t)p & (4 * size - 1)) == 0 && ld % 4 == 0 && (batch <= 1 || batch_stride % 4 == 0);
}

int run(const void* A, int a_dtype, int lda, size_t a_batch, const void* W, int w_dtype, int ldw, size_t w_batch, void* C,
        int c_dtype, int ldc, size_t c_batch, int M, int N, int K, int batch, cudaStream_t stream) {
  GemmParams p{A, W, C, lda, ldw, ldc, M, N, K, a_batch, w_batch, c_batch, 0, 0};
  p.a_vec = rows_aligned(A, a_dtype == 0 ? 4 : 2, lda, a_batch, batch);
  // the asynchronous copies of rows_kernel also want whole 16 bytes at a row's end
  p.w_vec = rows_aligned(W, w_dtype == 0 ? 4 : 2, ldw, w_batch, batch) && (M > 16 || K % 4 == 0);
  JV_DISPATCH_DTYPE(a_dtype, TA, JV_DISPATCH_DTYPE(w_dtype, TW, JV_DISPATCH_DTYPE(c_dtype, TC,
      return (dispatch<TA, TW, TC>(p, batch, stream)))));
  return JV_ERR_UNSUPPORTED;
}
}  // namespace

// A: [M, K] rows of lda elements; W: [N, K] rows of ldw elements; C: [M, N] rows of ldc.
JV_EXPORT int jv_gemm_tn_simt(const void* A, int a_dtype, int lda, const void* W, int w_dtype, int ldw,
                              void* C, int c_dtype, int ldc, int M, int N, int K,
                              cudaStream_t stream) {
  if (M == 0 || N == 0) return JV_OK;
  if ((M + BM - 1) / BM > 65535) return JV_ERR_UNSUPPORTED;
  return run(A, a_dtype, lda, 0, W, w_dtype, ldw, 0, C, c_dtype, ldc, 0, M, N, K, 1, stream);
}

// `batch` products of the same sizes in one launch: product b reads A + b*a_batch, W + b*w_batch and writes
// C + b*c_batch (strides in elements; rows of one product may lie between rows of another).
JV_EXPORT int jv_gemm_tn_simt_batched(const void* A, int a_dtype, int lda, long long a_batch, const void* W, int w_dtype,
                                      int ldw, long long w_batch, void* C, int c_dtype, int ldc, long long c_batch,
                                      int M, int N, int K, int batch, cudaStream_t stream) {
  if (M == 0 || N == 0 || batch == 0) return JV_OK;
  if ((M + BM - 1) / BM > 65535 || batch > 65535) return JV_ERR_UNSUPPORTED;
  return run(A, a_dtype, lda, (size_t)a_batch, W, w_dtype, ldw, (size_t)w_batch, C, c_dtype, ldc, (size_t)c_batch, M, N, K, batch,
             stream);
}
