// Grouped fp32-accurate inverse of damped symmetric positive-definite matrices on the tensor cores:
//     out_m = (A_m + damping_m * I)^-1        for m = 0 .. count-1, sizes n_m arbitrary.
//
// Cholesky factor L, X = L^-1 row by row beside it, then X^T X, in 128 x 128 tiles.  A tile is one task:
//
//   DIAG(j)      S = A_jj - sum_{k<j} L_jk L_jk^T;   T_j = chol(S)^-1 on the CUDA cores (L_jj itself is not stored)
//   FACTOR(i,j)  S = A_ij - sum_{k<j} L_ik L_jk^T;   L_ij = S T_j^T                       for i > j
//   INV(i,j)     W = sum_{j<=k<i} L_ik X_kj;         X_ij = -T_i W                        for i > j  (X_jj = T_j)
//   OUT(i,j)     out_ij = sum_{r>=i} X_ri^T X_rj, mirrored                                for i >= j
//
// ONE persistent launch runs the tasks of all matrices.  CTAs claim them in the order of a list in which a task stands behind
// everything it needs, and a task waits for its operands K block by K block: per block row of a matrix there are two progress
// words, the number of finished tiles of that row of L and of that column of X.  Since the first unfinished task of the list
// never waits for a later one, any number of resident CTAs makes progress.  The sums run ahead of the chain
// DIAG -> FACTOR -> DIAG: only their last K blocks remain when a diagonal block is done.
//
// Sums are formed by the tensor cores from three-way bf16 splits of the fp32 values (v = hi + mid + lo carries the whole
// significand; six significant part products, small magnitudes first, as in the split3 flavour of umma_gemm2.cuh): every
// 64-wide K block goes to a fresh TMEM accumulator that the eight epilogue warps read back and add to a running fp32 sum in
// registers; A enters at the end (a sum that starts from -A has roundings of A's size in every step: 5 % more error in the
// inverse).  The second product of FACTOR and INV takes that sum from the same CTA: the epilogue writes its three parts into
// the operand half of a ring stage whose other half TMA fills with T.
//
// What bounds it: the chain of diagonal blocks (DIAG, one FACTOR tile, the last K panel of the next DIAG), and beside it the
// operand traffic of the ring, 96 KiB per K block of 1536 tensor cycles.  The former version ran the same arithmetic
// right-looking in 28 (six factors up to 784) to 121 (the 107 factors of ResNet-50) dependent launches: every K = 128 update
// read and wrote the fp32 matrix, each lane a row of its own, and every launch drained before the next began.
// Six factors 784, 4 x 512, 10: 597 -> 252 us; ResNet-50's 107 factors, pass after pass at the power limit: 8.04 -> 3.55 ms.
//
// Tables, task lists and the bf16 split buffers depend only on the addresses and sizes of the matrices; they are built once
// and cached (prepared_cache.h), so a repeated call (the K-FAC state) issues no host-to-device copy and can be captured in a
// CUDA graph, which then keeps them.  Inputs are not modified; a non-positive pivot sets the status word to ERR_NOT_SPD and the
// factorisation continues with pivot 1.
//
// Stands in for asdl/utils.py:91-96 (torch.linalg.cholesky + cholesky_inverse).
#include <cstring>

#include "gemm2_host.h"
#include "packed_fp32.cuh"
#include "prepared_cache.h"

namespace b200 {

namespace {

constexpr int TB = 128;  // tile

enum : int { TASK_DIAG = 0, TASK_FACTOR = 1, TASK_INV = 2, TASK_OUT = 3, TASK_END = 4 };

// L and X are kept as the images that the products want in shared memory.  Tile (i, j) of X, j <= i, has index i (i + 1) / 2 + j; L
// is kept below the diagonal only, tile (i, j), j < i, at i (i - 1) / 2 + j.  A tile consists of two halves of 64 columns; a half is three parts (hi, mid, lo) of 128 rows of 128 bytes, the 16-byte pieces of a row
// exchanged as the 128-byte swizzle does it.  A half of a part is a K block of a K-major operand (16 KiB, one copy); its rows
// [64 b, 64 b + 64) are 64 columns of K block b of an MN-major operand (8 KiB).  Rows and columns past the matrix are stored too.
constexpr int PART_BYTES = 128 * 128, TILE_BYTES = 6 * PART_BYTES;

struct TcMat {
  const float* A;          // input n x n (pitch lda)
  float* out;              // n x n
  uint8_t* L;              // tiles of L below the diagonal
  uint8_t* X;              // tiles of X
  int* row_l;              // finished tiles of block row i of L
  int* col_x;              // block column j of X is finished down to (not including) this block row
  int n, nb, lda, orig;
};

__device__ __forceinline__ uint8_t* tile_at(uint8_t* base, int i, int j) {
  return base + (static_cast<size_t>(i) * (i + 1) / 2 + j) * TILE_BYTES;
}
__device__ __forceinline__ uint8_t* below_at(uint8_t* base, int i, int j) {
  return base + (static_cast<size_t>(i) * (i - 1) / 2 + j) * TILE_BYTES;
}

struct Task {
  int mat, kind, i, j;
};

// K blocks of a task's sum
__host__ __device__ inline int task_blocks(int kind, int i, int j, int n) {
  if (kind == TASK_OUT) return (n - i * TB + G2_BK - 1) / G2_BK;
  return kind == TASK_INV ? 2 * (i - j) : 2 * j;
}

// ---- diagonal block: Cholesky factor and its inverse ----------------------------------------
// Four stages of 32 columns on the eight epilogue warps of a CTA.  Stage q, columns [kb, be):
//   factor   one warp, a row of the 32 x 32 block per lane, in registers.  Eight columns at a time: inside of the eight a column
//            is passed on by shuffles, so the chain from pivot to pivot is a product, a shuffle and a reciprocal square root;
//            then the eight are applied to the columns behind them;
//   panel    two warps, a thread takes two of the rows below (forward substitution with the block) or of the columns of the
//            inverse's rows [kb, be), eight columns behind the factor: with four warps of one row per thread, their loads took
//            the shared memory pipe from the factor's shuffles.  P[j][c] = T[kb + j][c] for c < be and L[c][kb + j] for c >= be;
//   update   S[i][c] -= sum_j P[j][i] P[j][c] for the rows i >= be: the trailing block right of be, the right-hand side of
//            the inverse left of it.  Finished columns of the factor are dead (only the inverse leaves the kernel), so both
//            share S.  A warp takes four rows of each row block, a lane one column of each column block up to the diagonal;
//   store    of the rows [kb, be) of T from P, by the other warps while the next stage is factored.
// Every entry sees the same roundings in the same order as a column-by-column elimination, and gives the same bits.  Two things
// bound it: the chain of pivots (80 clocks each), and the number of instructions that a single warp per scheduler issues:
// products are taken in pairs (fma.f32x2), and loops over groups of eight columns are not unrolled.  With each column applied at
// once to all behind it, in single products, the block took 49 000 clocks, 27 800 of them to factor; now 41 000.
constexpr int DG_SP = TB + 1;   // pitch of S: lanes on consecutive rows of a column, or on consecutive columns
constexpr int DG_PP = TB + 4;   // pitches of P and of the factored block: 16-byte reads
constexpr int DG_LP = 64;       // the entries from 32 on are zeros: what shifted registers past the block are updated with
constexpr int DG_SMEM = (TB * DG_SP + 2 * 32 * DG_PP + 32 * DG_LP + 32) * 4;

// Barrier of the eight epilogue warps.
__device__ __forceinline__ void epi_sync() { named_bar_sync(1, 256); }

// 1 / sqrt(pivot d); a pivot that is not positive is reported and replaced by 1.  The usual case has no branch in the chain:
// rsqrt.approx.ftz is exact enough for the Newton step that follows, and subnormal pivots go another way.
__device__ __forceinline__ float diag_pivot(float d, bool& bad) {
  float iv;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(iv) : "f"(d));
  if (!(d >= 1.17549435e-38f)) {
    if (!(d > 0.f)) {
      bad = true;
      d = 1.f;
    }
    iv = rsqrtf(d);
  }
  return iv * fmaf(-0.5f * d, iv * iv, 1.5f);   // one Newton step: full fp32 accuracy
}

// A row of 32 columns, of which the first eight are scalars and the others pairs.
struct DiagRow {
  float g[8];
  f32x2 v[12];
  // the next eight columns become the first ones
  __device__ __forceinline__ void shift() {
#pragma unroll
    for (int i = 0; i < 4; ++i) unpack2(v[i], g[2 * i], g[2 * i + 1]);
#pragma unroll
    for (int i = 0; i < 12; ++i) v[i] = i < 8 ? v[i + 4 < 12 ? i + 4 : 11] : 0ull;
  }
};

// Columns from the ninth on -= x[j] * o[j * DG_LP + 8 ...] for the eight finished columns j, in their order; N rows share the
// loads (a 16-byte load of a warp takes four clocks of the shared memory pipe even where all lanes read the same).
template <int N>
__device__ __forceinline__ void diag_apply(DiagRow (&row)[N], const float (&x)[N][8], const float* o) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    f32x2 m[N];
#pragma unroll
    for (int u = 0; u < N; ++u) m[u] = pack2(-x[u][j], -x[u][j]);
#pragma unroll
    for (int i = 0; i < 12; i += 2) {
      const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(o + j * DG_LP + 8 + 2 * i);
#pragma unroll
      for (int u = 0; u < N; ++u) {
        row[u].v[i] = fma2(m[u], q.x, row[u].v[i]);
        row[u].v[i + 1] = fma2(m[u], q.y, row[u].v[i + 1]);
      }
    }
  }
}

// Rows and columns behind stage KQ, whose columns are [32 KQ, 32 KQ + 32).
template <int KQ>
__device__ __forceinline__ void diag_update(float* S, const float* P, int warp, int lane) {
  constexpr int NB = 3 - KQ;   // row blocks
  f32x2 acc[NB][2][4];         // pairs of rows
  float* const rows = S + (32 * (KQ + 1) + 4 * warp) * DG_SP + lane;
#pragma unroll
  for (int b = 0; b < NB; ++b)
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int q = 0; q <= KQ + 1 + b; ++q) {
        const float* at = rows + (32 * b + 2 * r) * DG_SP + 32 * q;
        acc[b][r][q] = q == KQ ? 0ull : pack2(at[0], at[DG_SP]);
      }
#pragma unroll 4
  for (int j = 0; j < 32; ++j) {
    f32x2 pc[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float v = -P[j * DG_PP + lane + 32 * q];
      pc[q] = pack2(v, v);
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const ulonglong2 pr = *reinterpret_cast<const ulonglong2*>(P + j * DG_PP + 32 * (KQ + 1 + b) + 4 * warp);
#pragma unroll
      for (int q = 0; q <= KQ + 1 + b; ++q) {
        acc[b][0][q] = fma2(pr.x, pc[q], acc[b][0][q]);
        acc[b][1][q] = fma2(pr.y, pc[q], acc[b][1][q]);
      }
    }
  }
#pragma unroll
  for (int b = 0; b < NB; ++b)
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int q = 0; q <= KQ + 1 + b; ++q) {
        float* at = rows + (32 * b + 2 * r) * DG_SP + 32 * q;
        unpack2(acc[b][r][q], at[0], at[DG_SP]);
      }
}

// Factors the block that S (in shared memory, zeros above the diagonal, identity past the matrix) holds and stores its
// inverse T as the tile `image`.  `live`: rows of the matrix in the block (the others are padding).  `tid`: thread among the 256 of the epilogue warps.
__device__ __noinline__ void diag_block(uint8_t* image, int live, float* S, int tid, int* status) {
  float* const P0 = S + TB * DG_SP;            // TB * DG_SP is a multiple of four
  float* const Lk = P0 + 2 * 32 * DG_PP;
  float* const inv = Lk + 32 * DG_LP;
  const int lane = tid & 31, warp = tid >> 5;
  const int panel = warp == 1 || warp == 3 ? warp >> 1 : -1;   // warp 0 factors; the panel's warps are on other schedulers
  bool bad = false;
  auto store_row = [&](int r, int col, const uint32_t (&w)[3][2]) {   // columns col .. col + 3, col a multiple of four
    uint8_t* at = image + (col >> 6) * (3 * PART_BYTES) + r * 128 + ((((col & 63) >> 3) ^ (r & 7)) << 4) + (col & 4) * 2;
#pragma unroll
    for (int part = 0; part < 3; ++part) *reinterpret_cast<uint2*>(at + part * PART_BYTES) = make_uint2(w[part][0], w[part][1]);
  };
  // rows [kb, kb + 32) of the inverse are final: split and stored, zeros right of the diagonal
  auto store = [&](int kb, int first, int threads) {
    const float* P = P0 + (kb >> 5 & 1) * 32 * DG_PP;
#pragma unroll 1
    for (int e = first; e < 32 * (TB / 4); e += threads) {
      const int j = e >> 5, col = (e & 31) * 4;
      const float4 raw = *reinterpret_cast<const float4*>(P + j * DG_PP + col);
      const float t[4] = {raw.x, raw.y, raw.z, raw.w};
      uint32_t w[3][2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float x0 = col + 2 * h <= kb + j ? t[2 * h] : 0.f, x1 = col + 2 * h + 1 <= kb + j ? t[2 * h + 1] : 0.f;
#pragma unroll
        for (int part = 0; part < 3; ++part) {
          const __nv_bfloat16 b0 = __float2bfloat16_rn(x0), b1 = __float2bfloat16_rn(x1);
          w[part][h] = static_cast<uint32_t>(__bfloat16_as_ushort(b0)) | (static_cast<uint32_t>(__bfloat16_as_ushort(b1)) << 16);
          x0 -= __bfloat162float(b0);
          x1 -= __bfloat162float(b1);
        }
      }
      store_row(kb + j, col, w);
    }
  };
  for (int e = tid; e < 32 * DG_LP; e += 256) Lk[e] = 0.f;
#pragma unroll 1
  for (int kb = 0; kb < live; kb += 32) {
    epi_sync();
    float* const P = P0 + (kb >> 5 & 1) * 32 * DG_PP;
    if (warp == 0) {
      DiagRow a[1];   // entries above the diagonal: not used
      const float* from = S + (kb + lane) * DG_SP + kb;
#pragma unroll
      for (int i = 0; i < 8; ++i) a[0].g[i] = from[i];
#pragma unroll
      for (int i = 0; i < 12; ++i) a[0].v[i] = pack2(from[8 + 2 * i], from[9 + 2 * i]);
      float iv = diag_pivot(__shfl_sync(0xffffffffu, a[0].g[0], 0), bad);
#pragma unroll 1
      for (int j8 = 0; j8 < 32; j8 += 8) {
        float l[1][8];
        float* const column = Lk + j8 * DG_LP + lane;   // rows above a column's diagonal: not used
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          l[0][j] = a[0].g[j] * iv;
          // all shuffles of the column first: they share the latency of the pivot's
          float d = 0.f, row[8];
          if (j < 7) d = __shfl_sync(0xffffffffu, fmaf(-l[0][j], l[0][j], a[0].g[j < 7 ? j + 1 : 7]), j8 + j + 1);
#pragma unroll
          for (int c = j + 1; c < 8; ++c) row[c] = __shfl_sync(0xffffffffu, l[0][j], j8 + c);
          column[j * DG_LP] = l[0][j];
          if (lane == 0) inv[j8 + j] = iv;
          if (j < 7) iv = diag_pivot(d, bad);
#pragma unroll
          for (int c = j + 1; c < 8; ++c) a[0].g[c] = fmaf(-l[0][j], row[c], a[0].g[c]);
        }
        __syncwarp();
        asm volatile("barrier.cta.arrive %0, 96;" ::"r"(2 + (j8 >> 3)) : "memory");
        if (j8 == 24) break;
        diag_apply(a, l, Lk + j8 * DG_LP + j8);
        a[0].shift();
        iv = diag_pivot(__shfl_sync(0xffffffffu, a[0].g[0], j8 + 8), bad);
      }
    } else {
      if (kb > 0) store(kb - 32, tid - 32, 224);
      if (panel >= 0) {
        DiagRow v[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int block = 2 * panel + u, c = 32 * block + lane;
          const float* from = c >= kb + 32 ? S + c * DG_SP + kb : S + kb * DG_SP + c;
          const int pitch = c >= kb + 32 ? 1 : DG_SP;
          // the block's own columns of the inverse start from the identity
          auto entry = [&](int j) { return block == kb / 32 ? (j == lane ? 1.f : 0.f) : from[j * pitch]; };
#pragma unroll
          for (int i = 0; i < 8; ++i) v[u].g[i] = entry(i);
#pragma unroll
          for (int i = 0; i < 12; ++i) v[u].v[i] = pack2(entry(8 + 2 * i), entry(9 + 2 * i));
        }
#pragma unroll 1
        for (int j8 = 0; j8 < 32; j8 += 8) {
          named_bar_sync(2 + (j8 >> 3), 96);
          const float* const block = Lk + j8 * DG_LP + j8;
          float x[2][8];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 o0 = *reinterpret_cast<const float4*>(block + j * DG_LP), o1 = *reinterpret_cast<const float4*>(block + j * DG_LP + 4);
            const float o[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w}, iv = inv[j8 + j];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
              x[u][j] = v[u].g[j] * iv;
#pragma unroll
              for (int i = j + 1; i < 8; ++i) v[u].g[i] = fmaf(-x[u][j], o[i], v[u].g[i]);
            }
          }
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int j = 0; j < 8; ++j) P[(j8 + j) * DG_PP + 64 * panel + 32 * u + lane] = x[u][j];
          if (j8 == 24) break;
          diag_apply(v, x, block);
          v[0].shift();
          v[1].shift();
        }
      }
    }
    epi_sync();
    if (kb == 0)
      diag_update<0>(S, P, warp, lane);
    else if (kb == 32)
      diag_update<1>(S, P, warp, lane);
    else if (kb == 64)
      diag_update<2>(S, P, warp, lane);
  }
  const int stages = (live + 31) / 32;
  store(32 * stages - 32, tid, 256);
  constexpr uint32_t none[3][2] = {};
#pragma unroll 1
  for (int e = tid + stages * 32 * 32; e < TB * 32; e += 256) store_row(e >> 5, (e & 31) * 4, none);   // rows of padding
  if (bad && tid == 0) set_error(status, ERR_NOT_SPD);
}

// ---- the task kernel ------------------------------------------------------------------------------
// The ring holds two K blocks of six operand parts (roles), and every role of a block has a slot and an `empty` barrier of its
// own: a part is loaded again as soon as the last product that reads it is done, not when the block is.  Products are issued in
// the order (mid,mid) (lo,hi) (hi,lo) (mid,hi) (hi,mid) (hi,hi): small magnitudes first, and every role has at least a block's
// time between its release and its next use.
constexpr int TC_STAGES = 2, TC_ITEMS = 4, TC_EPI_WARPS = 8;
constexpr int TC_STAGE_BYTES = 6 * PART_BYTES;
enum : int { ROLE_A_HI = 0, ROLE_A_MID, ROLE_A_LO, ROLE_B_HI, ROLE_B_MID, ROLE_B_LO, ROLES };   // slots of a K block, in order
constexpr int TC_THREADS = 64 + 32 * TC_EPI_WARPS;
constexpr int TC_STAGING = 4096;                    // per epilogue warp
constexpr int TC_SMEM = 1024 /*alignment*/ + TC_STAGES * TC_STAGE_BYTES + TC_EPI_WARPS * TC_STAGING + 512 /*barriers, tasks*/;
static_assert(DG_SMEM <= TC_STAGES * TC_STAGE_BYTES && TC_SMEM <= 232448, "shared memory of the task kernel");

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// Orders this thread's generic accesses (global and shared) with the async proxy's (TMA, MMA operands).
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Waits until a progress word has reached `want`; `seen` remembers what was read.  Bounded in time; ends early when another
// CTA gave up.
__device__ __forceinline__ bool wait_progress(const int* word, int want, int& seen, const int* abort) {
  if (seen >= want) return true;
  seen = ld_acquire(word);
  if (seen < want) {
    const uint64_t t0 = globaltimer_ns();
    uint32_t spins = 0;
    while ((seen = ld_acquire(word)) < want)
      if ((++spins & 63) == 0 && (ld_acquire(abort) != 0 || globaltimer_ns() - t0 > B200_WAIT_NS)) return false;
  }
  proxy_fence();
  return true;
}

// Copy of `bytes` (a multiple of 16, both sides 16-byte aligned) from global to shared memory, counted on `bar`.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Warp-collective store of 32 lanes x 32 consecutive fp32 columns to tensor memory.
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]),
      "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]),
      "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// True on all 256 threads when `bad` is set on any of them.
__device__ __forceinline__ bool epi_any(bool bad) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, 256, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r)
      : "r"(static_cast<uint32_t>(bad))
      : "memory");
  return r != 0;
}

__device__ __forceinline__ float4 lds4(uint32_t at) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ float lds(uint32_t at) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
  return v;
}

// A warp's 32 x 32 patch of fp32 values in its staging memory: rows of 128 bytes, the 16-byte pieces of a row exchanged.
__device__ __forceinline__ void stage_patch(const float* v, uint8_t* stg, int lane) {
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 8; ++c)
    *reinterpret_cast<float4*>(stg + lane * 128 + ((c ^ (lane & 7)) << 4)) = make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
  __syncwarp();
}
// Three-way split of a staged patch, columns [32 h, 32 h + 32) of an image whose first row is at `base` (global or shared memory).
// A lane splits eight values at a time.  Code that runs once per tile is bound by instruction fetch (unrolled over the 64 values
// of a row per thread it took 5 us to split and store a tile), so it is a function.
__device__ __noinline__ void split_patch(uint32_t stg, uint8_t* base, int h, int lane) {
  const int g = lane & 3;
#pragma unroll 1
  for (int i = 0; i < 4; i += 2) {
    float v[2][8];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = (i + u) * 8 + (lane >> 2);
      const float4 lo = lds4(stg + r * 128 + (((2 * g) ^ (r & 7)) << 4)), hi = lds4(stg + r * 128 + (((2 * g + 1) ^ (r & 7)) << 4));
      v[u][0] = lo.x, v[u][1] = lo.y, v[u][2] = lo.z, v[u][3] = lo.w, v[u][4] = hi.x, v[u][5] = hi.y, v[u][6] = hi.z, v[u][7] = hi.w;
    }
#pragma unroll
    for (int part = 0; part < 3; ++part) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = (i + u) * 8 + (lane >> 2);
        uint32_t w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          float &x0 = v[u][2 * k], &x1 = v[u][2 * k + 1];
          const __nv_bfloat162 b = __floats2bfloat162_rn(x0, x1);
          w[k] = *reinterpret_cast<const uint32_t*>(&b);
          x0 -= __uint_as_float(w[k] << 16);
          x1 -= __uint_as_float(w[k] & 0xffff0000u);
        }
        *reinterpret_cast<uint4*>(base + part * PART_BYTES + r * 128 + (((4 * h + g) ^ (r & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
}
// Stores a staged patch (element (r, c) at r * 32 + (c ^ r)) to out[row0 ..][col0 ..], then its mirror image, eight loads in
// flight.  Stores that alternate between the two take twice as long (9600 clocks a tile, in two passes 5100).
__device__ __noinline__ void store_patch(uint32_t stg, float* out, int n, int row0, int col0, bool diag, int lane) {
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    const int first = pass == 0 ? row0 : col0, at = (pass == 0 ? col0 : row0) + lane;
#pragma unroll 1
    for (int i = 0; i < 32; i += 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        v[u] = lds(stg + (pass == 0 ? (i + u) * 32 + (lane ^ (i + u)) : lane * 32 + ((i + u) ^ lane)) * 4);
      float* to = out + static_cast<size_t>(first + i) * n + at;
#pragma unroll
      for (int u = 0; u < 8; ++u, to += n) {
        const int line = first + i + u;   // row of the output; the diagonal tile keeps its lower triangle
        if (line < n && at < n && (!diag || (pass == 0 ? at <= line : line < at))) *to = v[u];
      }
    }
  }
}

__global__ void __launch_bounds__(TC_THREADS, 1)
tc_tasks_kernel(const TcMat* __restrict__ mats, const Task* __restrict__ tasks, int n_tasks, const float* __restrict__ damping,
                int* ctrl, int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* staging = smem + TC_STAGES * TC_STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(staging + TC_EPI_WARPS * TC_STAGING);
  uint64_t* empty_bar = full_bar + TC_STAGES * 3;   // full: (mid, mid), (A lo, B hi), (A hi, B lo) of a block; empty: its roles
  uint64_t* acc_full = empty_bar + TC_STAGES * ROLES;
  uint64_t* acc_empty = acc_full + 2;
  uint64_t* item_full = acc_empty + 2;
  uint64_t* item_empty = item_full + TC_ITEMS;
  uint64_t* operand_bar = item_empty + TC_ITEMS;   // the epilogue's half of a stage of a second product is written
  uint64_t* diag_bar = operand_bar + 2;            // the epilogue has left the ring after a diagonal block
  Task* items = reinterpret_cast<Task*>(diag_bar + 2);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(items + TC_ITEMS);
  int* const next_task = ctrl;
  int* const abort = ctrl + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int b = 0; b < TC_STAGES * 3; ++b) mbar_init(&full_bar[b], 2);
    for (int b = 0; b < TC_STAGES * ROLES; ++b) mbar_init(&empty_bar[b], 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], TC_EPI_WARPS);
      mbar_init(&operand_bar[b], 4);   // the four warps that hold this K block of the operand
    }
    for (int b = 0; b < TC_ITEMS; ++b) {
      mbar_init(&item_full[b], 1);
      mbar_init(&item_empty[b], 1 + TC_EPI_WARPS);
    }
    mbar_init(diag_bar, 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);   // two accumulators and a tile of A
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  auto give_up = [&](int code) {
    set_error(status, code);
    atomicExch(abort, 1);
  };

  if (warp == 0) {
    // ---- claims tasks, waits for their operands, loads them
    if (lane == 0) {
      uint32_t it = 0, diags = 0;
      bool ok = true;
      for (uint32_t tk = 0; ok; ++tk) {
        const int idx = atomicAdd(next_task, 1);
        Task t;
        if (idx < n_tasks)
          t = tasks[idx];
        else
          t = {0, TASK_END, 0, 0};
        const uint32_t slot = tk % TC_ITEMS;
        if (!mbar_wait(&item_empty[slot], ((tk / TC_ITEMS) & 1) ^ 1)) {
          give_up(ERR_WAIT_EMPTY);
          break;
        }
        items[slot] = t;
        mbar_arrive(&item_full[slot]);
        if (t.kind == TASK_END) break;
        const TcMat& M = mats[t.mat];
        const int i0 = t.i * TB, j0 = t.j * TB;
        const bool two = t.kind == TASK_FACTOR || t.kind == TASK_INV;   // a second product follows
        const bool shared_ab = t.kind == TASK_DIAG || (t.kind == TASK_OUT && t.i == t.j);
        const int k0 = t.kind == TASK_INV ? j0 : (t.kind == TASK_OUT ? i0 : 0);
        // progress of the two operands: L by rows, X by columns
        const int* wa = t.kind == TASK_OUT ? M.col_x + t.i : M.row_l + t.i;
        const int* wb = t.kind == TASK_INV || t.kind == TASK_OUT ? M.col_x + t.j : M.row_l + t.j;
        int seen_a = -1, seen_b = -1;
        const int nkb = task_blocks(t.kind, t.i, t.j, M.n), total = nkb + (two ? 2 : 0);
        const bool a_k = t.kind != TASK_OUT, b_k = t.kind == TASK_FACTOR;   // operands of the sum: rows of L, columns of X
        for (int kb = 0; kb < total && ok; ++kb, ++it) {
          const uint32_t s = it % TC_STAGES, parity = ((it / TC_STAGES) & 1) ^ 1;
          const uint8_t *src_a = nullptr, *src_b = nullptr;   // null: nothing to load (shared, or written by the epilogue)
          bool major_a = a_k, major_b = b_k;
          if (kb < nkb) {
            const int k = k0 + kb * G2_BK, panel = k / TB, hb = (k / G2_BK) & 1;   // hb: half of the panel
            if (!wait_progress(wa, panel + 1, seen_a, abort) || (!shared_ab && !wait_progress(wb, panel + 1, seen_b, abort))) {
              give_up(ERR_WAIT_FULL);
              ok = false;
              break;
            }
            src_a = a_k ? below_at(M.L, t.i, panel) + hb * 3 * PART_BYTES : tile_at(M.X, panel, t.i) + hb * (PART_BYTES / 2);
            if (!shared_ab)
              src_b = b_k ? below_at(M.L, t.j, panel) + hb * 3 * PART_BYTES : tile_at(M.X, panel, t.j) + hb * (PART_BYTES / 2);
          } else {   // T, the other operand of the second product
            const int d = t.kind == TASK_FACTOR ? t.j : t.i;
            int seen = -1;
            if (!wait_progress(M.col_x + d, d + 1, seen, abort)) {
              give_up(ERR_WAIT_FULL);
              ok = false;
              break;
            }
            (t.kind == TASK_FACTOR ? src_b : src_a) = tile_at(M.X, d, d) + (kb - nkb) * 3 * PART_BYTES;
            major_a = major_b = true;
          }
          // roles in the order in which the block before the last releases them
          constexpr int ORDER[ROLES] = {ROLE_A_LO, ROLE_B_LO, ROLE_A_MID, ROLE_B_MID, ROLE_B_HI, ROLE_A_HI};
          constexpr int GROUP[ROLES] = {2, 0, 1, 1, 0, 2};   // full barrier of a role
#pragma unroll
          for (int o = 0; o < ROLES; ++o) {
            const int role = ORDER[o], part = role % 3;
            if (ok && !mbar_wait(&empty_bar[s * ROLES + role], parity)) {
              give_up(ERR_WAIT_EMPTY);
              ok = false;
            }
            if (!ok) break;
            const uint8_t* src = role < 3 ? src_a : src_b;
            const bool k_major = role < 3 ? major_a : major_b;
            uint64_t* const bar = &full_bar[s * 3 + GROUP[role]];
            uint8_t* const dst = smem + s * TC_STAGE_BYTES + role * PART_BYTES;
            if (src == nullptr) {
              mbar_arrive(bar);
              continue;
            }
            mbar_expect_tx(bar, PART_BYTES);
            if (k_major) {
              bulk_load(dst, src + part * PART_BYTES, PART_BYTES, bar);
            } else {   // 64 rows of both halves
              bulk_load(dst, src + part * PART_BYTES, PART_BYTES / 2, bar);
              bulk_load(dst + PART_BYTES / 2, src + (3 + part) * PART_BYTES, PART_BYTES / 2, bar);
            }
          }
        }
        if (ok && t.kind == TASK_DIAG) {   // the diagonal block is factored in the ring's memory
          if (!mbar_wait(diag_bar, diags & 1)) {
            give_up(ERR_WAIT_EMPTY);
            ok = false;
          }
          ++diags;
        }
      }
      if (!ok) {   // copies that are still in flight get a bounded chance to land before teardown
        for (uint32_t jt = it < 2 ? 0 : it - 2; jt <= it; ++jt)   // the last one may not have been loaded in full
          for (int g = 0; g < 3; ++g) mbar_wait(&full_bar[jt % TC_STAGES * 3 + g], (jt / TC_STAGES) & 1);
      }
    }
  } else if (warp == 1) {
    // ---- issues the products.  The whole warp runs the loop and one lane issues, so that addresses stay in uniform registers;
    // descriptors are a base and constants.  A loop of one lane that builds every descriptor needs 2206 clocks for the 24
    // products of a K block, this one 1587; the tensor core needs 1536.
    const bool lead = elect_one();
    uint32_t it = 0, seconds = 0;
    bool ok = true;
    for (uint32_t tk = 0; ok; ++tk) {
      const uint32_t slot = tk % TC_ITEMS;
      if (!mbar_wait(&item_full[slot], (tk / TC_ITEMS) & 1)) {
        give_up(ERR_WAIT_FULL);
        break;
      }
      const Task t = items[slot];
      __syncwarp();
      if (lead) mbar_arrive(&item_empty[slot]);
      if (t.kind == TASK_END) break;
      const bool two = t.kind == TASK_FACTOR || t.kind == TASK_INV;
      const bool shared_ab = t.kind == TASK_DIAG || (t.kind == TASK_OUT && t.i == t.j);
      const bool a_k = t.kind != TASK_OUT;                                // K-major operands
      const bool b_k = t.kind == TASK_DIAG || t.kind == TASK_FACTOR;      // ... in both products: L and T, X and W are alike
      const uint32_t idesc = make_idesc_bf16(TB, TB, !a_k, !b_k);
      // 16 elements of K: 32 bytes of a K-major row, 16 rows of 128 bytes of an MN-major operand
      const uint32_t step_a = a_k ? 2 : 128, step_b = b_k ? 2 : 128;
      const uint64_t desc_a = make_smem_desc_sw128(smem_u32(smem), a_k ? 16 : G2_BK * 128, 1024);
      const uint64_t desc_b = make_smem_desc_sw128(smem_u32(smem) + (shared_ab ? 0 : 3 * PART_BYTES), b_k ? 16 : G2_BK * 128, 1024);
      const int nkb = task_blocks(t.kind, t.i, t.j, mats[t.mat].n), total = nkb + (two ? 2 : 0);
      for (int kb = 0; kb < total; ++kb, ++it) {
        const uint32_t ab = it & 1, s = it % TC_STAGES;
        ok = mbar_wait(&acc_empty[ab], ((it >> 1) & 1) ^ 1) && (kb < nkb || mbar_wait(&operand_bar[kb - nkb], seconds & 1));
        const uint32_t tacc = tmem_base + ab * TB;
        constexpr int PART_A[6] = {1, 2, 0, 1, 0, 0};   // (mid,mid) (lo,hi) (hi,lo) (mid,hi) (hi,mid) (hi,hi)
        constexpr int PART_B[6] = {1, 0, 2, 0, 1, 0};
        constexpr int RELEASE[6] = {-1, ROLE_A_LO, ROLE_B_LO, ROLE_A_MID, ROLE_B_MID, ROLE_A_HI};   // done with after the product
#pragma unroll
        for (int pr = 0; pr < 6; ++pr) {
          if (pr < 3) {
            ok = ok && mbar_wait(&full_bar[s * 3 + pr], (it / TC_STAGES) & 1);
            // where A is both operands, (lo,hi) reads what (hi,lo) waits for
            if (pr == 1 && shared_ab) ok = ok && mbar_wait(&full_bar[s * 3 + 2], (it / TC_STAGES) & 1);
            if (!ok) break;
            tc_fence_after_sync();
          }
          const uint64_t da = desc_a + ((s * TC_STAGE_BYTES + PART_A[pr] * PART_BYTES) >> 4);
          const uint64_t db = desc_b + ((s * TC_STAGE_BYTES + PART_B[pr] * PART_BYTES) >> 4);
#pragma unroll
          for (int k = 0; k < G2_BK / 16; ++k)
            if (lead) umma_bf16(tacc, da + k * step_a, db + k * step_b, idesc, (pr | k) ? 1u : 0u);
          if (RELEASE[pr] >= 0 && !shared_ab && lead) umma_commit(&empty_bar[s * ROLES + RELEASE[pr]]);
        }
        if (!ok) {
          give_up(ERR_WAIT_FULL);
          break;
        }
        if (lead) {
          if (shared_ab)   // the parts of A are both operands: all roles are free at the end
            for (int role = 0; role < ROLES; ++role) umma_commit(&empty_bar[s * ROLES + role]);
          else
            umma_commit(&empty_bar[s * ROLES + ROLE_B_HI]);
          umma_commit(&acc_full[ab]);
        }
        __syncwarp();
      }
      if (two) ++seconds;
    }
  } else {
    // ---- epilogue: sums, splits, diagonal blocks, stores
    const int tid = threadIdx.x - 64, ew = warp - 2;
    const int q = warp & 3, half = ew >> 2;      // TMEM lanes [32 q, 32 q + 32), columns [64 half, 64 half + 64) of a tile
    const int row = q * 32 + lane;               // this thread's row of a tile
    uint8_t* const stg = staging + ew * TC_STAGING;
    float* const stgf = reinterpret_cast<float*>(stg);
    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + half * 64;
    uint32_t it = 0;
    bool ok = true;
    // A wait that runs out (`ok` false) only stops further waits: all warps pass the barriers of the task and leave together.
    for (uint32_t tk = 0;; ++tk) {
      const uint32_t slot = tk % TC_ITEMS;
      if (ok && !mbar_wait(&item_full[slot], (tk / TC_ITEMS) & 1)) {
        ok = false;
        give_up(ERR_WAIT_FULL);
      }
      if (epi_any(!ok)) break;
      const Task t = items[slot];
      __syncwarp();
      if (lane == 0) mbar_arrive(&item_empty[slot]);
      if (t.kind == TASK_END) break;
      const TcMat& M = mats[t.mat];
      const int n = M.n, i0 = t.i * TB, j0 = t.j * TB;
      const int row0 = i0 + q * 32, col0 = j0 + half * 64;   // of this warp's 32 x 64 patch
      const int nkb = task_blocks(t.kind, t.i, t.j, n);
      float run[64];
      if (t.kind == TASK_DIAG || t.kind == TASK_FACTOR) {
        // A + damping I waits in tensor memory: rows are read along the lanes and turned in shared memory, 32 loads in flight
        const float* A = M.A;
        const float d = damping[M.orig];
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {
          const int gc = col0 + 32 * h + lane;
          float v[32];
#pragma unroll
          for (int r = 0; r < 32; ++r)
            v[r] = row0 + r < n && gc < n ? __ldg(A + static_cast<size_t>(row0 + r) * M.lda + gc) : 0.f;
          __syncwarp();
#pragma unroll
          for (int r = 0; r < 32; ++r) stgf[r * 32 + (lane ^ r)] = row0 + r == gc ? v[r] + d : v[r];
          __syncwarp();
          uint32_t w[32];
#pragma unroll
          for (int c = 0; c < 32; ++c) w[c] = __float_as_uint(stgf[lane * 32 + (c ^ lane)]);
          tmem_st_32x32(taddr + 2 * TB + 32 * h, w);
        }
        tmem_st_wait();
      }
#pragma unroll
      for (int c = 0; c < 64; ++c) run[c] = 0.f;
      auto add_blocks = [&](int count) {
        for (int kb = 0; kb < count; ++kb, ++it) {
          const uint32_t ab = it & 1;
          if (ok && !mbar_wait(&acc_full[ab], (it >> 1) & 1)) {
            ok = false;
            give_up(ERR_WAIT_ACC);
          }
          __syncwarp();
          tc_fence_after_sync();
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t w[32];
            tmem_ld_32x32(taddr + ab * TB + 32 * h, w);
            tmem_ld_wait();
            if (h == 1) {
              tc_fence_before_sync();
              __syncwarp();
              if (lane == 0) mbar_arrive(&acc_empty[ab]);
            }
#pragma unroll
            for (int c = 0; c < 32; ++c) run[32 * h + c] += __uint_as_float(w[c]);
          }
        }
      };
      add_blocks(nkb);
      if (t.kind == TASK_DIAG || t.kind == TASK_FACTOR) {   // S = A - sum
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t w[32];
          tmem_ld_32x32(taddr + 2 * TB + 32 * h, w);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 32; ++c) run[32 * h + c] = __uint_as_float(w[c]) - run[32 * h + c];
        }
      }

      if (t.kind == TASK_DIAG) {
        // every product that read the ring is done (its accumulator was read) and the producer waits
        float* S = reinterpret_cast<float*>(smem);
        const int live = min(TB, n - i0);
#pragma unroll
        for (int c = 0; c < 64; ++c) S[row * DG_SP + half * 64 + c] = half * 64 + c <= row ? run[c] : 0.f;
        if (row >= live) {   // identity padding keeps the block factorisable
#pragma unroll 1
          for (int c = half * 64; c < half * 64 + 64; ++c) S[row * DG_SP + c] = row == c ? 1.f : 0.f;
        }
        diag_block(tile_at(M.X, t.j, t.j), live, S, tid, status);
        proxy_fence();
        epi_sync();
        if (tid == 0) {
          st_release(M.col_x + t.j, t.j + 1);
          mbar_arrive(diag_bar);
        }
        continue;
      }
      if (t.kind == TASK_OUT) {
        // lower tiles; diagonal tiles keep their lower triangle; both are mirrored, so the result is exactly symmetric
        const bool diag = t.i == t.j;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          __syncwarp();
#pragma unroll
          for (int c = 0; c < 32; ++c) stgf[lane * 32 + (c ^ lane)] = run[32 * h + c];
          __syncwarp();
          store_patch(smem_u32(stgf), M.out, n, row0, col0 + 32 * h, diag, lane);
        }
        continue;
      }

      // second product: the sum is the operand.  FACTOR: S (A operand, K-major), this warp's columns are K block `half`;
      // INV: W (B operand, MN-major), this warp's rows are in K block q / 2.
      const int kb2 = t.kind == TASK_FACTOR ? half : q >> 1;
      const uint32_t it2 = it + kb2, s2 = it2 % TC_STAGES;
      for (int part = 0; part < 3; ++part)
        if (ok && !mbar_wait(&empty_bar[s2 * ROLES + (t.kind == TASK_FACTOR ? ROLE_A_HI : ROLE_B_HI) + part], ((it2 / TC_STAGES) & 1) ^ 1)) {
          ok = false;
          give_up(ERR_WAIT_EMPTY);
        }
      __syncwarp();
      uint8_t* const stage = smem + s2 * TC_STAGE_BYTES;
      uint8_t* const operand = t.kind == TASK_FACTOR ? stage + q * 32 * 128
                                                     : stage + 3 * PART_BYTES + half * (G2_BK * 128) + (q & 1) * 32 * 128;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        stage_patch(run + 32 * h, stg, lane);
        split_patch(smem_u32(stg), operand, h, lane);
      }
      proxy_fence();
      __syncwarp();
      if (lane == 0) mbar_arrive(&operand_bar[kb2]);
#pragma unroll
      for (int c = 0; c < 64; ++c) run[c] = 0.f;
      add_blocks(2);
      if (t.kind == TASK_INV) {
#pragma unroll
        for (int c = 0; c < 64; ++c) run[c] = -run[c];
      }
      // parts of the result: this warp's 32 rows of a half are 4 KiB in a row
      uint8_t* const image = (t.kind == TASK_FACTOR ? below_at(M.L, t.i, t.j) : tile_at(M.X, t.i, t.j)) + half * (3 * PART_BYTES) + q * 32 * 128;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        stage_patch(run + 32 * h, stg, lane);
        split_patch(smem_u32(stg), image, h, lane);
      }
      proxy_fence();
      epi_sync();   // the release of one thread covers what the others stored before the barrier
      if (tid == 0) {
        if (t.kind == TASK_FACTOR)
          st_release(M.row_l + t.i, t.j + 1);
        else
          st_release(M.col_x + t.j, t.i + 1);
      }
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
  }
}

struct Prepared {
  std::vector<const void*> key;
  at::Tensor splits;     // tiles of L and X of all matrices
  at::Tensor d_mats;     // TcMat table
  at::Tensor d_tasks;    // Task list
  at::Tensor d_ctrl;     // claim counter, abort word, progress words: zeroed by every call
  int n_tasks = 0;
  GraphPins pins;
};

std::mutex g_cache_mutex;
// four sets of matrices beside those that graphs refer to; never destroyed (see PreparedCache)
PreparedCache<Prepared, 4>& g_cache = *new PreparedCache<Prepared, 4>;

// The task list of matrices of `sizes` for `ctas` CTAs.  Any order in which a task follows what it needs is correct; this one
// is made for speed.  Time is cut into slots of one step of a chain (DIAG, FACTOR of the next row, last panel of the next
// DIAG).  In a slot every matrix may take one step, and the longest remaining chains always do; shorter ones join while the
// slot has room, and OUT tiles, which nothing waits for, fill the rest.  The durations are rough (a step takes 34 us, a diagonal block 22)
// and the list does not depend on them much: STEP_US from 20 to 100, DIAG_US from 15 to 45 and AHEAD from 4 to 200 gave 256.5 - 256.9 us for
// six factors up to 784 (257.8 with nothing ahead) and 3.47 - 3.65 ms, in no order, for ResNet-50's 107.
std::vector<Task> make_tasks(const std::vector<int>& sizes, int ctas) {
  constexpr int STEP_US = 35, BLOCK_US = 1, TILE_US = 5, DIAG_US = 28, AHEAD = 12;
  const int count = static_cast<int>(sizes.size());
  std::vector<int> nb(count), step(count, 0), order(count), out_i(count, 0), out_j(count, 0), started(count, 0);
  for (int m = 0; m < count; ++m) {
    nb[m] = (sizes[m] + TB - 1) / TB;
    order[m] = m;
  }
  std::vector<Task> tasks;
  for (int m = 0; m < count; ++m) tasks.push_back({m, TASK_DIAG, 0, 0});
  std::stable_sort(tasks.begin(), tasks.end(), [&](const Task& a, const Task& b) { return nb[a.mat] > nb[b.mat]; });
  int left = count;
  const long long room = static_cast<long long>(ctas) * STEP_US;
  std::vector<int> taken;
  while (left > 0) {
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return nb[a] - step[a] > nb[b] - step[b]; });
    const int longest = nb[order[0]] - step[order[0]];
    long long used = 0;
    taken.clear();
    for (int m : order) {
      if (step[m] >= nb[m]) continue;
      const int j = step[m];
      const long long work = DIAG_US + 2 * BLOCK_US * j + static_cast<long long>(nb[m] - j - 1) * (2 * BLOCK_US * j + TILE_US) +
                             static_cast<long long>(j) * (TILE_US + BLOCK_US * (j + 1));
      if (nb[m] - j != longest && used + work > room) continue;
      used += work;
      taken.push_back(m);
    }
    int ahead = 0;
    for (int m : taken) {
      const int j = step[m];
      for (int i = started[m] > j ? j + 2 : j + 1; i < nb[m]; ++i) {
        tasks.push_back({m, TASK_FACTOR, i, j});
        if (i == j + 1) tasks.push_back({m, TASK_DIAG, i, i});
      }
      // the next step's first tile and diagonal block, so that they are not behind the rest of this slot
      if (4 * (nb[m] - j) >= 3 * longest && ahead < AHEAD && j + 2 < nb[m]) {
        tasks.push_back({m, TASK_FACTOR, j + 2, j + 1});
        tasks.push_back({m, TASK_DIAG, j + 2, j + 2});
        started[m] = j + 2;   // steps below this one have them
        ++ahead;
      }
    }
    for (int m : taken)
      for (int c = 0; c < step[m]; ++c) tasks.push_back({m, TASK_INV, step[m], c});
    for (int m : taken) ++step[m];
    for (int m : order) {   // OUT tiles of matrices whose chain has ended
      if (step[m] < nb[m] || out_i[m] >= nb[m]) continue;
      while (out_i[m] < nb[m] && (used < room || longest <= 1)) {
        tasks.push_back({m, TASK_OUT, out_i[m], out_j[m]});
        used += 2 * BLOCK_US * (nb[m] - out_i[m]) + TILE_US;
        if (++out_j[m] > out_i[m]) {
          ++out_i[m];
          out_j[m] = 0;
        }
      }
    }
    left = 0;
    for (int m = 0; m < count; ++m) left += out_i[m] < nb[m];
  }
  return tasks;
}

}  // namespace

void chol_inverse_tc(std::vector<at::Tensor> mats, std::vector<at::Tensor> outs, at::Tensor damping) {
  const int count = static_cast<int>(mats.size());
  TORCH_CHECK(count > 0 && outs.size() == mats.size(), "mats and outs must have the same length");
  TORCH_CHECK(damping.is_cuda() && damping.scalar_type() == at::kFloat && damping.is_contiguous() &&
                  damping.numel() == count, "damping must be a CUDA fp32 vector with one entry per matrix");
  const int dev = mats[0].get_device();
  c10::cuda::CUDAGuard guard(dev);
  const auto current = at::cuda::getCurrentCUDAStream(dev);
  const cudaStream_t stream = current.stream();
  std::vector<const void*> key;
  key.reserve(4 * count + 1);
  key.push_back(reinterpret_cast<const void*>(static_cast<intptr_t>(dev)));
  for (int i = 0; i < count; ++i) {
    const at::Tensor& a = mats[i];
    const at::Tensor& o = outs[i];
    TORCH_CHECK(a.is_cuda() && a.scalar_type() == at::kFloat && a.dim() == 2 && a.size(0) == a.size(1) &&
                    a.stride(1) == 1 && a.size(0) > 0, "matrices must be square fp32 CUDA tensors with unit column stride");
    TORCH_CHECK(o.is_cuda() && o.scalar_type() == at::kFloat && o.is_contiguous() && o.sizes() == a.sizes(),
                "outputs must be contiguous fp32 tensors of the same shape");
    TORCH_CHECK(o.data_ptr() != a.data_ptr(), "the inverse cannot be written over its input");
    TORCH_CHECK(a.size(0) < (1 << 24), "matrix too large");
    key.push_back(a.data_ptr());
    key.push_back(o.data_ptr());
    key.push_back(reinterpret_cast<const void*>(static_cast<intptr_t>(a.size(0))));
    key.push_back(reinterpret_cast<const void*>(static_cast<intptr_t>(a.stride(0))));
  }

  std::lock_guard<std::mutex> lock(g_cache_mutex);
  Prepared* prep = g_cache.find(key);
  if (prep == nullptr) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    B200_CUDA_CHECK(cudaStreamIsCapturing(stream, &cap));
    TORCH_CHECK(cap == cudaStreamCaptureStatusNone, "the first grouped inverse of a set of matrices builds its "
                "tables and cannot run inside a CUDA graph capture; call it once before capturing");
    Prepared P;
    P.key = key;
    int64_t total = 0, words = 2;
    std::vector<int64_t> base(count);
    std::vector<int> sizes(count);
    for (int i = 0; i < count; ++i) {
      const int64_t nb = (mats[i].size(0) + TB - 1) / TB;
      sizes[i] = static_cast<int>(mats[i].size(0));
      base[i] = total;
      total += nb * nb * TILE_BYTES;   // X with, L without the diagonal
      words += 2 * nb;
    }
    P.splits = at::empty({total}, at::TensorOptions().dtype(at::kByte).device(at::kCUDA, dev));
    P.d_ctrl = at::empty({words}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, dev));
    uint8_t* sp = P.splits.data_ptr<uint8_t>();
    TORCH_CHECK((reinterpret_cast<uintptr_t>(sp) & 15) == 0, "split buffers are not 16-byte aligned");
    int* progress = P.d_ctrl.data_ptr<int>() + 2;
    std::vector<TcMat> host(count);
    for (int i = 0; i < count; ++i) {
      TcMat& M = host[i];
      std::memset(&M, 0, sizeof(M));
      M.A = mats[i].data_ptr<float>();
      M.lda = static_cast<int>(mats[i].stride(0));
      M.out = outs[i].data_ptr<float>();
      M.n = sizes[i];
      M.nb = (M.n + TB - 1) / TB;
      M.orig = i;
      M.row_l = progress;
      M.col_x = progress + M.nb;
      progress += 2 * M.nb;
      M.L = sp + base[i];
      M.X = M.L + static_cast<size_t>(M.nb) * (M.nb - 1) / 2 * TILE_BYTES;
    }
    const std::vector<Task> tasks = make_tasks(sizes, g2_sm_count(dev));
    P.n_tasks = static_cast<int>(tasks.size());
    auto upload = [&](const void* src, size_t bytes) {
      at::Tensor hostt = at::empty({static_cast<int64_t>(bytes)}, at::TensorOptions().dtype(at::kByte).pinned_memory(true));
      std::memcpy(hostt.data_ptr(), src, bytes);
      at::Tensor d = hostt.to(at::Device(at::kCUDA, dev));
      return d;
    };
    P.d_mats = upload(host.data(), host.size() * sizeof(TcMat));
    P.d_tasks = upload(tasks.data(), tasks.size() * sizeof(Task));
    B200_CUDA_CHECK(cudaStreamSynchronize(stream));  // the pinned staging buffers are released after this
    prep = g_cache.insert(std::move(P));
  }
  prep->pins.use(current, {prep->splits, prep->d_mats, prep->d_tasks, prep->d_ctrl});

  int* ctrl = prep->d_ctrl.data_ptr<int>();
  B200_CUDA_CHECK(cudaMemsetAsync(ctrl, 0, prep->d_ctrl.numel() * sizeof(int), stream));
  B200_CUDA_CHECK(cudaFuncSetAttribute(tc_tasks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM));
  tc_tasks_kernel<<<std::min(prep->n_tasks, g2_sm_count(dev)), TC_THREADS, TC_SMEM, stream>>>(
      reinterpret_cast<const TcMat*>(prep->d_mats.data_ptr()), reinterpret_cast<const Task*>(prep->d_tasks.data_ptr()),
      prep->n_tasks, damping.data_ptr<float>(), ctrl, device_state(dev).status.data_ptr<int>());
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
}

// Drops the cached tables and split buffers of the tensor-core inverse that no captured graph refers to.
void chol_inverse_tc_clear_cache() {
  std::lock_guard<std::mutex> lock(g_cache_mutex);
  g_cache.drop_idle();
}

// (entries, entries that captured graphs refer to)
std::pair<int64_t, int64_t> chol_inverse_tc_cache_info() {
  std::lock_guard<std::mutex> lock(g_cache_mutex);
  return {static_cast<int64_t>(g_cache.size()), static_cast<int64_t>(g_cache.pinned())};
}

}  // namespace b200
