// Input-side Kronecker factor of a stride-1 convolution without its patch matrix.
//
//     out = scale * M^T M (+ beta * out),   M [n * ho * wo, c * kh * kw] the patches of x
//
// (asdl/utils.py:51-88 and asdl/operations/conv.py:80-88 build M with unfold.)  The block of M^T M of two taps t >= t' is a sum
// of x[q + d] x[q]^T over the input pixels q with d = t - t', and depends on the taps themselves only through which q count: the
// output pixels o with o + t' - p = q.  A k x k filter has ((2k - 1)^2 + 1) / 2 differences d (13 for 3 x 3, 41 for 5 x 5) instead of
// kk (kk + 1) / 2 blocks (45, 325).  So
//
//     block(t, t') = core_d + (edge rows) + (edge columns) + (edge pixels) that are in the window of t and t',
//
// where core_d has the pairs of pixels that are in the windows of all taps at the difference d, and every image row, column or
// pixel that is in some of them only is a product of its own.  These are few and short (3 x 3, padding 1: the first and last row for
// d = (0, dx), the first and last column for d = (dy, 0), the corners for d = 0).  All terms are sums of products, nothing is taken
// off: a tap that sees nothing but zeros has exact zeros, a diagonal entry is never negative, and an entry's error is relative to
// what its own window holds.  (Sums over all pixels, less the edges, took as long and kept the rounding of the larger sum.)
//
//   stage     x -> bf16 (hi, or hi and lo) rows [pixel, channel], ordered image row, image, column, with kw - 1 zeros behind each
//             image's row: a difference d is a constant offset of rows, and edge rows are K ranges.  Products that leave edge columns
//             out take the right or left pixels from a copy with zeros there.  The edge columns and the pixels at their ends are
//             staged once more by themselves, as K ranges of their own;
//   products  128 x 128 tiles of 64-channel chunks.  Each chunk is a TMA box with a row offset of its own, so a tile holds the
//             chunks of several differences.  Where one chunk holds all channels, B is two chunks too, the second with the row
//             before: it gives the difference next to that of the first;
//             a CTA takes one K range of a tile; hi and lo parts are loaded once for the three part products, of which (lo, hi) and
//             (hi, lo) have an accumulator of their own.  The tensor core truncates with every addition, so few of them should meet a
//             large sum: with one accumulator and ranges of any length 32 x 96 x 32 x 32, 5 x 5, had an error of 1.0e-4 against 64 bits
//             (patches in three segments 9.7e-5), with the second accumulator 4.5e-5, with ranges of 128 K blocks besides 6.8e-6;
//   reduce    sums the K ranges in order;
//   assemble  adds the terms of each entry and the moving average, writes entry and mirror image.
//
// The patch matrix was written and read before: 128 x 64 x 32 x 32 fp32, 3 x 3: 302 MB, 15 tiles of K = 131072 with three part
// products, each loading both operands, 337 -> 80 us (staging 20, products 44, reduction 4, assembly 9); 32 x 256 x 14 x 14
// bf16: 63 -> 41 us (5, 18, 4, 9).  The fp32 products are bound by what L2 delivers (64 KiB per K block of 768 tensor clocks), the
// staging by memory: each pixel is read once and written to all its places; strips that read their own pixels, 32 bytes of a
// sector per channel, and copies of them took 11 us more.  Masking the edge columns in shared memory instead of in a copy
// held the ring's stages too long (products 44 -> 60).
// Non-finite inputs give non-finite diagonal entries for all taps that see them, as patches do, and stay in their channels' rows and
// columns; which other taps of the channel meet them there depends on where zeros are multiplied.
#include <cstring>

#include "chained_launch.h"
#include "gemm2_host.h"

namespace b200 {

namespace {

constexpr int CG_MAX_K = 5;
constexpr int CG_MAX_PRODUCTS = 1024, CG_MAX_TERMS = 8192, CG_MAX_TILES = 32768;
constexpr int CG_TILE = 128 * 128;          // floats of a tile

// Staged rows: lead, copies of the images, column strips, pixel strips.  Every part is a multiple of 64 rows.
struct StageShape {
  int n, c, h, w, wp;                       // wp: with the zeros behind
  int ey, ex;                               // edge rows / columns on each side
  int lead, row_len, main_len, copies;      // rows before the images, of an image row, of a copy; copies
  int cols0, col_len, pix0, pix_len;        // first row of the strips, rows of a strip
  int total;
  long long sn, sc, sh, sw;                 // element strides of x
};

// Image row or column of edge strip e of 2 * edges: the first `edges` ones, then the last; and back.
__host__ __device__ inline int edge_at(int e, int edges, int extent) { return e < edges ? e : extent - 2 * edges + e; }
__host__ __device__ inline int edge_of(int at, int edges, int extent) { return at < edges ? at : at - (extent - 2 * edges); }

// Columns [lo, hi) that copy v of the images keeps: all, those of the right pixel at distance v - 1, those of the left pixel at
// distance v - ex of a pair whose left pixel is no edge column on the left and whose right pixel is none on the right.
__host__ __device__ inline void copy_columns(int v, int ex, int w, int& lo, int& hi) {
  lo = v == 0 ? 0 : (v <= ex ? ex : 2 * ex - v);
  hi = v == 0 ? w : (v <= ex ? w - ex + v - 1 : w - ex);
}
__host__ __device__ inline int copy_of(int dx, int ex) {   // of the pixel at q + dx
  const int d = dx < 0 ? -dx : dx;
  return d >= ex ? 0 : (dx >= 0 ? 1 + d : ex + d);
}

// The staging walks the pixels as the images hold them (a run of pixels is contiguous in x, whatever its place among the staged
// rows), then the rows of zeros: `at` counts them.  Returns the row among the images or the zeros behind a strip; img < 0: zeros.
__host__ __device__ inline int staged_row(const StageShape& s, int at, int& img, int& y, int& x) {
  const int pixels = s.n * s.h * s.w;
  img = -1;
  y = x = 0;
  if (at < pixels) {
    img = at / (s.h * s.w);
    at -= img * (s.h * s.w);
    y = at / s.w;
    x = at - y * s.w;
    return s.lead + y * s.row_len + img * s.wp + x;
  }
  at -= pixels;
  if (at < s.lead) return at;
  at -= s.lead;
  const int line = s.row_len - s.n * s.w, gap = s.wp - s.w;   // zeros of an image row, of them behind each image
  if (at < s.h * line) {
    const int row = at / line, k = at - row * line;
    return s.lead + row * s.row_len + (k < s.n * gap ? k / gap * s.wp + s.w + k % gap : s.n * s.w + k);
  }
  at -= s.h * line;
  const int below = s.main_len - s.h * s.row_len;
  if (at < below) return s.lead + s.h * s.row_len + at;
  at -= below;
  const int behind = s.col_len - s.n * s.h, strips = 2 * s.ex * (s.ey + 1);
  if (at < strips * behind) return s.cols0 + at / behind * s.col_len + s.n * s.h + at % behind;
  at -= strips * behind;
  const int rest = s.pix_len - s.n;
  return s.pix0 + at / rest * s.pix_len + s.n + at % rest;
}
// How many there are
__host__ __device__ inline int staged_rows(const StageShape& s) {
  return s.lead + s.main_len + 2 * s.ex * (s.ey + 1) * (s.col_len - s.n * s.h) + 4 * s.ex * s.ey * (s.pix_len - s.n);
}
// All rows that hold what staged_row found: put(row, true), or put(row, false) where a copy does not keep the pixel.
template <typename F>
__host__ __device__ __forceinline__ void staged_places(const StageShape& s, int row, int img, int y, int x, F&& put) {
  put(row, true);
  if (row < s.lead || row >= s.lead + s.main_len) return;
  for (int v = 1; v < s.copies; ++v) {
    int lo, hi;
    copy_columns(v, s.ex, s.w, lo, hi);
    put(row + v * s.main_len, x >= lo && x < hi);
  }
  if (img < 0 || (x >= s.ex && x < s.w - s.ex)) return;
  const int e = edge_of(x, s.ex, s.w);
  for (int v = 0; v <= s.ey; ++v)
    put(s.cols0 + (v * 2 * s.ex + e) * s.col_len + y * s.n + img, v == 0 || (y >= s.ey && y < s.h - s.ey + v - 1));
  if (y < s.ey || y >= s.h - s.ey) put(s.pix0 + (edge_of(y, s.ey, s.h) * 2 * s.ex + e) * s.pix_len + img, true);
}

template <typename T>
__device__ __forceinline__ float cg_f32(T v) { return static_cast<float>(v); }
template <>
__device__ __forceinline__ float cg_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float cg_f32<at::Half>(at::Half v) { return static_cast<float>(v); }

// 64 staged rows x 64 channels of a block: read along pixels or along channels, whichever is contiguous, and written as rows of
// 16-byte pieces, to every place that holds them.
template <typename T, bool LO>
__global__ void __launch_bounds__(256)
cg_stage_kernel(const T* __restrict__ x, const __grid_constant__ StageShape s, __nv_bfloat16* __restrict__ hi,
                __nv_bfloat16* __restrict__ lo, int ld) {
  __shared__ float tile[64][65];   // [channel][row]
  __shared__ long long base[64];
  __shared__ int4 place[64];   // row, image, y, x
  chain_next();
  const int r0 = blockIdx.x * 64, c0 = blockIdx.y * 64;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 64) {
    int img = -1, y = 0, xx = 0, row = -1;
    if (r0 + threadIdx.x < staged_rows(s)) row = staged_row(s, r0 + threadIdx.x, img, y, xx);
    base[threadIdx.x] = img >= 0 ? img * s.sn + y * s.sh + xx * s.sw : -1;
    place[threadIdx.x] = make_int4(row, img, y, xx);
  }
  __syncthreads();
  if (s.sc == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = warp * 8 + i;
      const long long b = base[r];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int ch = lane + 32 * h;
        tile[ch][r] = b >= 0 && c0 + ch < s.c ? cg_f32(x[b + c0 + ch]) : 0.f;
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int ch = warp * 8 + i;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const long long b = base[lane + 32 * h];
        tile[ch][lane + 32 * h] = b >= 0 && c0 + ch < s.c ? cg_f32(x[b + (c0 + ch) * s.sc]) : 0.f;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int r = warp * 8 + (lane >> 2), ch = ((lane & 3) + 4 * i) * 8;   // 8 rows x 4 pieces: no bank twice
    const int4 q = place[r];
    if (c0 + ch >= ld || q.x < 0) continue;
    uint32_t wh[4], wl[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float v0 = tile[ch + 2 * k][r], v1 = tile[ch + 2 * k + 1][r];
      const __nv_bfloat162 b = __floats2bfloat162_rn(v0, v1);
      wh[k] = *reinterpret_cast<const uint32_t*>(&b);
      if (LO) {
        const __nv_bfloat162 d = __floats2bfloat162_rn(v0 - __uint_as_float(wh[k] << 16), v1 - __uint_as_float(wh[k] & 0xffff0000u));
        wl[k] = *reinterpret_cast<const uint32_t*>(&d);
      }
    }
    const uint4 none = make_uint4(0, 0, 0, 0);
    staged_places(s, q.x, q.y, q.z, q.w, [&](int row, bool keep) {
      const size_t at = static_cast<size_t>(row) * ld + c0 + ch;
      *reinterpret_cast<uint4*>(hi + at) = keep ? make_uint4(wh[0], wh[1], wh[2], wh[3]) : none;
      if (LO) *reinterpret_cast<uint4*>(lo + at) = keep ? make_uint4(wl[0], wl[1], wl[2], wl[3]) : none;
    });
  }
}

// Products that share a K range and their B operand: A = slots (a first row each) x 64-channel chunks, B = one row offset, and the
// row before it where one chunk would not fill a tile (c <= 64), x chunks.  An item is one K range of one 128 x 128 tile.
struct Grid {
  int first;             // first item
  int rows_b, nkb;       // first row of B, K blocks
  int nsplit, tiles_b;   // K ranges; tiles along B
  int tile0, part0;      // first tile, first partial tile (nsplit > 1)
  int slot0;             // first slot; the next grid's is the end
};
constexpr int GRID_WORDS = sizeof(Grid) / 4;

template <int PARTS>
struct CgCfg {
  static constexpr int STAGES = 3;
  static constexpr int STAGE_BYTES = PARTS * 2 * G2_A_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
  static constexpr int TMEM_COLS = PARTS * 128;   // (lo, hi) and (hi, lo) have an accumulator of their own
};

// Tables: [Grid x n_grids, and one behind the last][rows of the slots][tables of the assembly].  Those of up to CG_SMALL words are
// kernel parameters; larger ones are written to memory first (cg_table_kernel).
constexpr int CG_SMALL = 896;
struct CgTables {
  const int* memory;   // null: `words`
  int n_grids, cc;     // cc: 64-channel chunks
  int assembly;        // first word of the assembly's tables
  int words[CG_SMALL];
};
__device__ __forceinline__ const int* table_words(const CgTables& t) { return t.memory != nullptr ? t.memory : t.words; }

// Last grid whose word `key` is not above `at`.
__device__ __forceinline__ const Grid* find_grid(const int* words, int n_grids, int Grid::*key, int at) {
  const Grid* grids = reinterpret_cast<const Grid*>(words);
  int lo = 0, hi = n_grids;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (grids[mid].*key <= at)
      lo = mid;
    else
      hi = mid;
  }
  return grids + lo;
}

// One K range of one tile per CTA.  Tiles are stored as 128 rows of 512 bytes whose 16-byte pieces p are at p ^ (row & 7).
template <int PARTS>
__global__ void __launch_bounds__(192, PARTS == 1 ? 2 : 1)
cg_product_kernel(const __grid_constant__ CUtensorMap tm_hi, const __grid_constant__ CUtensorMap tm_lo,
                  const __grid_constant__ CgTables tab, float* __restrict__ partials, float* __restrict__ tiles, int* status) {
  using Cfg = CgCfg<PARTS>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty_bar = full_bar + Cfg::STAGES;
  uint64_t* acc_bar = empty_bar + Cfg::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (tab.memory != nullptr) chain_wait();   // the tables were written by a kernel before
  const int* words = table_words(tab);
  const Grid* grid = find_grid(words, tab.n_grids, &Grid::first, blockIdx.x);
  const int* slot_rows = words + (tab.n_grids + 1) * GRID_WORDS + grid->slot0;
  const int slots = grid[1].slot0 - grid->slot0, cc = tab.cc, nb = cc == 1 ? 2 : 1;
  const int item = blockIdx.x - grid->first, nsplit = grid->nsplit, tile = item / nsplit, split = item - tile * nsplit;
  const int ia = tile / grid->tiles_b, ib = tile - ia * grid->tiles_b;
  // operand chunks: first row and channel.  Chunks past the last one read channels past the tensor: zeros.
  int row_a[2], row_b[2], ch_a[2], ch_b[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int a = 2 * ia + u, b = 2 * ib + u, sa = a / cc, sb = b / cc;
    row_a[u] = sa < slots ? slot_rows[sa] : grid->rows_b;
    ch_a[u] = (sa < slots ? a - sa * cc : cc) * 64;
    row_b[u] = grid->rows_b - (sb < nb ? sb : 0);
    ch_b[u] = (sb < nb ? b - sb * cc : cc) * 64;
  }
  const int kb0 = static_cast<int>(static_cast<long long>(split) * grid->nkb / nsplit);
  const int nkb = static_cast<int>(static_cast<long long>(split + 1) * grid->nkb / nsplit) - kb0, k0 = kb0 * G2_BK;
  float* const dst = (nsplit > 1 ? partials + static_cast<size_t>(grid->part0 + item) * CG_TILE
                                 : tiles + static_cast<size_t>(grid->tile0 + tile) * CG_TILE);

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_bar, 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  chain_next();
  chain_wait();   // for the staged rows, and for tables in memory

  if (warp == 0) {
    const bool lead = elect_one();
    bool ok = true;
    int kb = 0;
    for (; kb < nkb; ++kb) {
      const int s = kb % Cfg::STAGES;
      if (!mbar_wait(&empty_bar[s], ((kb / Cfg::STAGES) & 1) ^ 1)) {
        set_error(status, ERR_WAIT_EMPTY);
        ok = false;
        break;
      }
      if (lead) {
        uint8_t* stage = smem + s * Cfg::STAGE_BYTES;
        const int k = k0 + kb * G2_BK;
        mbar_expect_tx(&full_bar[s], Cfg::STAGE_BYTES);
#pragma unroll
        for (int part = 0; part < PARTS; ++part) {
          const CUtensorMap* tm = part == 0 ? &tm_hi : &tm_lo;
          uint8_t* a = stage + part * G2_A_BYTES;
          uint8_t* b = stage + (PARTS + part) * G2_A_BYTES;
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            tma_load_2d(a + u * (G2_A_BYTES / 2), tm, &full_bar[s], ch_a[u], row_a[u] + k);
            tma_load_2d(b + u * (G2_A_BYTES / 2), tm, &full_bar[s], ch_b[u], row_b[u] + k);
          }
        }
      }
      __syncwarp();
    }
    if (!ok)   // copies in flight get a bounded chance to land before teardown
      for (int j = kb < Cfg::STAGES ? 0 : kb - Cfg::STAGES; j < kb; ++j) mbar_wait(&full_bar[j % Cfg::STAGES], (j / Cfg::STAGES) & 1);
  } else if (warp == 1) {
    // the whole warp runs the loop and one lane issues: descriptors stay in uniform registers
    const bool lead = elect_one();
    const uint32_t idesc = make_idesc_bf16(128, 128, true, true);
    const uint64_t desc_a = make_smem_desc_sw128(smem_u32(smem), G2_BK * 128, 1024);
    const uint64_t desc_b = make_smem_desc_sw128(smem_u32(smem) + PARTS * G2_A_BYTES, G2_BK * 128, 1024);
    bool ok = true;
    for (int kb = 0; kb < nkb; ++kb) {
      const int s = kb % Cfg::STAGES;
      if (!mbar_wait(&full_bar[s], (kb / Cfg::STAGES) & 1)) {
        set_error(status, ERR_WAIT_FULL);
        ok = false;
        break;
      }
      tc_fence_after_sync();
      constexpr int NPROD = PARTS == 1 ? 1 : 3;
      constexpr int PART_A[3] = {PARTS - 1, 0, 0};   // (lo, hi) (hi, lo) (hi, hi)
      constexpr int PART_B[3] = {0, PARTS - 1, 0};
#pragma unroll
      for (int pr = 0; pr < NPROD; ++pr) {
        const uint64_t da = desc_a + ((s * Cfg::STAGE_BYTES + PART_A[pr] * G2_A_BYTES) >> 4);
        const uint64_t db = desc_b + ((s * Cfg::STAGE_BYTES + PART_B[pr] * G2_A_BYTES) >> 4);
#pragma unroll
        for (int k = 0; k < G2_BK / 16; ++k)
          if (lead) umma_bf16(tmem_base + (pr < NPROD - 1 ? 128 : 0), da + k * 128, db + k * 128, idesc, (kb | k) || pr == 1 ? 1u : 0u);
      }
      if (lead) umma_commit(&empty_bar[s]);
      __syncwarp();
    }
    if (ok && lead) umma_commit(acc_bar);
    __syncwarp();
  } else {
    const int q = warp & 3, row = q * 32 + lane;
    if (!mbar_wait(acc_bar, 0)) set_error(status, ERR_WAIT_ACC);
    __syncwarp();
    tc_fence_after_sync();
    // every product is done: the ring takes the tile, which leaves as one copy
#pragma unroll 1
    for (int h = 0; h < 4; ++h) {
      uint32_t v[32];
      tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + 32 * h, v);
      tmem_ld_wait();
      if constexpr (PARTS > 1) {
        uint32_t small[32];
        tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + 128 + 32 * h, small);
        tmem_ld_wait();
#pragma unroll
        for (int c = 0; c < 32; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) + __uint_as_float(small[c]));
      }
#pragma unroll
      for (int p = 0; p < 8; ++p)
        *reinterpret_cast<uint4*>(smem + row * 512 + (((8 * h + p) ^ (row & 7)) << 4)) = make_uint4(v[4 * p], v[4 * p + 1], v[4 * p + 2], v[4 * p + 3]);
    }
    asm volatile("fence.proxy.async;" ::: "memory");
    named_bar_sync(1, 128);
    if (threadIdx.x == 64) {
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(smem)), "r"(CG_TILE * 4)
                   : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// Sums the K ranges of a tile, in order.  grid: (16, tiles in ranges, which are the first), a thread has four values and eight
// ranges in flight.
__global__ void __launch_bounds__(256)
cg_reduce_kernel(const float4* partials, float4* tiles, const __grid_constant__ CgTables tab) {
  chain_next();
  chain_wait();
  const Grid* grid = find_grid(table_words(tab), tab.n_grids, &Grid::tile0, blockIdx.y);
  const int at = blockIdx.x * 256 + threadIdx.x, nsplit = grid->nsplit;
  const float4* from = partials + (grid->part0 + static_cast<size_t>(blockIdx.y - grid->tile0) * nsplit) * (CG_TILE / 4) + at;
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s = 0; s < nsplit; s += 8) {
    float4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      v[u] = s + u < nsplit ? from[static_cast<size_t>(s + u) * (CG_TILE / 4)] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      sum.x += v[u].x;
      sum.y += v[u].y;
      sum.z += v[u].z;
      sum.w += v[u].w;
    }
  }
  tiles[static_cast<size_t>(blockIdx.y) * (CG_TILE / 4) + at] = sum;
}

// Where a product is among the tiles, and which terms make up the block of two taps
struct ProductAt {
  int tile0;                    // first tile of the grid that it is in
  short tiles_b, a0, b0, pad;   // tiles along B of that grid; the product's first chunks there
};
struct AssembleShape {
  int n, c, taps, khwc;   // rows of the result, channels, filter taps, column order (kh, kw, c)
  int n_products, n_terms;
  float scale, beta;
};

// 32 x 32 patches on or below the diagonal; tables: [ProductAt x products][first term of tap pair t (t + 1) / 2 + t', and one
// past the last][terms: products].
__global__ void __launch_bounds__(256)
cg_assemble_kernel(const float* tiles, const __grid_constant__ AssembleShape a, const __grid_constant__ CgTables tables,
                   float* out, long long ldc) {
  extern __shared__ int tab[];
  __shared__ float patch[32][33];
  chain_wait();
  const int pairs = a.taps * (a.taps + 1) / 2, words = 3 * a.n_products + pairs + 1 + (a.n_terms + 1) / 2;
  const int* from = table_words(tables) + tables.assembly;
  for (int i = threadIdx.x; i < words; i += 256) tab[i] = from[i];
  const ProductAt* products = reinterpret_cast<const ProductAt*>(tab);
  const int* first = tab + 3 * a.n_products;
  const unsigned short* terms = reinterpret_cast<const unsigned short*>(first + pairs + 1);
  // patch of the lower triangle: blockIdx.x = by (by + 1) / 2 + bx
  int by = static_cast<int>((sqrtf(8.f * blockIdx.x + 1.f) - 1.f) * 0.5f);
  while ((by + 1) * (by + 2) / 2 <= static_cast<int>(blockIdx.x)) ++by;
  while (by * (by + 1) / 2 > static_cast<int>(blockIdx.x)) --by;
  const int bx = blockIdx.x - by * (by + 1) / 2;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int j = bx * 32 + tx;
  const int cj = a.khwc ? j % a.c : j / a.taps, tj = a.khwc ? j / a.c : j % a.taps;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int i = by * 32 + ty + 8 * k;
    float v = 0.f;
    if (i < a.n && j <= i) {
      const float before = a.beta != 0.f ? out[i * ldc + j] : 0.f;
      const int ci = a.khwc ? i % a.c : i / a.taps, ti = a.khwc ? i / a.c : i % a.taps;
      // a product's rows are the channels of the later tap
      const bool swap = ti < tj;
      const int t = swap ? tj : ti, u = swap ? ti : tj, row = swap ? cj : ci, col = swap ? ci : cj;
      const int pair = t * (t + 1) / 2 + u;
      float sum = 0.f;
      for (int e = first[pair]; e < first[pair + 1]; ++e) {
        const ProductAt p = products[terms[e]];
        const int ca = p.a0 + (row >> 6), cb = p.b0 + (col >> 6);
        const int r = (ca & 1) * 64 + (row & 63), c = (cb & 1) * 64 + (col & 63);
        const float* tile = tiles + static_cast<size_t>(p.tile0 + (ca >> 1) * p.tiles_b + (cb >> 1)) * CG_TILE;
        sum += tile[r * 128 + ((((c >> 2) ^ (r & 7)) << 2) | (c & 3))];
      }
      v = a.scale * sum;
      if (a.beta != 0.f) v += a.beta * before;
      out[i * ldc + j] = v;
    }
    patch[ty + 8 * k][tx] = v;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = bx * 32 + ty + 8 * k, c = by * 32 + tx;   // mirror image
    if (r < c && c < a.n) out[r * ldc + c] = patch[tx][ty + 8 * k];
  }
}

// The same where a 64 x 64 block of the result is one block of channels of two taps: order (kh, kw, c) and whole 64-channel
// chunks.  The terms belong to the whole block, and all accesses have 16 bytes: 32 x 256 x 14 x 14, 2304 x 2304 result:
// 26 us with a look-up per entry, 8.7 so.
__global__ void __launch_bounds__(256)
cg_assemble_blocks_kernel(const float* tiles, const __grid_constant__ AssembleShape a, const __grid_constant__ CgTables tables,
                          float* out, long long ldc, bool vec) {
  __shared__ float patch[64][65];
  chain_wait();
  const int* tab = table_words(tables) + tables.assembly;
  const ProductAt* products = reinterpret_cast<const ProductAt*>(tab);
  const int pairs = a.taps * (a.taps + 1) / 2;
  const int* first = tab + 3 * a.n_products;
  const unsigned short* terms = reinterpret_cast<const unsigned short*>(first + pairs + 1);
  int by = static_cast<int>((sqrtf(8.f * blockIdx.x + 1.f) - 1.f) * 0.5f);
  while ((by + 1) * (by + 2) / 2 <= static_cast<int>(blockIdx.x)) ++by;
  while (by * (by + 1) / 2 > static_cast<int>(blockIdx.x)) --by;
  const int bx = blockIdx.x - by * (by + 1) / 2, cc = a.c / 64;
  const int t = by / cc, u = bx / cc, chunk_i = by - t * cc, chunk_j = bx - u * cc;   // t >= u
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // columns 4 tx .. 4 tx + 3 of rows ty + 16 k
  float4 before[4];
  if (a.beta != 0.f) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float* at = out + (by * 64ll + ty + 16 * k) * ldc + bx * 64 + 4 * tx;
      before[k] = vec ? *reinterpret_cast<const float4*>(at) : make_float4(at[0], at[1], at[2], at[3]);
    }
  }
  float sum[4][4] = {};
  const int pair = t * (t + 1) / 2 + u, end = first[pair + 1];
  for (int e = first[pair]; e < end; ++e) {
    const ProductAt p = products[terms[e]];
    const int ca = p.a0 + chunk_i, cb = p.b0 + chunk_j;
    const float* tile = tiles + static_cast<size_t>(p.tile0 + (ca >> 1) * p.tiles_b + (cb >> 1)) * CG_TILE + (ca & 1) * (64 * 128);
    float4 w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int r = ty + 16 * k;
      w[k] = *reinterpret_cast<const float4*>(tile + r * 128 + ((((cb & 1) * 16 + tx) ^ (r & 7)) << 2));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      sum[k][0] += w[k].x;
      sum[k][1] += w[k].y;
      sum[k][2] += w[k].z;
      sum[k][3] += w[k].w;
    }
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = ty + 16 * k;
    float v[4];
    const float b[4] = {before[k].x, before[k].y, before[k].z, before[k].w};
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      v[h] = a.scale * sum[k][h];
      if (a.beta != 0.f) v[h] += a.beta * b[h];
      patch[r][4 * tx + h] = v[h];
    }
    if (by != bx) {
      float* at = out + (by * 64ll + r) * ldc + bx * 64 + 4 * tx;
      if (vec)
        *reinterpret_cast<float4*>(at) = make_float4(v[0], v[1], v[2], v[3]);
      else
        for (int h = 0; h < 4; ++h) at[h] = v[h];
    }
  }
  __syncthreads();
  // mirror image; of a block on the diagonal, which is symmetric up to its last bits, the lower triangle goes to both sides
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int r = ty + 16 * k;
    float v[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const int c = 4 * tx + h;
      v[h] = by == bx && c < r ? patch[r][c] : patch[c][r];
    }
    float* at = out + (bx * 64ll + r) * ldc + by * 64 + 4 * tx;
    if (vec)
      *reinterpret_cast<float4*>(at) = make_float4(v[0], v[1], v[2], v[3]);
    else
      for (int h = 0; h < 4; ++h) at[h] = v[h];
  }
}

// Tables reach the device as kernel parameters, by value, so a captured launch does not refer to host memory.
constexpr int CG_CHUNK = 28 * 1024;
struct CgChunk {
  int words[CG_CHUNK / 4];
};
__global__ void cg_table_kernel(const __grid_constant__ CgChunk chunk, int* dst, int words) {
  for (int i = threadIdx.x; i < words; i += blockDim.x) dst[i] = chunk.words[i];
}

int ceil_to(long long v, int m) { return static_cast<int>((v + m - 1) / m * m); }

// What a call stages, multiplies and adds, which depends on the shapes alone.
struct Plan {
  StageShape s;
  int cc, n_grids, assembly, n_products, n_terms;
  int tiles, split_tiles, partial_tiles, items;
  std::vector<int> words;   // tables, see CgTables
};

// False: the shape is outside of what the tables hold.
bool make_plan(Plan& P, int64_t n, int64_t c, int64_t h, int64_t w, int kh, int kw, int ph, int pw, int resident, int longest_sum) {
  const int64_t ho = h + 2 * ph - kh + 1, wo = w + 2 * pw - kw + 1;
  const int taps = kh * kw;
  if (kh < 1 || kw < 1 || kh > CG_MAX_K || kw > CG_MAX_K || taps < 2 || ph < 0 || pw < 0 || ph >= kh || pw >= kw || ho < 1 || wo < 1 ||
      n < 1 || c < 1 || c > 4096 || n > (1 << 24) || h > (1 << 24) || w > (1 << 24))
    return false;
  // ---- staged rows
  StageShape& s = P.s;
  std::memset(&s, 0, sizeof(s));
  const int ey = kh - 1 - ph, ex = kw - 1 - pw;
  if (2 * ey > h || 2 * ex > w) return false;   // a row or column would be among the first and among the last
  const int64_t row_len = (n * (w + kw - 1) + 63) / 64 * 64, col_len = (n * (h + kh - 1) + 63) / 64 * 64, pix_len = (n + 63) / 64 * 64;
  const int64_t copies = ex > 0 ? 2 * ex : 1, col_strips = ex > 0 ? (ey + 1) * 2 * ex : 0;
  if ((h + ph) > (1ll << 30) / (row_len * copies) || col_strips * col_len > (1ll << 28) || 4 * ey * ex * pix_len > (1ll << 28)) return false;
  s.n = static_cast<int>(n);
  s.c = static_cast<int>(c);
  s.h = static_cast<int>(h);
  s.w = static_cast<int>(w);
  s.wp = static_cast<int>(w + kw - 1);
  s.ey = ey;
  s.ex = ex;
  s.lead = 64;
  s.row_len = static_cast<int>(row_len);
  s.main_len = static_cast<int>(row_len * (h + ph));
  s.copies = static_cast<int>(copies);
  s.cols0 = s.lead + s.main_len * s.copies;
  s.col_len = static_cast<int>(col_len);
  s.pix0 = s.cols0 + static_cast<int>(col_strips * col_len);
  s.pix_len = static_cast<int>(pix_len);
  s.total = s.pix0 + 4 * ey * ex * s.pix_len;

  // ---- products.  A pair of pixels at distance (dy, dx) is named by the row of the upper one and the column of the left one.
  const int cc = P.cc = static_cast<int>((c + 63) / 64);
  struct HostGrid {
    int rows_b, nkb;
    std::vector<int> slots;
  };
  struct Product {
    int grid, slot, e;
  };
  std::vector<HostGrid> grids;
  std::vector<Product> products;
  auto add_grid = [&](int rows_b, int nkb) {
    grids.push_back({rows_b, nkb, {}});
    return static_cast<int>(grids.size()) - 1;
  };
  auto add_product = [&](int grid, int e) {
    products.push_back({grid, static_cast<int>(grids[grid].slots.size()) - 1, e});
    return static_cast<int>(products.size()) - 1;
  };
  const int nr = 2 * ey, nc = 2 * ex, nx = 2 * kw - 1;   // edge rows and columns; values of dx
  auto edge_row = [&](int dy, int y) { return y >= 0 && y + dy < h && dy < ey && (y < ey - dy || y >= h - ey); };
  auto edge_col = [&](int dx, int l) { return l >= 0 && l + std::abs(dx) < w && std::abs(dx) < ex && (l < ex - std::abs(dx) || l >= w - ex); };
  auto inner_rows = [&](int dy) { return dy < ey ? h > nr - dy : h > dy; };   // pairs that are in every window
  auto inner_cols = [&](int dx) { const int d = std::abs(dx); return d < ex ? w > nc - d : w > d; };
  // core[dy, dx]: rows and columns in every window; rows[dy, dx, y]: one edge row; cols[dy, dx, l]: one edge column; pixels: both
  std::vector<int> core(kh * nx, -1), rows(kh * nx * nr, -1), cols(kh * nx * nc, -1), pixels(kh * nx * nr * nc, -1);
  auto at = [&](int dy, int dx) { return dy * nx + dx + kw - 1; };
  // the pairs of rows (y0 + k, y0 + dy + k) of every dx
  auto add_rows = [&](int grid, int dy, int y0, auto&& product) {
    for (int dx = dy == 0 ? 0 : 1 - kw; dx < kw; ++dx) {
      if (!inner_cols(dx)) continue;
      const int copy = copy_of(dx, ex);
      grids[grid].slots.push_back(s.lead + copy * s.main_len + (y0 + dy) * s.row_len + dx);
      product(dx) = add_product(grid, 0);
      // B's row before belongs to the next dx, where that one takes the images without a mask too
      if (cc == 1 && copy == 0 && dx + 1 < kw && inner_cols(dx + 1) && copy_of(dx + 1, ex) == 0) {
        ++dx;
        product(dx) = add_product(grid, 1);
      }
    }
  };
  for (int g = 0; g <= ey; ++g) {   // dy < ey have rows of their own; all others share theirs
    const int y0 = ey - g, y1 = static_cast<int>(h) - ey;
    if (y1 <= y0) continue;
    const int grid = add_grid(s.lead + y0 * s.row_len, (y1 - y0) * (s.row_len / 64));
    for (int dy = g; dy < (g < ey ? g + 1 : kh); ++dy)
      if (inner_rows(dy)) add_rows(grid, dy, y0, [&](int dx) -> int& { return core[at(dy, dx)]; });
  }
  for (int e = 0; e < nr; ++e) {
    const int y = edge_at(e, ey, s.h);
    for (int dy = 0; dy < ey; ++dy)
      if (edge_row(dy, y)) {
        const int grid = add_grid(s.lead + y * s.row_len, s.row_len / 64);
        add_rows(grid, dy, y, [&](int dx) -> int& { return rows[at(dy, dx) * nr + e]; });
      }
  }
  for (int e = 0; e < nc; ++e) {   // column under the earlier tap
    const int q = edge_at(e, ex, s.w);
    const int grid = add_grid(s.cols0 + e * s.col_len, s.col_len / 64);
    for (int dy = 0; dy < kh; ++dy)
      for (int dx = dy == 0 ? 0 : 1 - kw; dx < kw; ++dx) {
        const int l = std::min(q, q + dx);
        if (!inner_rows(dy) || !edge_col(dx, l)) continue;
        const int copy = dy < ey ? 1 + dy : 0;
        grids[grid].slots.push_back(s.cols0 + (copy * nc + edge_of(q + dx, ex, s.w)) * s.col_len + dy * s.n);
        cols[at(dy, dx) * nc + edge_of(l, ex, s.w)] = add_product(grid, 0);
      }
  }
  for (int e = 0; e < nr * nc; ++e) {
    const int y = edge_at(e / nc, ey, s.h), q = edge_at(e % nc, ex, s.w);
    const int grid = add_grid(s.pix0 + e * s.pix_len, s.pix_len / 64);
    for (int dy = 0; dy < ey; ++dy)
      for (int dx = dy == 0 ? 0 : 1 - kw; dx < kw; ++dx) {
        const int l = std::min(q, q + dx);
        if (!edge_row(dy, y) || !edge_col(dx, l)) continue;
        grids[grid].slots.push_back(s.pix0 + (edge_of(y + dy, ey, s.h) * nc + edge_of(q + dx, ex, s.w)) * s.pix_len);
        pixels[(at(dy, dx) * nr + e / nc) * nc + edge_of(l, ex, s.w)] = add_product(grid, 0);
      }
  }

  // ---- which products make up the block of taps t >= u
  std::vector<int> terms, first(1, 0);
  for (int t = 0; t < taps; ++t)
    for (int u = 0; u <= t; ++u) {
      const int dy = t / kw - u / kw, dx = t % kw - u % kw, d = at(dy, dx);
      const int64_t top = u / kw - ph, left = std::min(t % kw, u % kw) - pw;   // of the window
      auto add = [&](int product) {
        if (product >= 0) terms.push_back(product);
      };
      auto row_counts = [&](int e) { const int64_t y = edge_at(e, ey, s.h); return y >= top && y < top + ho; };
      auto col_counts = [&](int e) { const int64_t l = edge_at(e, ex, s.w); return l >= left && l < left + wo; };
      add(core[d]);
      for (int e = 0; e < nr; ++e)
        if (row_counts(e)) add(rows[d * nr + e]);
      for (int f = 0; f < nc; ++f)
        if (col_counts(f)) add(cols[d * nc + f]);
      for (int e = 0; e < nr; ++e)
        for (int f = 0; f < nc; ++f)
          if (row_counts(e) && col_counts(f)) add(pixels[(d * nr + e) * nc + f]);
      first.push_back(static_cast<int>(terms.size()));
    }

  // ---- tiles and items: long grids first, K ranges as short as it takes to give every resident CTA one, or equal parts of them
  const int nb = cc == 1 ? 2 : 1, tiles_b = (nb * cc + 1) / 2;
  std::vector<int> order;
  int64_t tiles = 0, blocks = 0;
  int longest = 0;
  auto grid_tiles = [&](const HostGrid& g) { return static_cast<int64_t>((g.slots.size() * cc + 1) / 2) * tiles_b; };
  for (size_t g = 0; g < grids.size(); ++g) {
    if (grids[g].slots.empty()) continue;
    order.push_back(static_cast<int>(g));
    tiles += grid_tiles(grids[g]);
    blocks += grid_tiles(grids[g]) * grids[g].nkb;
    longest = std::max(longest, grids[g].nkb);
  }
  if (order.empty() || products.size() > CG_MAX_PRODUCTS || terms.size() > CG_MAX_TERMS || tiles > CG_MAX_TILES) return false;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return grids[a].nkb > grids[b].nkb; });
  auto ranges = [&](const HostGrid& g, int64_t len) { return static_cast<int>((g.nkb + len - 1) / len); };
  int64_t len = std::max<int64_t>(4, blocks / resident);
  for (; len < longest; len += 1 + len / 32) {
    int64_t items = 0;
    for (int g : order) items += grid_tiles(grids[g]) * ranges(grids[g], len);
    if (items <= resident) break;
  }
  // a longer sum loses more to the tensor core's truncation than patches did: the same share of every CTA in equal parts
  len = std::min<int64_t>(len, longest);
  len = (len + (len + longest_sum - 1) / longest_sum - 1) / ((len + longest_sum - 1) / longest_sum);
  P.n_grids = static_cast<int>(order.size());
  P.tiles = P.split_tiles = P.partial_tiles = P.items = 0;
  std::vector<Grid> out(P.n_grids + 1);
  std::vector<int> where(grids.size(), -1), slot_rows;
  for (int k = 0; k < P.n_grids; ++k) {
    const HostGrid& g = grids[order[k]];
    const int count = static_cast<int>(grid_tiles(g)), nsplit = ranges(g, len);
    out[k] = {P.items, g.rows_b, g.nkb, nsplit, tiles_b, P.tiles, P.partial_tiles, static_cast<int>(slot_rows.size())};
    where[order[k]] = k;
    P.items += count * nsplit;
    P.tiles += count;
    if (nsplit > 1) {   // a prefix of the grids
      P.split_tiles += count;
      P.partial_tiles += count * nsplit;
    }
    slot_rows.insert(slot_rows.end(), g.slots.begin(), g.slots.end());
  }
  out[P.n_grids] = {P.items, 0, 0, 1, tiles_b, P.tiles, P.partial_tiles, static_cast<int>(slot_rows.size())};

  // ---- tables
  static_assert(sizeof(ProductAt) == 12, "tables hold three words per product");
  std::vector<int>& words = P.words;
  const size_t slots_at = out.size() * GRID_WORDS, assembly = slots_at + slot_rows.size(), first_at = assembly + 3 * products.size();
  words.assign(first_at + first.size() + (terms.size() + 1) / 2, 0);
  std::memcpy(words.data(), out.data(), out.size() * sizeof(Grid));
  std::copy(slot_rows.begin(), slot_rows.end(), words.begin() + slots_at);
  for (size_t p = 0; p < products.size(); ++p) {
    const Grid& g = out[where[products[p].grid]];
    const ProductAt place = {g.tile0, static_cast<short>(tiles_b), static_cast<short>(products[p].slot * cc), static_cast<short>(products[p].e * cc), 0};
    std::memcpy(&words[assembly + 3 * p], &place, sizeof(place));
  }
  std::copy(first.begin(), first.end(), words.begin() + first_at);
  unsigned short* packed = reinterpret_cast<unsigned short*>(words.data() + first_at + first.size());
  for (size_t i = 0; i < terms.size(); ++i) packed[i] = static_cast<unsigned short>(terms[i]);
  P.assembly = static_cast<int>(assembly);
  P.n_products = static_cast<int>(products.size());
  P.n_terms = static_cast<int>(terms.size());
  return true;
}

int resident_ctas(int sms, bool x3) { return sms * (x3 ? 1 : 2); }
// K blocks of a range, for the error of the sums (above); the shorter ranges also fill the last wave of many tiles: 32 x 128 x 32 x 32,
// 5 x 5, 157 tiles, 462 -> 274 us, 32 x 192 x 32 x 32, 3 x 3, 181 -> 147.  bf16 products have a third of the additions; their errors are below
// those of patches with ranges of any length.
int longest_sum_of(bool x3) { return x3 ? 128 : 1 << 30; }

}  // namespace

bool gemm_batch_is_open();

// The plan of a shape, for tests: {row shape, counts, tables}, empty where there is none.
std::vector<std::vector<int64_t>> conv_gram_plan(int64_t n, int64_t c, int64_t h, int64_t w, int64_t kh, int64_t kw, int64_t ph, int64_t pw,
                                                 int64_t sms, bool x3) {
  Plan P;
  if (!make_plan(P, n, c, h, w, static_cast<int>(kh), static_cast<int>(kw), static_cast<int>(ph), static_cast<int>(pw),
                 resident_ctas(static_cast<int>(sms), x3), longest_sum_of(x3)))
    return {};
  const StageShape& s = P.s;
  // every row that is staged, with what it holds: (row, image, y, x), image -1: zeros
  std::vector<int64_t> staged;
  for (int at = 0; at < staged_rows(s); ++at) {
    int img, y, x;
    const int first = staged_row(s, at, img, y, x);
    staged_places(s, first, img, y, x, [&](int row, bool keep) { staged.insert(staged.end(), {row, keep ? img : -1, y, x}); });
  }
  return {{s.total, P.cc, P.n_grids, P.assembly, P.n_products, P.n_terms, P.tiles, P.split_tiles, P.partial_tiles, P.items},
          std::vector<int64_t>(P.words.begin(), P.words.end()), staged};
}

// Returns false, with nothing done, where the general path has to be taken: a batch of products is being recorded (the products
// of the general path run together there), or the shape is outside of what the tables here hold.
bool conv_gram(at::Tensor x, at::Tensor out, int64_t kh, int64_t kw, int64_t ph, int64_t pw, double scale, double beta, bool khwc,
               bool x3) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 4, "x must be a 4-d CUDA tensor");
  TORCH_CHECK(x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16 || x.scalar_type() == at::kHalf, "x must be fp32, bf16 or fp16");
  const int dev = x.get_device();
  const int64_t c = x.size(1), taps = kh * kw, ncol = taps * c;
  Plan P;
  if (gemm_batch_is_open() || kh > CG_MAX_K || kw > CG_MAX_K ||
      !make_plan(P, x.size(0), c, x.size(2), x.size(3), static_cast<int>(kh), static_cast<int>(kw), static_cast<int>(ph), static_cast<int>(pw),
                 resident_ctas(g2_sm_count(dev), x3), longest_sum_of(x3)))
    return false;
  TORCH_CHECK(out.is_cuda() && out.scalar_type() == at::kFloat && out.dim() == 2 && out.size(0) == ncol && out.size(1) == ncol &&
                  out.stride(1) == 1, "out must be a [c kh kw, c kh kw] fp32 CUDA matrix with unit column stride");
  TORCH_CHECK(out.get_device() == dev, "x and out must be on one device");
  StageShape& s = P.s;
  s.sn = x.stride(0);
  s.sc = x.stride(1);
  s.sh = x.stride(2);
  s.sw = x.stride(3);

  c10::cuda::CUDAGuard guard(dev);
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream(dev).stream();
  const int ld = ceil_to(c, 8);
  auto bytes = at::TensorOptions().dtype(at::kByte).device(at::kCUDA, dev);
  auto f32 = at::TensorOptions().dtype(at::kFloat).device(at::kCUDA, dev);
  at::Tensor staged = at::empty({(x3 ? 2 : 1) * static_cast<int64_t>(s.total) * ld * 2}, bytes);
  __nv_bfloat16* hi = reinterpret_cast<__nv_bfloat16*>(staged.data_ptr());
  __nv_bfloat16* lo = x3 ? hi + static_cast<size_t>(s.total) * ld : nullptr;
  at::Tensor partials;
  if (P.partial_tiles > 0) partials = at::empty({static_cast<int64_t>(P.partial_tiles) * CG_TILE}, f32);
  at::Tensor tiles = at::empty({static_cast<int64_t>(P.tiles) * CG_TILE}, f32);

  const std::vector<int>& host = P.words;
  CgTables tables;
  tables.memory = nullptr;
  tables.n_grids = P.n_grids;
  tables.cc = P.cc;
  tables.assembly = P.assembly;
  at::Tensor table;
  if (host.size() <= CG_SMALL) {
    std::memcpy(tables.words, host.data(), host.size() * 4);
  } else {
    table = at::empty({static_cast<int64_t>(host.size()) * 4}, bytes);
    int* d_table = reinterpret_cast<int*>(table.data_ptr());
    tables.memory = d_table;
    for (size_t at = 0; at < host.size(); at += CG_CHUNK / 4) {
      CgChunk chunk;
      const int words = static_cast<int>(std::min<size_t>(CG_CHUNK / 4, host.size() - at));
      std::memcpy(chunk.words, host.data() + at, words * 4);
      cg_table_kernel<<<1, 256, 0, stream>>>(chunk, d_table + at, words);
      B200_CUDA_CHECK(cudaGetLastError());
      count_launch();
    }
  }

  const dim3 sgrid((staged_rows(s) + 63) / 64, (ld + 63) / 64);
  auto stage = [&](auto* p) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(p)>>;
    if (x3)
      cg_stage_kernel<T, true><<<sgrid, 256, 0, stream>>>(p, s, hi, lo, ld);
    else
      cg_stage_kernel<T, false><<<sgrid, 256, 0, stream>>>(p, s, hi, nullptr, ld);
  };
  if (x.scalar_type() == at::kFloat)
    stage(x.data_ptr<float>());
  else if (x.scalar_type() == at::kBFloat16)
    stage(reinterpret_cast<const __nv_bfloat16*>(x.data_ptr()));
  else
    stage(x.data_ptr<at::Half>());
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();

  CUtensorMap tm_hi, tm_lo;
  g2_encode_operand(&tm_hi, hi, c, s.total, ld, false, 0);
  g2_encode_operand(&tm_lo, x3 ? lo : hi, c, s.total, ld, false, 0);
  int* status = device_state(dev).status.data_ptr<int>();
  float* dp = P.partial_tiles > 0 ? partials.data_ptr<float>() : nullptr;
  auto run = [&](auto kernel, int smem) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    launch_chained(kernel, dim3(P.items), dim3(192), smem, stream, tm_hi, tm_lo, tables, dp, tiles.data_ptr<float>(), status);
  };
  if (x3)
    run(cg_product_kernel<2>, CgCfg<2>::SMEM_BYTES);
  else
    run(cg_product_kernel<1>, CgCfg<1>::SMEM_BYTES);
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
  if (P.split_tiles > 0) {
    launch_chained(cg_reduce_kernel, dim3(CG_TILE / 4 / 256, P.split_tiles), dim3(256), 0, stream, reinterpret_cast<const float4*>(dp),
                   reinterpret_cast<float4*>(tiles.data_ptr<float>()), tables);
    B200_CUDA_CHECK(cudaGetLastError());
    count_launch();
  }
  AssembleShape a;
  a.n = static_cast<int>(ncol);
  a.c = static_cast<int>(c);
  a.taps = static_cast<int>(taps);
  a.khwc = khwc;
  a.n_products = P.n_products;
  a.n_terms = P.n_terms;
  a.scale = static_cast<float>(scale);
  a.beta = static_cast<float>(beta);
  float* result = out.data_ptr<float>();
  if (khwc && c % 64 == 0) {
    const int nb = a.n / 64;
    const bool vec = out.stride(0) % 4 == 0 && (reinterpret_cast<uintptr_t>(result) & 15) == 0;
    launch_chained(cg_assemble_blocks_kernel, dim3(nb * (nb + 1) / 2), dim3(256), 0, stream, tiles.data_ptr<float>(), a, tables, result, out.stride(0), vec);
  } else {
    const int nb = (a.n + 31) / 32, tab_bytes = static_cast<int>(host.size() - P.assembly) * 4;
    // launched plainly: resident beside the products, whose shared memory leaves little of an SM's memory to the L1 cache, its look-ups take
    // longer than the launch (128 x 64 x 32 x 32 fp32: 85.3 us chained, 78.6 so; 8 x 64 x 16 x 16: 31.5 and 25.4)
    launch_behind(false, cg_assemble_kernel, dim3(nb * (nb + 1) / 2), dim3(256), tab_bytes, stream, tiles.data_ptr<float>(), a, tables, result, out.stride(0));
  }
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
  return true;
}

}  // namespace b200
