// Input-side Kronecker factor of a stride-1 convolution without its patch matrix.
//
//     out = scale * M^T M (+ beta * out),   M [n * ho * wo, c * kh * kw] the patches of x
//
// (asdl/utils.py:51-88 and asdl/operations/conv.py:80-88 build M with unfold.)  The block of M^T M of two taps t >= t' is a sum
// of x[q + d] x[q]^T over the input pixels q with d = t - t', and depends on the taps themselves only through which q count: the
// output pixels o with o + t' - p = q.  So
//
//     block(t, t') = R_d - (rows of q outside of the window) - (columns outside) + (pixels in both),
//     R_d = sum of x[q + d] x[q]^T over all q with both pixels in the image
//
// A k x k filter has ((2k - 1)^2 + 1) / 2 differences d (13 for 3 x 3, 41 for 5 x 5) instead of kk (kk + 1) / 2 blocks (45, 325),
// and the rows, columns and pixels to take off are few and short (3 x 3, padding 1: the first and last row for d = (0, dx), the
// first and last column for d = (dy, 0), the corners for d = 0).
//
//   stage     x -> bf16 (hi, or hi and lo) rows [pixel, channel]: every image with kw - 1 zeros behind each row and kh - 1 zero
//             rows behind the last, so that a difference d is a constant offset of rows; then the same for each edge row, edge
//             column and corner alone ("strips": the K ranges of what is taken off);
//   products  128 x 128 tiles of 64-channel chunks.  Each chunk is a TMA box with a row offset of its own, so a tile holds the
//             chunks of two shifts where 64 channels would not fill it (c <= 64: A = pairs of shifts f - 1, B = {-1, 0}: differences
//             f and f - 1).  A CTA takes one K range of a tile; hi and lo parts are loaded once for the three part products;
//   reduce    sums the K ranges in order;
//   assemble  looks up the terms of each entry, adds the moving average, writes entry and mirror image.
//
// The patch matrix was written and read before: 128 x 64 x 32 x 32 fp32, 3 x 3: 302 MB, 15 tiles of K = 131072 with three part
// products, each loading both operands, 337 -> 85 us (staging 20, products 47, reduction 4, assembly 8); 32 x 256 x 14 x 14
// bf16: 63 -> 45 us (5, 19, 3, 9, and the host's 28).  The fp32 products are bound by what L2 delivers (64 KiB per K block of 768
// tensor clocks).  A non-finite input gives a non-finite factor as with patches, but where a window leaves such a pixel out,
// what is taken off is not finite either: more entries are affected.
#include <cstring>

#include "chained_launch.h"
#include "gemm2_host.h"

namespace b200 {

namespace {

constexpr int CG_MAX_K = 5;
constexpr int CG_MAX_SHIFTS = 48;
constexpr int CG_MAX_PRODUCTS = 1024;
constexpr int CG_TILE = 128 * 128;          // floats of a tile

// Staged rows: lead, images, row strips, column strips, pixel strips.  Every part is a multiple of 64 rows.
struct StageShape {
  int n, c, h, w, hp, wp;                   // hp, wp: with the zeros behind
  int ey, ex;                               // edge rows / columns on each side that strips exist of
  int lead, rows0, cols0, pix0, total;      // first row of the parts
  int row_len, col_len, pix_len;            // rows of a strip
  long long sn, sc, sh, sw;                 // element strides of x
};

// Image row or column of edge strip e of 2 * edges: the first `edges` ones, then the last.
__host__ __device__ inline int edge_at(int e, int edges, int extent) { return e < edges ? e : extent - 2 * edges + e; }

// Input pixel of a staged row; false: a row of zeros
__device__ __forceinline__ bool staged_pixel(const StageShape& s, int r, int& img, int& y, int& x) {
  if (r < s.lead) return false;
  if (r < s.rows0) {
    r -= s.lead;
    x = r % s.wp;
    r /= s.wp;
    y = r % s.hp;
    img = r / s.hp;
    return img < s.n && y < s.h && x < s.w;
  }
  if (r < s.cols0) {
    r -= s.rows0;
    y = edge_at(r / s.row_len, s.ey, s.h);
    r %= s.row_len;
    x = r % s.wp;
    img = r / s.wp;
    return img < s.n && x < s.w;
  }
  if (r < s.pix0) {
    r -= s.cols0;
    x = edge_at(r / s.col_len, s.ex, s.w);
    r %= s.col_len;
    y = r % s.hp;
    img = r / s.hp;
    return img < s.n && y < s.h;
  }
  r -= s.pix0;
  const int e = r / s.pix_len;
  img = r % s.pix_len;
  if (img >= s.n) return false;
  y = edge_at(e / (2 * s.ex), s.ey, s.h);
  x = edge_at(e % (2 * s.ex), s.ex, s.w);
  return true;
}

template <typename T>
__device__ __forceinline__ float cg_f32(T v) { return static_cast<float>(v); }
template <>
__device__ __forceinline__ float cg_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float cg_f32<at::Half>(at::Half v) { return static_cast<float>(v); }

// 64 staged rows x 64 channels of a block: read along pixels or along channels, whichever is contiguous, and written as rows of
// 16-byte pieces.
template <typename T, bool LO>
__global__ void __launch_bounds__(256)
cg_stage_kernel(const T* __restrict__ x, const __grid_constant__ StageShape s, __nv_bfloat16* __restrict__ hi,
                __nv_bfloat16* __restrict__ lo, int ld) {
  __shared__ float tile[64][65];   // [channel][row]
  __shared__ long long base[64];
  chain_next();
  const int r0 = blockIdx.x * 64, c0 = blockIdx.y * 64;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < 64) {
    int img, y, xx;
    base[threadIdx.x] = staged_pixel(s, r0 + threadIdx.x, img, y, xx) ? img * s.sn + y * s.sh + xx * s.sw : -1;
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
    const int piece = threadIdx.x + 256 * i, r = piece >> 3, ch = (piece & 7) * 8;
    if (c0 + ch >= ld) continue;
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
    const size_t at = static_cast<size_t>(r0 + r) * ld + c0 + ch;
    *reinterpret_cast<uint4*>(hi + at) = make_uint4(wh[0], wh[1], wh[2], wh[3]);
    if (LO) *reinterpret_cast<uint4*>(lo + at) = make_uint4(wl[0], wl[1], wl[2], wl[3]);
  }
}

// The main products: A = shifts x channel chunks, B = shifts {0} or {-1, 0} x channel chunks, K = all images.  A correction: A and B =
// channel chunks of two strips, K = a strip.
struct GemmShape {
  int cc;                             // 64-channel chunks
  int main_rows, main_blocks;         // first row and K blocks of the images
  int ta, tb, nsplit;                 // main tiles and K ranges
  int n_shift_a, n_shift_b;
  int shift_a[CG_MAX_SHIFTS];
  int tc;                             // tiles of a correction along a side
  int n_corr;
  int kind_first[4];                  // corrections [kind_first[k], kind_first[k + 1]) have blocks[k] K blocks (rows, columns, pixels)
  int kind_blocks[3];
};
// strips of a correction: first rows of A and B
struct Correction {
  int a, b;
};

template <int PARTS>
struct CgCfg {
  static constexpr int STAGES = 3;
  static constexpr int STAGE_BYTES = PARTS * 2 * G2_A_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
};

// Tables of up to this many words are kernel parameters; larger ones are written to memory first (cg_table_kernel).
constexpr int CG_SMALL = 896;
struct CgTables {
  const int* memory;   // null: `words`
  int corr_words;      // the corrections come first
  int words[CG_SMALL];
};

// One K range of one tile per CTA.  Tiles are stored as 128 rows of 512 bytes whose 16-byte pieces p are at p ^ (row & 7).
template <int PARTS>
__global__ void __launch_bounds__(192, PARTS == 1 ? 2 : 1)
cg_product_kernel(const __grid_constant__ CUtensorMap tm_hi, const __grid_constant__ CUtensorMap tm_lo,
                  const __grid_constant__ GemmShape g, const __grid_constant__ CgTables tab, float* __restrict__ partials,
                  float* __restrict__ tiles, int* status) {
  using Cfg = CgCfg<PARTS>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::STAGES * Cfg::STAGE_BYTES);
  uint64_t* empty_bar = full_bar + Cfg::STAGES;
  uint64_t* acc_bar = empty_bar + Cfg::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // operand chunks: first row and channel
  int row_a[2], row_b[2], ch_a[2], ch_b[2], k0, nkb;
  float* dst;
  const int n_main = g.ta * g.tb * g.nsplit;
  if (static_cast<int>(blockIdx.x) < n_main) {
    const int tile = blockIdx.x / g.nsplit, split = blockIdx.x - tile * g.nsplit;
    const int ia = tile / g.tb, ib = tile - ia * g.tb;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int a = 2 * ia + u, b = 2 * ib + u, sa = a / g.cc, sb = b / g.cc;
      // chunks past the last one read channels past the tensor: zeros
      row_a[u] = g.main_rows + (sa < g.n_shift_a ? g.shift_a[sa] : 0);
      ch_a[u] = (sa < g.n_shift_a ? a - sa * g.cc : g.cc) * 64;
      row_b[u] = g.main_rows + (sb < g.n_shift_b ? sb : 0) - (g.n_shift_b - 1);   // shifts 0, or -1 and 0
      ch_b[u] = (sb < g.n_shift_b ? b - sb * g.cc : g.cc) * 64;
    }
    const int kb0 = static_cast<int>(static_cast<long long>(split) * g.main_blocks / g.nsplit);
    nkb = static_cast<int>(static_cast<long long>(split + 1) * g.main_blocks / g.nsplit) - kb0;
    k0 = kb0 * G2_BK;
    dst = g.nsplit > 1 ? partials + static_cast<size_t>(blockIdx.x) * CG_TILE : tiles + static_cast<size_t>(tile) * CG_TILE;
  } else {
    const int item = blockIdx.x - n_main, per = g.tc * g.tc, p = item / per, t = item - p * per;
    if (tab.memory != nullptr) chain_wait();   // the tables were written by a kernel before
    const Correction q = tab.memory != nullptr ? Correction{tab.memory[2 * p], tab.memory[2 * p + 1]} : Correction{tab.words[2 * p], tab.words[2 * p + 1]};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      row_a[u] = q.a;
      row_b[u] = q.b;
      ch_a[u] = min(2 * (t / g.tc) + u, g.cc) * 64;
      ch_b[u] = min(2 * (t % g.tc) + u, g.cc) * 64;
    }
    k0 = 0;
    nkb = p < g.kind_first[1] ? g.kind_blocks[0] : (p < g.kind_first[2] ? g.kind_blocks[1] : g.kind_blocks[2]);
    dst = tiles + static_cast<size_t>(g.ta * g.tb + item) * CG_TILE;
  }

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(acc_bar, 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 128);
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
          if (lead) umma_bf16(tmem_base, da + k * 128, db + k * 128, idesc, (kb | pr | k) ? 1u : 0u);
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
    tmem_dealloc(tmem_base, 128);
  }
}

// Sums the K ranges of the main tiles, in order.  grid: (16, tiles), a thread has four values and eight ranges in flight.
__global__ void __launch_bounds__(256)
cg_reduce_kernel(const float4* partials, float4* tiles, int nsplit) {
  chain_next();
  chain_wait();
  const int at = blockIdx.x * 256 + threadIdx.x;
  const float4* from = partials + static_cast<size_t>(blockIdx.y) * nsplit * (CG_TILE / 4) + at;
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
  short tiles_b, a0, b0, pad;   // tiles along B of that grid; its first chunks there
};
struct AssembleShape {
  int n, c, taps, khwc;   // rows of the result, channels, filter taps, column order (kh, kw, c)
  int n_products, n_terms;
  float scale, beta;
};

// 32 x 32 patches on or below the diagonal; tables: [ProductAt x products][first term of tap pair t (t + 1) / 2 + t', and one
// past the last][terms: product, + 0x8000 for those that are taken off].
__global__ void __launch_bounds__(256)
cg_assemble_kernel(const float* tiles, const __grid_constant__ AssembleShape a, const __grid_constant__ CgTables tables,
                   float* out, long long ldc) {
  extern __shared__ int tab[];
  __shared__ float patch[32][33];
  chain_wait();
  const int pairs = a.taps * (a.taps + 1) / 2, words = 3 * a.n_products + pairs + 1 + (a.n_terms + 1) / 2;
  for (int i = threadIdx.x; i < words; i += 256)
    tab[i] = tables.memory != nullptr ? tables.memory[tables.corr_words + i] : tables.words[tables.corr_words + i];
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
        const int term = terms[e];
        const ProductAt p = products[term & 0x7fff];
        const int ca = p.a0 + (row >> 6), cb = p.b0 + (col >> 6);
        const int r = (ca & 1) * 64 + (row & 63), c = (cb & 1) * 64 + (col & 63);
        const float* tile = tiles + static_cast<size_t>(p.tile0 + (ca >> 1) * p.tiles_b + (cb >> 1)) * CG_TILE;
        const float w = tile[r * 128 + ((((c >> 2) ^ (r & 7)) << 2) | (c & 3))];
        sum += term & 0x8000 ? -w : w;
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
  const int* tab = tables.memory != nullptr ? tables.memory + tables.corr_words : tables.words + tables.corr_words;
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
    const int term = terms[e];
    const ProductAt p = products[term & 0x7fff];
    const int ca = p.a0 + chunk_i, cb = p.b0 + chunk_j;
    const float* tile = tiles + static_cast<size_t>(p.tile0 + (ca >> 1) * p.tiles_b + (cb >> 1)) * CG_TILE + (ca & 1) * (64 * 128);
    const float sign = term & 0x8000 ? -1.f : 1.f;
    float4 w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int r = ty + 16 * k;
      w[k] = *reinterpret_cast<const float4*>(tile + r * 128 + ((((cb & 1) * 16 + tx) ^ (r & 7)) << 2));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      sum[k][0] += sign * w[k].x;
      sum[k][1] += sign * w[k].y;
      sum[k][2] += sign * w[k].z;
      sum[k][3] += sign * w[k].w;
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

}  // namespace

bool gemm_batch_is_open();

// Returns false, with nothing done, where the general path has to be taken: a batch of products is being recorded (the products
// of the general path run together there), or the shape is outside of what the tables here hold.
bool conv_gram(at::Tensor x, at::Tensor out, int64_t kh, int64_t kw, int64_t ph, int64_t pw, double scale, double beta, bool khwc,
               bool x3) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 4, "x must be a 4-d CUDA tensor");
  TORCH_CHECK(x.scalar_type() == at::kFloat || x.scalar_type() == at::kBFloat16 || x.scalar_type() == at::kHalf, "x must be fp32, bf16 or fp16");
  const int64_t n = x.size(0), c = x.size(1), h = x.size(2), w = x.size(3);
  const int64_t ho = h + 2 * ph - kh + 1, wo = w + 2 * pw - kw + 1, taps = kh * kw, ncol = taps * c;
  if (gemm_batch_is_open() || kh < 1 || kw < 1 || kh > CG_MAX_K || kw > CG_MAX_K || taps < 2 || ph < 0 || pw < 0 || ph >= kh ||
      pw >= kw || ho < 1 || wo < 1 || n < 1 || c < 1 || c > 4096)
    return false;
  TORCH_CHECK(out.is_cuda() && out.scalar_type() == at::kFloat && out.dim() == 2 && out.size(0) == ncol && out.size(1) == ncol &&
                  out.stride(1) == 1, "out must be a [c kh kw, c kh kw] fp32 CUDA matrix with unit column stride");
  const int dev = x.get_device();
  TORCH_CHECK(out.get_device() == dev, "x and out must be on one device");

  // ---- staged rows
  StageShape s;
  std::memset(&s, 0, sizeof(s));
  s.n = static_cast<int>(n);
  s.c = static_cast<int>(c);
  s.h = static_cast<int>(h);
  s.w = static_cast<int>(w);
  s.hp = static_cast<int>(h + kh - 1);
  s.wp = static_cast<int>(w + kw - 1);
  s.ey = static_cast<int>(kh - 1 - ph);
  s.ex = static_cast<int>(kw - 1 - pw);
  if (s.ey > h || s.ex > w) return false;
  const long long images = static_cast<long long>(n) * s.hp * s.wp;
  const long long row_len = (static_cast<long long>(n) * s.wp + 63) / 64 * 64, col_len = (static_cast<long long>(n) * s.hp + 63) / 64 * 64;
  if (images + 2 * s.ey * row_len + 2 * s.ex * col_len + 4ll * s.ey * s.ex * (n + 64) > (1ll << 30)) return false;
  s.lead = 64;
  s.row_len = static_cast<int>(row_len);
  s.col_len = static_cast<int>(col_len);
  s.pix_len = ceil_to(n, 64);
  s.rows0 = s.lead + ceil_to(images, 64);
  s.cols0 = s.rows0 + 2 * s.ey * s.row_len;
  s.pix0 = s.cols0 + 2 * s.ex * s.col_len;
  s.total = s.pix0 + 4 * s.ey * s.ex * s.pix_len;
  s.sn = x.stride(0);
  s.sc = x.stride(1);
  s.sh = x.stride(2);
  s.sw = x.stride(3);

  // ---- products: main ones by difference, corrections by strips
  GemmShape g;
  std::memset(&g, 0, sizeof(g));
  g.cc = static_cast<int>((c + 63) / 64);
  g.main_rows = s.lead;
  g.main_blocks = (s.rows0 - s.lead) / 64;
  g.n_shift_b = g.cc == 1 ? 2 : 1;   // a chunk of 64 channels takes two shifts to fill a tile
  std::vector<int> main_of((kh) * (2 * kw - 1), -1);   // product of a difference (dy, dx + kw - 1)
  std::vector<ProductAt> products;
  for (int dy = 0; dy < kh; ++dy)
    for (int dx = dy == 0 ? 0 : -static_cast<int>(kw) + 1; dx < kw; dx += g.n_shift_b) {
      // against B's shift of -1 + e (or 0 alone) a shift of `last` - 1 (`last`) gives the difference `last` - e
      const int last = dx + g.n_shift_b - 1;
      if (g.n_shift_a >= CG_MAX_SHIFTS) return false;
      g.shift_a[g.n_shift_a] = dy * s.wp + last - (g.n_shift_b - 1);
      for (int e = 0; e < g.n_shift_b; ++e) {
        const int d = last - e;
        if (d >= kw) continue;
        main_of[dy * (2 * kw - 1) + d + kw - 1] = static_cast<int>(products.size());
        products.push_back({0, 0, static_cast<short>(g.n_shift_a * g.cc), static_cast<short>(e * g.cc), 0});
      }
      ++g.n_shift_a;
    }
  const int n_main_products = static_cast<int>(products.size());
  g.ta = (g.n_shift_a * g.cc + 1) / 2;
  g.tb = (g.n_shift_b * g.cc + 1) / 2;
  g.tc = (g.cc + 1) / 2;
  for (ProductAt& p : products) p.tiles_b = static_cast<short>(g.tb);

  // strip of an image row, column or pixel (the first or last ones)
  auto edge_of = [](int at, int edges, int extent) { return at < edges ? at : at - (extent - 2 * edges); };
  std::vector<Correction> corr[3];
  const int nr = 2 * s.ey, nc = 2 * s.ex;
  std::vector<int> known[3] = {std::vector<int>(nr * nr * (2 * kw - 1), -1), std::vector<int>(nc * nc * kh, -1),
                               std::vector<int>(nr * nc * nr * nc, -1)};
  auto correction = [&](int kind, int key, int a, int b) {
    int& at = known[kind][key];
    if (at < 0) {
      at = static_cast<int>(corr[kind].size());
      corr[kind].push_back({a, b});
    }
    return at;
  };
  struct Term {
    int kind, index, off;   // kind 3: a main product
  };
  std::vector<Term> terms;
  std::vector<int> first(1, 0);
  for (int t = 0; t < taps; ++t)
    for (int u = 0; u <= t; ++u) {
      const int ty = static_cast<int>(t / kw), tx = static_cast<int>(t % kw), uy = static_cast<int>(u / kw), ux = static_cast<int>(u % kw);
      const int dy = ty - uy, dx = tx - ux, ax = std::abs(dx), mx = std::min(tx, ux);
      terms.push_back({3, main_of[dy * (2 * kw - 1) + dx + kw - 1], 0});
      // image rows (of the pixel under the earlier tap) and columns (the left one of the two pixels) outside of the window
      int rows[2 * CG_MAX_K], cols[2 * CG_MAX_K], n_rows = 0, n_cols = 0;
      auto add_row = [&](int i) {
        if (i >= 0 && i + dy < s.h) rows[n_rows++] = i;   // otherwise there is no such pair of pixels
      };
      auto add_col = [&](int l) {
        if (l >= 0 && l + ax < s.w) cols[n_cols++] = dx >= 0 ? l : l + ax;   // column of the pixel under the earlier tap
      };
      for (int i = 0; i < uy - ph; ++i) add_row(i);
      for (int i = 0; i < static_cast<int>(kh) - 1 - ph - ty; ++i) add_row(s.h - dy - 1 - i);
      for (int i = 0; i < mx - pw; ++i) add_col(i);
      for (int i = 0; i < static_cast<int>(kw) - 1 - pw - (mx + ax); ++i) add_col(s.w - ax - 1 - i);
      for (int i = 0; i < n_rows; ++i) {
        const int ea = edge_of(rows[i] + dy, s.ey, s.h), eb = edge_of(rows[i], s.ey, s.h);
        const int key = (ea * nr + eb) * (2 * static_cast<int>(kw) - 1) + dx + static_cast<int>(kw) - 1;
        terms.push_back({0, correction(0, key, s.rows0 + ea * s.row_len + dx, s.rows0 + eb * s.row_len), 1});
      }
      for (int i = 0; i < n_cols; ++i) {
        const int ea = edge_of(cols[i] + dx, s.ex, s.w), eb = edge_of(cols[i], s.ex, s.w);
        terms.push_back({1, correction(1, (ea * nc + eb) * static_cast<int>(kh) + dy, s.cols0 + ea * s.col_len + dy, s.cols0 + eb * s.col_len), 1});
      }
      for (int i = 0; i < n_rows; ++i)
        for (int l = 0; l < n_cols; ++l) {
          const int ea = edge_of(rows[i] + dy, s.ey, s.h) * nc + edge_of(cols[l] + dx, s.ex, s.w);
          const int eb = edge_of(rows[i], s.ey, s.h) * nc + edge_of(cols[l], s.ex, s.w);
          terms.push_back({2, correction(2, ea * nr * nc + eb, s.pix0 + ea * s.pix_len, s.pix0 + eb * s.pix_len), 0});
        }
      first.push_back(static_cast<int>(terms.size()));
    }
  std::vector<Correction> all_corr;
  for (int k = 0; k < 3; ++k) {
    g.kind_first[k] = static_cast<int>(all_corr.size());
    all_corr.insert(all_corr.end(), corr[k].begin(), corr[k].end());
  }
  g.n_corr = g.kind_first[3] = static_cast<int>(all_corr.size());
  g.kind_blocks[0] = s.row_len / 64;
  g.kind_blocks[1] = s.col_len / 64;
  g.kind_blocks[2] = s.pix_len / 64;
  for (int p = 0; p < g.n_corr; ++p)
    products.push_back({g.ta * g.tb + p * g.tc * g.tc, static_cast<short>(g.tc), 0, 0, 0});
  if (products.size() > CG_MAX_PRODUCTS || terms.size() > 8192 || g.n_corr * g.tc * g.tc > 16384) return false;

  // ---- K ranges: one CTA for each, as many as are resident beside the long corrections
  const int resident = g2_sm_count(dev) * (x3 ? 1 : 2), per_corr = g.tc * g.tc;
  const int long_corr = (2 * g.kind_blocks[0] >= 8 ? (g.kind_first[1] - g.kind_first[0]) + (g.kind_first[2] - g.kind_first[1]) : 0) * per_corr;
  const int main_tiles = g.ta * g.tb;
  g.nsplit = std::max(1, std::min({(resident - std::min(long_corr, resident / 2)) / main_tiles, g.main_blocks / 4, 64}));

  c10::cuda::CUDAGuard guard(dev);
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream(dev).stream();
  const int ld = ceil_to(c, 8);
  auto bytes = at::TensorOptions().dtype(at::kByte).device(at::kCUDA, dev);
  auto f32 = at::TensorOptions().dtype(at::kFloat).device(at::kCUDA, dev);
  at::Tensor staged = at::empty({(x3 ? 2 : 1) * static_cast<int64_t>(s.total) * ld * 2}, bytes);
  __nv_bfloat16* hi = reinterpret_cast<__nv_bfloat16*>(staged.data_ptr());
  __nv_bfloat16* lo = x3 ? hi + static_cast<size_t>(s.total) * ld : nullptr;
  at::Tensor partials;
  if (g.nsplit > 1) partials = at::empty({static_cast<int64_t>(main_tiles) * g.nsplit * CG_TILE}, f32);
  at::Tensor tiles = at::empty({static_cast<int64_t>(main_tiles + g.n_corr * per_corr) * CG_TILE}, f32);

  // tables: corrections, products, first terms, terms
  std::vector<int> host;
  host.reserve(2 * all_corr.size() + 3 * products.size() + first.size() + terms.size() / 2 + 8);
  for (const Correction& q : all_corr) {
    host.push_back(q.a);
    host.push_back(q.b);
  }
  const size_t asm_at = host.size();
  static_assert(sizeof(ProductAt) == 12, "tables hold three words per product");
  host.resize(asm_at + 3 * products.size());
  std::memcpy(host.data() + asm_at, products.data(), products.size() * sizeof(ProductAt));
  host.insert(host.end(), first.begin(), first.end());
  const size_t terms_at = host.size();
  host.resize(terms_at + (terms.size() + 1) / 2, 0);
  unsigned short* ht = reinterpret_cast<unsigned short*>(host.data() + terms_at);
  for (size_t i = 0; i < terms.size(); ++i) {
    const Term& q = terms[i];
    const int index = q.kind == 3 ? q.index : n_main_products + g.kind_first[q.kind] + q.index;
    ht[i] = static_cast<unsigned short>(index | (q.off ? 0x8000 : 0));
  }
  CgTables tables;
  tables.memory = nullptr;
  tables.corr_words = static_cast<int>(asm_at);
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

  const dim3 sgrid(s.total / 64, (ld + 63) / 64);
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
  const int items = main_tiles * g.nsplit + g.n_corr * per_corr;
  float* dp = g.nsplit > 1 ? partials.data_ptr<float>() : nullptr;
  auto run = [&](auto kernel, int smem) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    launch_chained(kernel, dim3(items), dim3(192), smem, stream, tm_hi, tm_lo, g, tables, dp, tiles.data_ptr<float>(), status);
  };
  if (x3)
    run(cg_product_kernel<2>, CgCfg<2>::SMEM_BYTES);
  else
    run(cg_product_kernel<1>, CgCfg<1>::SMEM_BYTES);
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
  if (g.nsplit > 1) {
    launch_chained(cg_reduce_kernel, dim3(CG_TILE / 4 / 256, main_tiles), dim3(256), 0, stream, reinterpret_cast<const float4*>(dp),
                   reinterpret_cast<float4*>(tiles.data_ptr<float>()), g.nsplit);
    B200_CUDA_CHECK(cudaGetLastError());
    count_launch();
  }
  AssembleShape a;
  a.n = static_cast<int>(ncol);
  a.c = static_cast<int>(c);
  a.taps = static_cast<int>(taps);
  a.khwc = khwc;
  a.n_products = static_cast<int>(products.size());
  a.n_terms = static_cast<int>(terms.size());
  a.scale = static_cast<float>(scale);
  a.beta = static_cast<float>(beta);
  float* result = out.data_ptr<float>();
  if (khwc && c % 64 == 0) {
    const int nb = a.n / 64;
    const bool vec = out.stride(0) % 4 == 0 && (reinterpret_cast<uintptr_t>(result) & 15) == 0;
    launch_chained(cg_assemble_blocks_kernel, dim3(nb * (nb + 1) / 2), dim3(256), 0, stream, tiles.data_ptr<float>(), a, tables, result, out.stride(0), vec);
  } else {
    const int nb = (a.n + 31) / 32, tab_bytes = static_cast<int>(host.size() - asm_at) * 4;
    launch_chained(cg_assemble_kernel, dim3(nb * (nb + 1) / 2), dim3(256), tab_bytes, stream, tiles.data_ptr<float>(), a, tables, result, out.stride(0));
  }
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
  return true;
}

}  // namespace b200
