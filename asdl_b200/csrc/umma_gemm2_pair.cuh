// CTA-pair flavour of the persistent tcgen05 GEMM / SYRK (umma_gemm2.cuh): `tcgen05.mma.cta_group::2`.
//
// Two CTAs of a cluster - on the two SMs of one TPC - share every tile.  A pair tile is 256 x 256:
// CTA r of the pair stages rows [128 r, 128 r + 128) of the A tile and columns [128 r, 128 r + 128) of
// the B tile in its own shared memory (32 KiB per 64-wide K block, a ring of six stages), the leader CTA
// (rank 0) issues one 256 x 256 x 16 MMA per K step that reads both CTAs' shared memory, and every
// CTA ends up with its 128 rows of the 256-column accumulator in its own TMEM.  Per FLOP a pair
// moves two thirds of the shared-memory bytes of a 128 x 256 tile and half those of a 128 x 128 tile.
//
// With PARTS = 2 ("bf16x3" products of (hi, lo) pairs, G2F_SPLIT2) a stage holds both parts of both operands, loaded once
// (64 KiB per CTA and K block, a ring of three), and three part products are issued from it: (lo, hi) (hi, lo) (hi, hi).
// 128 x 256 tiles of single CTAs take 96 KiB for the same work in a ring of two, which left the load latency exposed (1.6 us per
// K block against 0.83 of the tensor cores); three segments of the plain flavour load both operands for each part product.
// (lo, hi) and (hi, lo) go to an accumulator of their own, which the epilogue adds: the tensor core truncates with every addition,
// by a last bit of the accumulator, and so only a third of the additions meet the large one.  The two accumulators of a tile
// take all of TMEM, so a pair's next tile waits for its epilogue; most launches are one wave.
// 1024 x 4096 between fp32 factors: 183 -> 137 us with the casts (graph replay), error against 64 bits 1.0e-5 -> 8.1e-6.
//
// HALVES = 2: tiles of 256 x 512, whose two 256-column halves take the two accumulators.  Both CTAs bring 48 KiB per K block of 1024
// tensor clocks instead of 32 KiB per 512, which is less than L2 delivers (53 bytes per clock and SM) instead of more; a half
// past the diagonal of a symmetric result is neither loaded nor multiplied.  A pair's next tile waits for its epilogue; gemm2_pair.cu has
// the rule and what it measured.
//
// Signals inside a pair:
//   full[s]      lives in the leader.  The leader's producer arms it with the bytes of BOTH CTAs'
//                loads; each CTA's TMA loads (no cluster multicast: every CTA fetches its own
//                tiles) complete on it.
//   empty[s]     one per CTA; `tcgen05.commit` with a CTA mask arrives on both when the MMAs that
//                read the stage have finished.
//   acc_full[b]  one per CTA, signalled the same way when a tile's last MMA has finished.
//   acc_empty[b] lives in the leader and counts the epilogue warps of both CTAs (the peer's arrive
//                through the cluster's shared-memory window).
// Every wait is bounded in wall time as in the other flavours; the cluster barriers at the start
// and the end are reached by every thread on every path, error paths included.
//
// A problem of this flavour uses the tensor maps of the 128-wide flavour (boxes of 128 rows) and
// the tile grid and split-K scratch layout of the 256-wide flavour: the two halves of a pair tile
// are exactly the 128 x 256 tiles (2 TM + r, TN) of that grid, so the split-K reduction kernel of
// the wide flavour finishes a pair launch unchanged.
#pragma once
#include "umma_gemm2.cuh"

namespace b200 {

template <int PARTS, int HALVES>
struct G2PairCfg {
  static_assert(PARTS == 1 || HALVES == 1, "one or the other takes both accumulators");
  static constexpr int STAGE_BYTES = PARTS * (1 + HALVES) * G2_A_BYTES;   // this CTA's A rows and B columns of one K block
  static constexpr int STAGES = 6 * 2 * G2_A_BYTES / STAGE_BYTES;
};
constexpr int G2P_EPI_WARPS = 8;
constexpr int G2P_THREADS = 64 + 32 * G2P_EPI_WARPS;
constexpr int G2P_TMEM_COLS = 512;                          // two 256-column accumulators
constexpr int G2P_PATCH = 32;                               // columns of a result that an epilogue warp stages at a time
constexpr int G2P_SMEM_BYTES = 6 * 2 * G2_A_BYTES + 1024 + 256 + G2P_EPI_WARPS * 32 * G2P_PATCH * 4;

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// address of the same shared-memory object in CTA `rank` of the cluster (shared::cluster window)
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 2-D tiled load into this CTA's shared memory whose completion is counted on a barrier that may
// live in the other CTA of the pair (`bar_cluster_addr` is a shared::cluster address).
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const void* tmap, uint32_t bar_cluster_addr, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, "
      "{%3, %4}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar_cluster_addr), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
// `bar` (same offset in both CTAs of the pair) observes completion of all MMAs issued so far.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(mask)
      : "memory");
}

struct G2PairItem {
  int TM, TN;        // pair tile (256 x 256 units)
  int kb0, nkb;      // K blocks of this split
  int split;
};

template <int HALVES>
__device__ __forceinline__ G2PairItem g2_pair_decode(const GemmProblem2& P, int idx) {
  G2PairItem it;
  const int t = idx / P.nsplit;
  it.split = idx - t * P.nsplit;
  if (P.flags & G2F_SYM) {
    int TM = 0, rem = t;
    while (rem > TM / HALVES) {   // row TM of the pair grid holds TM / HALVES + 1 tiles
      rem -= TM / HALVES + 1;
      ++TM;
    }
    it.TM = TM;
    it.TN = rem;
  } else {
    const int across = (P.tiles_n + HALVES - 1) / HALVES;
    it.TM = t / across;
    it.TN = t - it.TM * across;
  }
  const int kb_total = (P.K + G2_BK - 1) / G2_BK;
  it.kb0 = static_cast<int>((static_cast<long long>(it.split) * kb_total) / P.nsplit);
  const int kb1 = static_cast<int>((static_cast<long long>(it.split + 1) * kb_total) / P.nsplit);
  it.nkb = kb1 - it.kb0;
  return it;
}

// Halves of a tile that have columns to compute
template <int HALVES>
__device__ __forceinline__ int g2_pair_halves(const GemmProblem2& P, const G2PairItem& w) {
  if (HALVES == 1) return 1;
  return (P.flags & G2F_SYM ? w.TN * HALVES + 1 <= w.TM : w.TN * HALVES + 1 < P.tiles_n) ? 2 : 1;
}

template <int PARTS, int HALVES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(G2P_THREADS, 1)
umma_gemm2_pair_kernel(const __grid_constant__ GemmProblem2 P0, int n_work) {
  constexpr int STAGES = G2PairCfg<PARTS, HALVES>::STAGES, STAGE_BYTES = G2PairCfg<PARTS, HALVES>::STAGE_BYTES;
  constexpr bool ALL_TMEM = PARTS > 1 || HALVES > 1;   // one tile takes both accumulators
  constexpr int BN = 256;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* acc_full = empty_bar + STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

  const GemmProblem2& P = P0;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const bool leader = rank == 0;
  const int pair_id = blockIdx.x >> 1;
  const int n_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 2 * G2P_EPI_WARPS);  // the epilogue warps of both CTAs
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, G2P_TMEM_COLS);
    tmem_relinquish_pair();
  }
  chain_wait();   // operands and outputs: nothing is touched before
  tc_fence_before_sync();
  cluster_sync_all();   // barriers of both CTAs are initialised before anything arrives on them
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) --------------------------
    if (lane == 0) {
      const bool a_k = (P.flags & G2F_A_KMAJOR) != 0;
      const bool b_k = (P.flags & G2F_B_KMAJOR) != 0;
      uint32_t it = 0;
      bool ok = true;
      for (int wi = pair_id; wi < n_work && ok; wi += n_pairs) {
        const G2PairItem w = g2_pair_decode<HALVES>(P, wi);
        const int a_mn = w.TM * 256 + static_cast<int>(rank) * G2_BM;
        const int b_mn = w.TN * 256 * HALVES + static_cast<int>(rank) * G2_BM;
        const int halves = g2_pair_halves<HALVES>(P, w);
        const int nseg = PARTS > 1 ? 1 : P.nseg;
        for (int seg = 0; seg < nseg && ok; ++seg) {
          for (int kb = 0; kb < w.nkb; ++kb, ++it) {
            const int s = it % STAGES;
            const uint32_t ph = (it / STAGES) & 1;
            if (!mbar_wait(&empty_bar[s], ph ^ 1)) {
              set_error(P.status, ERR_WAIT_EMPTY);
              ok = false;
              break;
            }
            if (leader) mbar_expect_tx(&full_bar[s], HALVES > 1 ? 2 * (1 + halves) * G2_A_BYTES : 2 * STAGE_BYTES);
            const uint32_t bar = mapa_shared(smem_u32(&full_bar[s]), 0);
            const int k = (w.kb0 + kb) * G2_BK;
#pragma unroll
            for (int part = 0; part < PARTS; ++part) {
              const CUtensorMap* ta = &P.tmA[PARTS > 1 ? part : seg];
              const CUtensorMap* tb = &P.tmB[PARTS > 1 ? part : seg];
              uint8_t* sA = smem + s * STAGE_BYTES + part * G2_A_BYTES;
              uint8_t* sB = sA + PARTS * G2_A_BYTES;
              if (a_k) {
                tma_load_2d_pair(sA, ta, bar, k, a_mn);
              } else {
                tma_load_2d_pair(sA, ta, bar, a_mn, k);
                tma_load_2d_pair(sA + G2_BK * 128, ta, bar, a_mn + 64, k);
              }
#pragma unroll
              for (int h = 0; h < HALVES; ++h) {
                if (h >= halves) break;
                if (b_k) {
                  tma_load_2d_pair(sB + h * G2_A_BYTES, tb, bar, k, b_mn + 256 * h);
                } else {
                  tma_load_2d_pair(sB + h * G2_A_BYTES, tb, bar, b_mn + 256 * h, k);
                  tma_load_2d_pair(sB + h * G2_A_BYTES + G2_BK * 128, tb, bar, b_mn + 256 * h + 64, k);
                }
              }
            }
          }
        }
      }
      if (!ok && leader) {
        // give copies that are still in flight a bounded chance to land before teardown
        const uint32_t pending = it < static_cast<uint32_t>(STAGES) ? it : static_cast<uint32_t>(STAGES);
        for (uint32_t j = 0; j < pending; ++j) {
          const uint32_t jt = it - 1 - j;
          mbar_wait(&full_bar[jt % STAGES], (jt / STAGES) & 1);
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader CTA only) ----------------------
    if (leader && lane == 0) {
      const bool a_k = (P.flags & G2F_A_KMAJOR) != 0;
      const bool b_k = (P.flags & G2F_B_KMAJOR) != 0;
      const uint32_t idesc = make_idesc_bf16(256, BN, !a_k, !b_k);
      uint32_t it = 0, ch = 0;
      bool ok = true;
      for (int wi = pair_id; wi < n_work && ok; wi += n_pairs) {
        const G2PairItem w = g2_pair_decode<HALVES>(P, wi);
        if (w.nkb <= 0) continue;
        const int halves = g2_pair_halves<HALVES>(P, w);
        const uint32_t ab = ALL_TMEM ? 0 : ch & 1;
        if (!mbar_wait(&acc_empty[ab], (ALL_TMEM ? ch & 1 : (ch >> 1) & 1) ^ 1)) {
          set_error(P.status, ERR_WAIT_ACC);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        const uint32_t tacc = tmem_base + ab * BN;
        uint32_t first = 1;
        const int nseg = PARTS > 1 ? 1 : P.nseg;
        for (int seg = 0; seg < nseg && ok; ++seg) {
          for (int kb = 0; kb < w.nkb; ++kb, ++it) {
            const int s = it % STAGES;
            if (!mbar_wait(&full_bar[s], (it / STAGES) & 1)) {
              set_error(P.status, ERR_WAIT_FULL);
              ok = false;
              break;
            }
            tc_fence_after_sync();
            constexpr int NPROD = PARTS > 1 ? 3 : 1;
            constexpr int PART_A[3] = {PARTS - 1, 0, 0};   // (lo, hi) (hi, lo) (hi, hi)
            constexpr int PART_B[3] = {0, PARTS - 1, 0};
#pragma unroll
            for (int pr = 0; pr < NPROD; ++pr) {
              const uint32_t aA = smem_u32(smem + s * STAGE_BYTES) + PART_A[pr] * G2_A_BYTES;
              const uint32_t aB = smem_u32(smem + s * STAGE_BYTES) + (PARTS + PART_B[pr]) * G2_A_BYTES;
#pragma unroll
              for (int k = 0; k < G2_BK / 16; ++k) {
                const uint64_t da = a_k ? make_smem_desc_sw128(aA + k * 32, 16, 1024)
                                        : make_smem_desc_sw128(aA + k * 16 * 128, G2_BK * 128, 1024);
                const uint64_t db = b_k ? make_smem_desc_sw128(aB + k * 32, 16, 1024)
                                        : make_smem_desc_sw128(aB + k * 16 * 128, G2_BK * 128, 1024);
                if (PARTS > 1) {
                  const bool begins = kb == 0 && k == 0 && pr != 1;
                  umma_bf16_pair(tacc + (pr < 2 ? BN : 0), da, db, idesc, begins ? 0u : 1u);
                } else {
                  umma_bf16_pair(tacc, da, db, idesc, first ? 0u : 1u);
                  if (HALVES > 1 && halves > 1) umma_bf16_pair(tacc + BN, da, db + (G2_A_BYTES >> 4), idesc, first ? 0u : 1u);
                  first = 0;
                }
              }
            }
            umma_commit_pair(&empty_bar[s]);
          }
        }
        if (ok) umma_commit_pair(&acc_full[ab]);
        ++ch;
      }
    }
  } else {
    // ------------------------------ epilogue (both CTAs) ------------------------------
    const int q = warp & 3;                                   // TMEM lane quarter this warp may access
    constexpr int COLS = HALVES * BN / (G2P_EPI_WARPS / 4);   // columns per warp
    const int col_base = ((warp - 2) >> 2) * COLS;
    const int row = q * 32 + lane;
    const G2Epi E = g2_epi(P);
    const bool sym = (E.flags & G2F_SYM) != 0;
    const bool atomic = (E.flags & G2F_ATOMIC) != 0;
    const bool to_ws = E.nsplit > 1 && !atomic, staged = !to_ws && (PARTS > 1 ? g2_only_c(E) : g2_staged(E)), images = g2_only_images(E);
    const uint32_t stg = smem_u32(smem + STAGES * STAGE_BYTES + 256) + (warp - 2) * 32 * G2P_PATCH * 4;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    uint32_t ch = 0;
    bool ok = true;
    for (int wi = pair_id; wi < n_work && ok; wi += n_pairs) {
      const G2PairItem w = g2_pair_decode<HALVES>(P, wi);
      const int c_row = w.TM * 256 + static_cast<int>(rank) * G2_BM;
      const int c_col = w.TN * 256 * HALVES;
      const int tm = 2 * w.TM + static_cast<int>(rank);
      const int tile_id = sym ? w.TM * (w.TM + 1) + static_cast<int>(rank) * (w.TM + 1) + w.TN : tm * E.full->tiles_n + w.TN;
      const int gr = c_row + row;
      const bool have = w.nkb > 0;
      const uint32_t ab = ALL_TMEM ? 0 : ch & 1;
      const uint32_t from = tmem_base + lane_addr + ab * BN + col_base;
      auto ready = [&] {
        bool there = !have || mbar_wait(&acc_full[ab], ALL_TMEM ? ch & 1 : (ch >> 1) & 1);
        if (!there) set_error(P.status, ERR_WAIT_ACC);
        there = __all_sync(0xffffffffu, there);
        tc_fence_after_sync();
        return there;
      };
      auto read = [&](int c, float (&v)[G2P_PATCH]) {
        uint32_t r[G2P_PATCH] = {};
        if (have) {
          tmem_ld_32x32(from + c, r);
          tmem_ld_wait();
        }
#pragma unroll
        for (int j = 0; j < G2P_PATCH; ++j) v[j] = __uint_as_float(r[j]);
        if (PARTS > 1 && have) {   // the accumulator of the small part products
          tmem_ld_32x32(from + BN + c, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < G2P_PATCH; ++j) v[j] += __uint_as_float(r[j]);
        }
      };
      auto release = [&] {   // this warp's share has been read: hand the accumulator back to the leader
        tc_fence_before_sync();
        __syncwarp();
        if (have && lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&acc_empty[ab]), 0));
      };
      if (staged) {
        ok = g2_store_columns<G2P_PATCH, COLS>(E, stg, c_row, c_row + q * 32, c_col + col_base, lane, ready, read, release);
        if (have) ++ch;
        continue;
      }
      ok = ready();
      if (!ok) break;
      float* const part = E.ws + (static_cast<size_t>(tile_id) * E.nsplit + w.split) * (G2_BM * BN);
      // one patch after the other: unrolled, each kind of output is too much code for a tile (instruction fetch)
#pragma unroll 1
      for (int c = 0; c < COLS; c += G2P_PATCH) {
        float v[G2P_PATCH];
        read(c, v);
        if (c + G2P_PATCH == COLS) release();
        if (c_row >= E.M) continue;   // the lower half of the last pair row of an odd tile count: nothing to write
        const int col0 = col_base + c, gc0 = c_col + col0;
        if (HALVES == 1 && to_ws) {   // tiles of 512 columns are not split
          g2_store_partial(part, v, row, col0);
          continue;
        }
        // a symmetric problem's pair tile on the diagonal reaches past the diagonal block: skip that part
        const bool beyond = sym && (gc0 / G2_BM) > (c_row / G2_BM);
        const bool diag = sym && (gc0 / G2_BM) == (c_row / G2_BM);
        if (gc0 >= E.N || beyond) continue;
        if (PARTS > 1 && images)
          g2_store_images(E, stg, v, c_row + q * 32, gc0, lane);
        else if (diag && gc0 > gr)
          continue;
        else if (atomic)
          g2_reduce_chunk(E, v, gr, gc0, diag);
        else
          g2_store_chunk(E, v, gr, gc0, diag);
      }
      if (have) ++ch;
    }
  }

  tc_fence_before_sync();
  cluster_sync_all();   // nobody frees TMEM or leaves while the other CTA may still signal it
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc_pair(tmem_base, G2P_TMEM_COLS);
  }
}

}  // namespace b200
