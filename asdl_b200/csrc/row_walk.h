// Walk of bandwidth-bound kernels over a row-major [rows, n] matrix in 16-byte vectors: a thread keeps ONE vector column
// (what depends on the column stays in registers, and no index is divided inside the loop) and goes down the rows;
// the row lanes of a CTA are consecutive rows, so its accesses cover consecutive memory when its groups span a row.
#pragma once
#include <algorithm>

namespace b200 {

struct Walk {
  int groups, lanes, chunks;   // vector columns and row lanes of a CTA of 256 threads, CTAs across a row
};

// The split of `vecs` vectors per row with the fewest idle threads; a CTA covers at least eight vectors (128 bytes) of
// a row unless the row is shorter.
inline Walk walk_plan(int vecs) {
  Walk best{0, 0, 0};
  long long best_active = -1;
  for (int chunks = (vecs + 255) / 256; chunks <= vecs; ++chunks) {
    const int groups = (vecs + chunks - 1) / chunks;
    if (best_active >= 0 && (groups < 8 || chunks > 64 + (vecs + 255) / 256)) break;
    const int used = (vecs + groups - 1) / groups;                              // chunks that have work
    const long long active = static_cast<long long>(vecs) * (256 / groups) * 4096 / used;   // ~ threads with work per CTA
    if (active > best_active) {
      best_active = active;
      best = {groups, 256 / groups, used};
    }
    if (active == 256 * 4096) break;   // no idle thread: the search takes up to 0.7 us of host time
  }
  return best;
}

// One wave of CTAs (`per_sm` resident on each SM), fewer where a thread would have no row.  The CTAs across a row are on y,
// at most MAX_WALK_CHUNKS of them.  On x they cost 25 % where the loads are scalar (16 x 1000003 fp32 -> hi, lo: 25.0 and
// 31.3 us): neighbouring CTAs then share a row instead of a column.
constexpr int MAX_WALK_CHUNKS = 65535;
inline dim3 walk_grid(const Walk& w, long long rows, int per_sm) {
  const long long most = (rows + w.lanes - 1) / w.lanes;
  const long long wave = std::max<long long>(1, (148LL * per_sm + w.chunks - 1) / w.chunks);
  return dim3(static_cast<unsigned>(std::min(most, wave)), static_cast<unsigned>(w.chunks));
}

// The same for any number of them: the CTA across a row is blockIdx.z * gridDim.y + blockIdx.y, the last ones may have no work.
inline dim3 walk_grid_layers(const Walk& w, long long rows, int per_sm) {
  dim3 grid = walk_grid(w, rows, per_sm);
  grid.z = (grid.y + MAX_WALK_CHUNKS - 1) / MAX_WALK_CHUNKS;
  grid.y = (grid.y + grid.z - 1) / grid.z;
  return grid;
}

}  // namespace b200
