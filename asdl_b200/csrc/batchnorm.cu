// Training-mode BatchNorm2d for NHWC (channels_last) bf16 activations with fp32 parameters and
// statistics.  The activation tensor is treated as a row-major [rows = n*h*w, c] matrix; every
// thread owns 8 consecutive channels (one 16-byte load) and walks down the rows, so all global
// accesses are full 128-byte lines and each pass moves exactly the bytes it has to:
//
//   forward    bn_sums (read x)            -> per-split partial sums and sums of squares
//              bn_fwd_finalize             -> mean, 1/std, running statistics, scale/shift
//              bn_apply   (read x, write y)   y = x * scale + shift
//   backward   bn_bwd_sums (read x, dy)    -> per-split partial sums of dy and dy * xhat
//              bn_bwd_finalize             -> dweight, dbias and the three dx coefficients
//              bn_dx      (read x, dy, write dx)
//
// The last kernel of a direction walks the rows from the end, where the sums kernel has stopped: what that one has read last is
// still in L2, and what it reads itself goes first when room is needed.  Of the backward pass of 32 x 256 x 56 x 56 (x and dy are 103 MB)
// bn_dx reads 38 MB from memory instead of 78, the forward's bn_apply 3 of 51.
//
// Both directions pass after pass in graphs, before and with the ring, packed arithmetic, mask bits and that order: 32 x 256 x 56 x 56 with
// residual and ReLU 111.5 -> 88.6 us, with ReLU alone 90.6 -> 68.4, 32 x 512 x 28 x 28 45.4 -> 39.7, 32 x 128 x 28 x 28 29.7 -> 21.5,
// 32 x 512 x 7 x 7 17.0 -> 17.0.  A sums kernel takes 11 us for 51 MB where a plain read of them takes 9.3; its CTAs come in waves that
// load and add in step.  Tried and not taken: one cooperative launch per direction with the rows kept in shared memory (16 warps per SM
// cannot issue fast enough, and small layers pay 3 - 9 us: 122.6 us, 8 x 64 x 14 x 14 15.4 -> 33.3), and CTAs that walk over several
// splits (the same time, small layers 1 us more).
//
// The three kernels of a direction are chained (chained_launch.h), which takes about 1 us off a direction: the forward of 8 x 64 x 14 x 14
// in a graph 7.0 -> 5.8 us, of 32 x 512 x 7 x 7 7.9 -> 6.6.  In large layers and whole steps it is within what repeats differ by (32 x 256 x
// 56 x 56, both directions, 127 and 125 us; ten K-FAC steps of a bottleneck ResNet 29.35 and 29.35 ms).
//
// Partial sums are combined in double precision by the finalize kernels (one warp per channel),
// which keeps var = E[x^2] - E[x]^2 accurate.
#include <cuda_bf16.h>

#include "chained_launch.h"
#include "host_utils.h"
#include "packed_fp32.cuh"
#include "row_walk.h"

#include <type_traits>

namespace b200 {

namespace {

constexpr int GROUPS = 8;    // channel groups of 8 channels per CTA -> 64 channels
constexpr int LANES = 32;    // row lanes of a split
constexpr int THREADS = GROUPS * LANES;
constexpr int MIN_ROWS = 512;   // of a split, where there are more

// Sums and transforms work on packed pairs of values: issue slots are what these kernels run out of beside the memory.

// 8 bf16 values as 4 words -> 4 pairs, and back
__device__ __forceinline__ void unpack(const uint32_t (&w)[4], f32x2 (&out)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) out[i] = pack2(w[i] << 16, w[i] & 0xffff0000u);
}
__device__ __forceinline__ uint32_t pack(f32x2 v) {
  const float2 f = unpack2(v);
  const __nv_bfloat162 h = __floats2bfloat162_rn(f.x, f.y);
  return reinterpret_cast<const uint32_t&>(h);
}
__device__ __forceinline__ uint32_t relu2(uint32_t w) {
  const __nv_bfloat162 h = __hmax2(reinterpret_cast<const __nv_bfloat162&>(w), __float2bfloat162_rn(0.f));
  return reinterpret_cast<const uint32_t&>(h);
}
__device__ __forceinline__ void load_pairs(const float* p, f32x2 (&out)[4]) {
  const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p), b = *reinterpret_cast<const ulonglong2*>(p + 4);
  out[0] = a.x, out[1] = a.y, out[2] = b.x, out[3] = b.y;
}

// The ReLU's mask, one bit per value of a vector: bits 0 - 3 for channels 0, 2, 4, 6 and bits 4 - 7 for 1, 3, 5, 7.  Of values that are
// not below zero, as the ReLU leaves them, each half that is above it carries into its highest bit.
__device__ __forceinline__ unsigned char mask_of(const uint32_t (&w)[4]) {
  uint32_t t = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) t |= ((w[i] + 0x7fff7fffu) & 0x80008000u) >> (3 - i);
  return static_cast<unsigned char>(((t >> 12) & 0xf) | ((t >> 24) & 0xf0));
}
__device__ __forceinline__ void apply_mask(uint32_t bits, uint32_t (&w)[4]) {
  const uint32_t spread = bits | bits << 12;
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] &= ((spread >> i) & 0x00010001u) * 0xffffu;
}

// Rows come through a ring of 16-byte vectors in shared memory, three batches ahead (cp.async; a thread reads back only what it has
// copied itself, so no barrier is needed): 48 KiB in flight per CTA without a register for them.  `TENSORS` are walked together.
constexpr int RING = 12, AHEAD = 3;
template <int TENSORS>
struct Ring {
  static constexpr int BATCH = RING / AHEAD / TENSORS;   // rows
  uint32_t base;   // of this thread, shared address
  __device__ __forceinline__ explicit Ring(const void* memory)
      : base(static_cast<uint32_t>(__cvta_generic_to_shared(memory)) + threadIdx.x * 16) {}
  __device__ __forceinline__ uint32_t at(int place, int row, int tensor) const {
    return base + ((place * BATCH + row) * TENSORS + tensor) * THREADS * 16;
  }
  template <bool LAST>
  __device__ __forceinline__ void copy(int place, int row, int tensor, const __nv_bfloat16* from, unsigned long long policy) const {
    if (LAST)
      asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(at(place, row, tensor)), "l"(from), "l"(policy) : "memory");
    else
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at(place, row, tensor)), "l"(from) : "memory");
  }
  __device__ __forceinline__ void read(int place, int row, int tensor, uint32_t (&w)[4]) const {
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(at(place, row, tensor)) : "memory");
  }
  static __device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
  static __device__ __forceinline__ void wait() { asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD - 1) : "memory"); }
};
// For data that is read for the last time, or that this direction does not read again: other lines stay in L2 instead.
__device__ __forceinline__ unsigned long long last_use() {
  unsigned long long policy;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  return policy;
}
// Results are not read again in their direction: streaming stores.
__device__ __forceinline__ void store(__nv_bfloat16* p, const uint32_t (&w)[4]) {
  asm volatile("st.global.cs.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}

// How the backward kernels find the ReLU mask: no activation, from the bits that the forward pass has left (a sixteenth of the
// bytes of y), or recomputed from x (y > 0 exactly when x * scale[c] + shift[c] > 0; only without a residual).
enum : int { MASK_NONE = 0, MASK_BITS = 1, MASK_FROM_X = 2 };
__device__ __forceinline__ void mask_from_x(const f32x2 (&x)[4], const f32x2 (&scale)[4], const f32x2 (&shift)[4], uint32_t (&g)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 y = unpack2(fma2(x[i], scale[i], shift[i]));
    g[i] = (y.x > 0.f ? g[i] & 0xffffu : 0u) | (y.y > 0.f ? g[i] & 0xffff0000u : 0u);
  }
}

// Partial sums of one split of the rows, 32 row lanes added up one after the other, for `groups` vector columns:
// forward (BWD false) sums of x and x^2, backward of g and xhat * g with g the masked dy.  part[(split * channels + c) * 2].
template <bool BWD, int MASK>
__global__ void __launch_bounds__(THREADS, MASK == MASK_FROM_X ? 3 : 4)
bn_sums(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy, const unsigned char* __restrict__ mask,
        const float* __restrict__ mean, const float* __restrict__ invstd, const float* __restrict__ weight,
        const float* __restrict__ bias, float* __restrict__ part, long long rows, int channels, int groups, long long rows_per_split) {
  chain_next();
  using R = Ring<BWD ? 2 : 1>;
  __shared__ uint4 memory[RING * THREADS];
  const R ring(memory);
  const int t = threadIdx.x, lane = t / groups;
  const int c0 = (blockIdx.x * groups + t - lane * groups) * 8;
  const long long r_begin = blockIdx.y * rows_per_split;
  // rows of this lane
  const int count = c0 < channels ? (static_cast<int>(min(rows, r_begin + rows_per_split) - r_begin) - lane + LANES - 1) / LANES : 0;
  const long long step = static_cast<long long>(LANES) * channels, first_at = (r_begin + lane) * channels + c0;
  const __nv_bfloat16 *bx = x + first_at, *bg = dy + first_at;
  int fetched = 0;
  auto fetch = [&](int place) {
#pragma unroll
    for (int u = 0; u < R::BATCH; ++u) {
      if (fetched + u < count) {
        ring.template copy<false>(place, u, 0, bx, 0);
        if (BWD) ring.template copy<false>(place, u, 1, bg, 0);
      }
      bx += step;
      bg += step;
    }
    fetched += R::BATCH;
    R::commit();
  };
#pragma unroll
  for (int place = 0; place < AHEAD; ++place) fetch(place);
  const unsigned char* bm = mask + (first_at >> 3);
  uint32_t bits[R::BATCH], next[R::BATCH];
  auto fetch_bits = [&](int from) {
#pragma unroll
    for (int u = 0; u < R::BATCH; ++u) {
      if (MASK == MASK_BITS && from + u < count) next[u] = __ldg(bm);
      bm += step >> 3;
    }
  };
  if (MASK == MASK_BITS) fetch_bits(0);
  f32x2 minus_mu[4], is[4], sc[4], sh[4], first[4], second[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) first[i] = second[i] = 0;
  if (BWD && count > 0) {
    load_pairs(mean + c0, minus_mu);
    load_pairs(invstd + c0, is);
    if (MASK == MASK_FROM_X) {   // the forward pass's scale and shift, same roundings
      load_pairs(weight + c0, sc);
      load_pairs(bias + c0, sh);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      minus_mu[i] ^= 0x8000000080000000ull;
      if (MASK == MASK_FROM_X) {
        sc[i] = mul2(sc[i], is[i]);
        sh[i] = fma2(minus_mu[i], sc[i], sh[i]);
      }
    }
  }
  for (int k = 0, place = 0; k < count; k += R::BATCH) {
    if (MASK == MASK_BITS) {
#pragma unroll
      for (int u = 0; u < R::BATCH; ++u) bits[u] = next[u];
      fetch_bits(k + R::BATCH);
    }
    R::wait();
#pragma unroll
    for (int u = 0; u < R::BATCH; ++u) {
      if (k + u < count) {
        uint32_t wx[4], wg[4];
        f32x2 xv[4], gv[4];
        ring.read(place, u, 0, wx);
        unpack(wx, xv);
        if (BWD) {
          ring.read(place, u, 1, wg);
          if (MASK == MASK_BITS) apply_mask(bits[u], wg);
          if (MASK == MASK_FROM_X) mask_from_x(xv, sc, sh, wg);
          unpack(wg, gv);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          first[i] = add2(first[i], BWD ? gv[i] : xv[i]);
          second[i] = BWD ? fma2(mul2(add2(xv[i], minus_mu[i]), is[i]), gv[i], second[i]) : fma2(xv[i], xv[i], second[i]);
        }
      }
    }
    fetch(place);
    place = place + 1 == AHEAD ? 0 : place + 1;
  }
  // lane after lane; the sums take the place of the ring
  __syncthreads();
  float4* red = reinterpret_cast<float4*>(memory);   // [pair of channels][lane][group]
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 a = unpack2(first[i]), b = unpack2(second[i]);
    red[i * THREADS + t] = make_float4(a.x, b.x, a.y, b.y);
  }
  __syncthreads();
  if (t < groups * 16) {
    const int j = t / (4 * groups), rest = t - j * 4 * groups;   // rest: group, then channel of the pair, then first or second
    const float* at = reinterpret_cast<const float*>(red + j * THREADS) + rest;
    float s = 0.f;
#pragma unroll
    for (int l = 0; l < LANES; ++l) s += at[l * 4 * groups];
    const int c = (blockIdx.x * groups + rest / 4) * 8 + 2 * j + (rest % 4) / 2;
    if (c < channels) part[(static_cast<size_t>(blockIdx.y) * channels + c) * 2 + (rest & 1)] = s;
  }
}

// coef layout (fp32, [5, c]): scale, shift (forward); k_dy, k_x, k_const (backward)
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Both sums of a channel over the splits, one warp, in double precision.
__device__ __forceinline__ void sums_of_channel(const float* part, int c, int lane, int channels, int splits, double& first, double& second) {
  first = second = 0.0;
#pragma unroll 8
  for (int k = lane; k < splits; k += 32) {
    const float2 v = *reinterpret_cast<const float2*>(part + (static_cast<size_t>(k) * channels + c) * 2);
    first += v.x;
    second += v.y;
  }
  first = warp_sum(first);
  second = warp_sum(second);
}

// One warp per channel.
__global__ void __launch_bounds__(256)
bn_fwd_finalize(const float* part, const float* __restrict__ weight,
                const float* __restrict__ bias, float* __restrict__ running_mean,
                float* __restrict__ running_var, float* __restrict__ mean_out,
                float* __restrict__ invstd_out, float* __restrict__ coef, long long* __restrict__ tracked,
                int channels, int splits, long long rows, float momentum, float eps) {
  chain_next();
  chain_wait();
  const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (c >= channels) return;  // whole warp
  double s, q;
  sums_of_channel(part, c, lane, channels, splits, s, q);
  if (lane != 0) return;
  if (c == 0 && tracked != nullptr) *tracked += 1;
  const double mean = s / static_cast<double>(rows);
  double var = q / static_cast<double>(rows) - mean * mean;
  var = var > 0.0 ? var : 0.0;
  const float invstd = static_cast<float>(1.0 / sqrt(var + static_cast<double>(eps)));
  mean_out[c] = static_cast<float>(mean);
  invstd_out[c] = invstd;
  // explicit roundings: the backward pass recomputes scale and shift bit for bit (ReLU mask from x)
  const float scale = __fmul_rn(weight[c], invstd);
  coef[c] = scale;
  coef[channels + c] = __fmaf_rn(-static_cast<float>(mean), scale, bias[c]);
  if (running_mean != nullptr) {
    const double unbiased = rows > 1 ? var * static_cast<double>(rows) / static_cast<double>(rows - 1) : var;
    running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * static_cast<float>(mean);
    running_var[c] = (1.f - momentum) * running_var[c] + momentum * static_cast<float>(unbiased);
  }
}

// y = act(x * scale[c] + shift[c] (+ residual)) and, with MASK, the ReLU's mask.  A thread keeps its eight channels (row_walk.h), so
// scale and shift stay in registers.  The bytes bound it: 32 x 256 x 56 x 56 with a residual and the mask (157 MB, 108 from and to memory
// while it runs) 22.8 us.
template <bool RES, bool RELU, bool MASK>
__global__ void __launch_bounds__(THREADS, 4)
bn_apply(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ res,
         const float* scale, const float* shift, __nv_bfloat16* __restrict__ y, unsigned char* __restrict__ mask,
         long long rows, int channels, int groups, int lanes) {
  using R = Ring<RES ? 2 : 1>;
  __shared__ uint4 memory[RING * THREADS];
  const R ring(memory);
  const int lane = threadIdx.x / groups;
  const int c0 = ((blockIdx.z * gridDim.y + blockIdx.y) * groups + threadIdx.x % groups) * 8;
  if (lane >= lanes || c0 >= channels) return;
  const long long first = static_cast<long long>(blockIdx.x) * lanes + lane, back = -static_cast<long long>(gridDim.x) * lanes * channels;
  long long at = (rows - 1 - first) * channels + c0, ahead = at;   // from the end, where bn_sums has stopped
  const unsigned long long policy = last_use();
  auto fetch = [&](auto place) {
#pragma unroll
    for (int u = 0; u < R::BATCH; ++u) {
      if (ahead >= 0) {
        ring.template copy<true>(place, u, 0, x + ahead, policy);
        if (RES) ring.template copy<true>(place, u, 1, res + ahead, policy);
      }
      ahead += back;
    }
    R::commit();
  };
  fetch(std::integral_constant<int, 0>());
  fetch(std::integral_constant<int, 1>());
  fetch(std::integral_constant<int, 2>());   // x and res are older than the chain, whose first kernel, bn_sums, is launched plainly
  chain_wait();
  f32x2 a[4], b[4];
  load_pairs(scale + c0, a);
  load_pairs(shift + c0, b);
  auto use = [&](auto place) {
    R::wait();
#pragma unroll
    for (int u = 0; u < R::BATCH; ++u) {
      if (at >= 0) {
        uint32_t w[4], wr[4];
        f32x2 v[4], r[4];
        ring.read(place, u, 0, w);
        unpack(w, v);
        if (RES) {
          ring.read(place, u, 1, wr);
          unpack(wr, r);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          v[i] = fma2(v[i], a[i], b[i]);
          if (RES) v[i] = add2(v[i], r[i]);
          w[i] = pack(v[i]);
          if (RELU) w[i] = relu2(w[i]);
        }
        store(y + at, w);
        if (MASK) mask[at >> 3] = mask_of(w);
      }
      at += back;
    }
    fetch(place);
  };
  while (at >= 0) {
    use(std::integral_constant<int, 0>());
    use(std::integral_constant<int, 1>());
    use(std::integral_constant<int, 2>());
  }
}

// g = masked dy;   dx = g * k_dy[c] + x * k_x[c] + k_const[c];   dres = g (optional).  Rows are walked as in bn_apply (the same size
// with a mask and dres, 209 MB, 102 from and to memory: 35.4 -> 27.5 us).
template <int MASK, bool DRES>
__global__ void __launch_bounds__(THREADS, MASK == MASK_FROM_X ? 3 : 4)
bn_dx(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
      const unsigned char* mask, const float* scale, const float* shift, const float* k_dy, const float* k_x, const float* k_const,
      __nv_bfloat16* __restrict__ dx, __nv_bfloat16* __restrict__ dres, long long rows, int channels, int groups, int lanes) {
  using R = Ring<2>;
  __shared__ uint4 memory[RING * THREADS];
  const R ring(memory);
  const int lane = threadIdx.x / groups;
  const int c0 = ((blockIdx.z * gridDim.y + blockIdx.y) * groups + threadIdx.x % groups) * 8;
  if (lane >= lanes || c0 >= channels) return;
  const long long first = static_cast<long long>(blockIdx.x) * lanes + lane, back = -static_cast<long long>(gridDim.x) * lanes * channels;
  long long at = (rows - 1 - first) * channels + c0, ahead = at;   // from the end, where bn_sums has stopped
  const unsigned long long policy = last_use();
  auto fetch = [&](auto place) {
#pragma unroll
    for (int u = 0; u < R::BATCH; ++u) {
      if (ahead >= 0) {
        ring.template copy<true>(place, u, 0, x + ahead, policy);
        ring.template copy<true>(place, u, 1, dy + ahead, policy);
      }
      ahead += back;
    }
    R::commit();
  };
  fetch(std::integral_constant<int, 0>());
  fetch(std::integral_constant<int, 1>());
  fetch(std::integral_constant<int, 2>());
  uint32_t next[R::BATCH];
  auto fetch_bits = [&](long long from) {
#pragma unroll
    for (int u = 0; u < R::BATCH; ++u)
      if (MASK == MASK_BITS && from + u * back >= 0) next[u] = mask[(from + u * back) >> 3];
  };
  if (MASK == MASK_BITS) fetch_bits(at);   // x, dy and mask are older than the chain
  chain_wait();
  f32x2 a[4], b[4], c[4], sc[4], sh[4];
  load_pairs(k_dy + c0, a);
  load_pairs(k_x + c0, b);
  load_pairs(k_const + c0, c);
  if (MASK == MASK_FROM_X) {
    load_pairs(scale + c0, sc);
    load_pairs(shift + c0, sh);
  }
  auto use = [&](auto place) {
    uint32_t bits[R::BATCH];
    if (MASK == MASK_BITS) {
#pragma unroll
      for (int u = 0; u < R::BATCH; ++u) bits[u] = next[u];
      fetch_bits(at + R::BATCH * back);
    }
    R::wait();
#pragma unroll
    for (int u = 0; u < R::BATCH; ++u) {
      if (at >= 0) {
        uint32_t wx[4], wg[4];
        f32x2 xv[4], g[4];
        ring.read(place, u, 0, wx);
        ring.read(place, u, 1, wg);
        unpack(wx, xv);
        if (MASK == MASK_BITS) apply_mask(bits[u], wg);
        if (MASK == MASK_FROM_X) mask_from_x(xv, sc, sh, wg);
        unpack(wg, g);
#pragma unroll
        for (int i = 0; i < 4; ++i) wx[i] = pack(fma2(g[i], a[i], fma2(xv[i], b[i], c[i])));
        store(dx + at, wx);
        if (DRES) store(dres + at, wg);
      }
      at += back;
    }
    fetch(place);
  };
  while (at >= 0) {
    use(std::integral_constant<int, 0>());
    use(std::integral_constant<int, 1>());
    use(std::integral_constant<int, 2>());
  }
}

// dx = w*invstd * (dy - mean(dy) - xhat * mean(dy*xhat))
//    = dy * k_dy + x * k_x + k_const  with
//   k_dy = w*invstd, k_x = -k_dy * invstd * m2, k_const = -k_dy * (m1 - mean * invstd * m2)
__global__ void __launch_bounds__(256)
bn_bwd_finalize(const float* part, const float* __restrict__ weight, const float* __restrict__ bias,
                const float* __restrict__ mean, const float* __restrict__ invstd,
                float* __restrict__ dweight, float* __restrict__ dbias,
                float* __restrict__ coef, int channels, int splits, long long rows) {
  chain_next();
  chain_wait();
  const int c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (c >= channels) return;  // whole warp
  double s1, s2;
  sums_of_channel(part, c, lane, channels, splits, s1, s2);
  if (lane != 0) return;
  dbias[c] = static_cast<float>(s1);
  dweight[c] = static_cast<float>(s2);
  const double m1 = s1 / static_cast<double>(rows), m2 = s2 / static_cast<double>(rows);
  const double k_dy = static_cast<double>(weight[c]) * invstd[c];
  coef[2 * channels + c] = static_cast<float>(k_dy);
  coef[3 * channels + c] = static_cast<float>(-k_dy * invstd[c] * m2);
  coef[4 * channels + c] = static_cast<float>(-k_dy * (m1 - static_cast<double>(mean[c]) * invstd[c] * m2));
  if (bias != nullptr) {   // the forward pass's scale and shift (rows 0 and 1) for a ReLU mask recomputed from x
    const float scale = __fmul_rn(weight[c], invstd[c]);
    coef[c] = scale;
    coef[channels + c] = __fmaf_rn(-mean[c], scale, bias[c]);
  }
}

struct Shape {
  long long rows;
  int channels;
  int chunks, groups;   // CTAs across the channels, vectors of 8 channels in each
  int splits;
  long long rows_per_split;
};

Shape plan(const at::Tensor& x) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 4 && x.scalar_type() == at::kBFloat16 &&
                  x.is_contiguous(at::MemoryFormat::ChannelsLast),
              "expected a 4-d channels_last bf16 CUDA tensor");
  Shape s;
  s.channels = static_cast<int>(x.size(1));
  s.rows = x.size(0) * x.size(2) * x.size(3);
  TORCH_CHECK(s.channels % 8 == 0 && s.rows > 0, "the channel count must be a multiple of 8");
  TORCH_CHECK((reinterpret_cast<uintptr_t>(x.data_ptr()) & 15) == 0, "16-byte alignment required");
  s.chunks = (s.channels + GROUPS * 8 - 1) / (GROUPS * 8);
  s.groups = (s.channels / 8 + s.chunks - 1) / s.chunks;
  long long want = (148 * 8 + s.chunks - 1) / s.chunks;                   // ~8 CTAs per SM in total
  long long most = (s.rows + MIN_ROWS - 1) / MIN_ROWS;
  long long splits = std::max<long long>(1, std::min(want, most));
  s.rows_per_split = (s.rows + splits - 1) / splits;
  s.splits = static_cast<int>((s.rows + s.rows_per_split - 1) / s.rows_per_split);
  return s;
}

void check_vec(const at::Tensor& t, int c, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous() && t.numel() == c, name,
              " must be a contiguous fp32 CUDA vector with one entry per channel");
}

void check_like(const at::Tensor& t, const at::Tensor& x, const char* name) {
  TORCH_CHECK(t.sizes() == x.sizes() && t.scalar_type() == at::kBFloat16 && t.is_cuda() &&
                  t.is_contiguous(at::MemoryFormat::ChannelsLast) &&
                  (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0,
              name, " must match x (channels_last bf16, 16-byte aligned)");
}

}  // namespace

// y = act(batch_norm(x) (+ residual)).  Returns (y, mean, invstd) and, with `want_mask`, the ReLU's mask (one byte per eight channels
// of a position).  running_mean / running_var and the batch counter are updated in place when given.
std::vector<at::Tensor> bn_forward_train(at::Tensor x, at::Tensor weight, at::Tensor bias,
                                         c10::optional<at::Tensor> running_mean,
                                         c10::optional<at::Tensor> running_var,
                                         c10::optional<at::Tensor> num_batches_tracked, double momentum,
                                         double eps, c10::optional<at::Tensor> residual, bool relu, bool want_mask) {
  TORCH_CHECK(relu || !want_mask, "a mask needs a ReLU");
  const Shape s = plan(x);
  check_vec(weight, s.channels, "weight");
  check_vec(bias, s.channels, "bias");
  float *rm = nullptr, *rv = nullptr;
  if (running_mean.has_value() && running_var.has_value()) {
    check_vec(*running_mean, s.channels, "running_mean");
    check_vec(*running_var, s.channels, "running_var");
    rm = running_mean->data_ptr<float>();
    rv = running_var->data_ptr<float>();
  }
  long long* tracked = nullptr;
  if (num_batches_tracked.has_value()) {
    TORCH_CHECK(num_batches_tracked->is_cuda() && num_batches_tracked->scalar_type() == at::kLong &&
                    num_batches_tracked->numel() == 1, "num_batches_tracked must be a CUDA int64 scalar");
    tracked = reinterpret_cast<long long*>(num_batches_tracked->data_ptr<int64_t>());
  }
  const __nv_bfloat16* rp = nullptr;
  if (residual.has_value()) {
    check_like(*residual, x, "residual");
    rp = reinterpret_cast<const __nv_bfloat16*>(residual->data_ptr());
  }
  const int dev = x.get_device();
  c10::cuda::CUDAGuard guard(dev);
  auto stream = at::cuda::getCurrentCUDAStream(dev).stream();
  auto f32 = weight.options();
  auto mean = at::empty({s.channels}, f32), invstd = at::empty({s.channels}, f32);
  auto y = at::empty_like(x);
  at::Tensor mask;
  if (want_mask) mask = at::empty({s.rows, s.channels / 8}, x.options().dtype(at::kByte));
  const auto* xp = reinterpret_cast<const __nv_bfloat16*>(x.data_ptr());
  auto* yp = reinterpret_cast<__nv_bfloat16*>(y.data_ptr());
  unsigned char* maskp = want_mask ? mask.data_ptr<unsigned char>() : nullptr;
  const float mom = static_cast<float>(momentum), ep = static_cast<float>(eps);
  auto part = at::empty({s.splits, s.channels, 2}, f32);
  auto coef = at::empty({2, s.channels}, f32);
  float* partp = part.data_ptr<float>();
  // plainly: bn_apply reads x and the residual ahead of its wait
  bn_sums<false, MASK_NONE><<<dim3(s.chunks, s.splits), LANES * s.groups, 0, stream>>>(
      xp, xp, nullptr, nullptr, nullptr, nullptr, nullptr, partp, s.rows, s.channels, s.groups, s.rows_per_split);
  launch_chained(bn_fwd_finalize, dim3((s.channels + 7) / 8), dim3(256), 0, stream, partp, weight.data_ptr<float>(),
                 bias.data_ptr<float>(), rm, rv, mean.data_ptr<float>(), invstd.data_ptr<float>(), coef.data_ptr<float>(), tracked,
                 s.channels, s.splits, s.rows, mom, ep);
  const Walk w = walk_plan(s.channels / 8);
  const dim3 grid = walk_grid_layers(w, s.rows, 4);
  const float* scale = coef.data_ptr<float>();
  auto run = [&](auto kernel) {
    launch_chained(kernel, grid, dim3(256), 0, stream, xp, rp, scale, scale + s.channels, yp, maskp, s.rows, s.channels, w.groups, w.lanes);
  };
  if (want_mask)
    rp != nullptr ? run(bn_apply<true, true, true>) : run(bn_apply<false, true, true>);
  else if (relu)
    rp != nullptr ? run(bn_apply<true, true, false>) : run(bn_apply<false, true, false>);
  else
    rp != nullptr ? run(bn_apply<true, false, false>) : run(bn_apply<false, false, false>);
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch(3);
  if (want_mask) return {y, mean, invstd, mask};
  return {y, mean, invstd};
}

// Backward of y = act(batch_norm(x) (+ residual)).  The ReLU mask is the forward pass's `mask`, or - when `bias_for_mask` is given
// instead (ReLU without a residual) - is recomputed from x.
// Returns (dx, dweight, dbias) and, with `want_dres`, the gradient of the residual (dy masked by
// the activation; without an activation it is dy itself and is not returned).
std::vector<at::Tensor> bn_backward_train(at::Tensor x, at::Tensor dy, at::Tensor weight, at::Tensor mean,
                                          at::Tensor invstd, c10::optional<at::Tensor> mask, bool want_dres,
                                          c10::optional<at::Tensor> bias_for_mask) {
  const Shape s = plan(x);
  check_like(dy, x, "dy");
  check_vec(weight, s.channels, "weight");
  check_vec(mean, s.channels, "mean");
  check_vec(invstd, s.channels, "invstd");
  const bool from_x = bias_for_mask.has_value();
  TORCH_CHECK(!(from_x && (mask.has_value() || want_dres)), "the mask is recomputed from x only without a residual");
  const bool relu = mask.has_value() || from_x;
  const unsigned char* maskp = nullptr;
  if (mask.has_value()) {
    TORCH_CHECK(mask->is_cuda() && mask->get_device() == x.get_device() && mask->scalar_type() == at::kByte && mask->is_contiguous() &&
                    mask->numel() == s.rows * (s.channels / 8), "the mask must be the one that the forward pass has returned");
    maskp = mask->data_ptr<unsigned char>();
  }
  const float* bp = nullptr;
  if (from_x) {
    check_vec(*bias_for_mask, s.channels, "bias");
    bp = bias_for_mask->data_ptr<float>();
  }
  const bool dres_out = want_dres && relu;
  const int dev = x.get_device();
  c10::cuda::CUDAGuard guard(dev);
  auto stream = at::cuda::getCurrentCUDAStream(dev).stream();
  auto f32 = weight.options();
  auto dweight = at::empty({s.channels}, f32), dbias = at::empty({s.channels}, f32);
  auto dx = at::empty_like(x);
  at::Tensor dres;
  if (dres_out) dres = at::empty_like(x);
  const auto* xp = reinterpret_cast<const __nv_bfloat16*>(x.data_ptr());
  const auto* gp = reinterpret_cast<const __nv_bfloat16*>(dy.data_ptr());
  auto* dxp = reinterpret_cast<__nv_bfloat16*>(dx.data_ptr());
  auto* drp = dres_out ? reinterpret_cast<__nv_bfloat16*>(dres.data_ptr()) : nullptr;
  const float *wp = weight.data_ptr<float>(), *mp = mean.data_ptr<float>(), *ip = invstd.data_ptr<float>();
  auto part = at::empty({s.splits, s.channels, 2}, f32);
  auto coef = at::empty({5, s.channels}, f32);
  float* partp = part.data_ptr<float>();
  auto sums = [&](auto kernel) {   // plainly: bn_dx reads x, dy and the mask ahead of its wait
    kernel<<<dim3(s.chunks, s.splits), LANES * s.groups, 0, stream>>>(xp, gp, maskp, mp, ip, wp, bp, partp, s.rows, s.channels, s.groups,
                                                                   s.rows_per_split);
  };
  if (from_x)
    sums(bn_sums<true, MASK_FROM_X>);
  else if (relu)
    sums(bn_sums<true, MASK_BITS>);
  else
    sums(bn_sums<true, MASK_NONE>);
  launch_chained(bn_bwd_finalize, dim3((s.channels + 7) / 8), dim3(256), 0, stream, partp, wp, bp, mp, ip,
                 dweight.data_ptr<float>(), dbias.data_ptr<float>(), coef.data_ptr<float>(), s.channels, s.splits, s.rows);
  const Walk w = walk_plan(s.channels / 8);
  const dim3 grid = walk_grid_layers(w, s.rows, from_x ? 3 : 4);
  const float* k = coef.data_ptr<float>();
  const long long c = s.channels;
  auto run = [&](auto kernel) {
    launch_chained(kernel, grid, dim3(256), 0, stream, gp, xp, maskp, k, k + c, k + 2 * c, k + 3 * c, k + 4 * c, dxp, drp, s.rows,
                   s.channels, w.groups, w.lanes);
  };
  if (from_x)
    run(bn_dx<MASK_FROM_X, false>);
  else if (relu && dres_out)
    run(bn_dx<MASK_BITS, true>);
  else if (relu)
    run(bn_dx<MASK_BITS, false>);
  else
    run(bn_dx<MASK_NONE, false>);
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch(3);
  if (dres_out) return {dx, dweight, dbias, dres};
  return {dx, dweight, dbias};
}

}  // namespace b200
