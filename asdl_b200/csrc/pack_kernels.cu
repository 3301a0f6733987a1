// Bandwidth-bound staging kernels that feed the tcgen05 GEMMs:
//   * cast_pad_bf16  : [rows, n] fp32/bf16 -> bf16 with a TMA-legal row pitch, optional residual
//                      ("lo") so that hi+lo carries ~16 mantissa bits.
//   * im2col_bf16    : conv input (any strides: NCHW or channels_last) -> patch matrix
//                      [N*Ho*Wo, ld] bf16, columns ordered (kh, kw, c) or (c, kh, kw).
#include "chained_launch.h"
#include "host_utils.h"
#include "row_walk.h"
#include <cuda_bf16.h>

#include <type_traits>

#include <cmath>

namespace b200 {

template <typename T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float to_f32<__half>(__half v) { return __half2float(v); }

// [rows, n] -> PARTS bf16 matrices of pitch ldo (a multiple of eight) whose sum carries the value: hi, hi + lo, or
// hi + mid + lo.  Columns past n are zeros.  One thread writes eight columns (16 bytes per part) of a row and walks down
// the rows (row_walk.h) with the loads of CAST_ROWS rows in flight; VEC: the source rows are 16-byte aligned.
// The kernel does nothing but move bytes; one element per thread with a 64-bit division each ran at 2.6 TB/s
// (12608 x 768 fp32 -> hi, lo: 29.4 us).
constexpr int CAST_ROWS = 2;
template <typename T, int PARTS, bool VEC>
__device__ __forceinline__ void cast_rows(const T* __restrict__ src, long long lds, float scale, __nv_bfloat16* __restrict__ p0,
                                          __nv_bfloat16* __restrict__ p1, __nv_bfloat16* __restrict__ p2, long long ldo,
                                          long long rows, int n, long long c0, long long first, long long step) {
  for (long long r = first; r < rows; r += CAST_ROWS * step) {
    float v[CAST_ROWS][8];
#pragma unroll
    for (int u = 0; u < CAST_ROWS; ++u) {
      const T* from = src + (r + u * step) * lds + c0;
      const bool row_in = r + u * step < rows;
      if (VEC && row_in && c0 + 8 <= n) {
        uint4 raw[sizeof(T) / 2];
#pragma unroll
        for (int h = 0; h < static_cast<int>(sizeof(T) / 2); ++h) raw[h] = __ldg(reinterpret_cast<const uint4*>(from) + h);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[u][k] = to_f32<T>(reinterpret_cast<const T*>(raw)[k]);
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[u][k] = (row_in && c0 + k < n) ? to_f32<T>(from[k]) : 0.f;
      }
    }
#pragma unroll
    for (int u = 0; u < CAST_ROWS; ++u) {
      if (r + u * step >= rows) break;
      uint32_t w[PARTS][4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float a = v[u][2 * k] * scale, b = v[u][2 * k + 1] * scale;
#pragma unroll
        for (int part = 0; part < PARTS; ++part) {
          const __nv_bfloat16 ha = __float2bfloat16_rn(a), hb = __float2bfloat16_rn(b);
          w[part][k] = static_cast<uint32_t>(__bfloat16_as_ushort(ha)) | (static_cast<uint32_t>(__bfloat16_as_ushort(hb)) << 16);
          a -= __bfloat162float(ha);
          b -= __bfloat162float(hb);
        }
      }
      const long long at = (r + u * step) * ldo + c0;
      *reinterpret_cast<uint4*>(p0 + at) = make_uint4(w[0][0], w[0][1], w[0][2], w[0][3]);
      if (PARTS > 1) *reinterpret_cast<uint4*>(p1 + at) = make_uint4(w[PARTS > 1][0], w[PARTS > 1][1], w[PARTS > 1][2], w[PARTS > 1][3]);
      if (PARTS > 2)
        *reinterpret_cast<uint4*>(p2 + at) =
            make_uint4(w[PARTS - 1][0], w[PARTS - 1][1], w[PARTS - 1][2], w[PARTS - 1][3]);
    }
  }
}
template <typename T, int PARTS, bool VEC>
__global__ void __launch_bounds__(256)
cast_parts_kernel(const T* __restrict__ src, long long lds, float scale, __nv_bfloat16* __restrict__ p0,
                  __nv_bfloat16* __restrict__ p1, __nv_bfloat16* __restrict__ p2, long long ldo, long long rows, int n,
                  int groups, int lanes) {
  chain_next();
  const int lane = threadIdx.x / groups;
  const long long c0 = (static_cast<long long>(blockIdx.y) * groups + threadIdx.x % groups) * 8;
  if (lane >= lanes || c0 >= ldo) return;
  cast_rows<T, PARTS, VEC>(src, lds, scale, p0, p1, p2, ldo, rows, n, c0, static_cast<long long>(blockIdx.x) * lanes + lane,
                           static_cast<long long>(gridDim.x) * lanes);
}

// Several fp32 matrices -> hi, lo in one launch: one wave of blocks, shared out by size.  The operands of a two-sided product:
// 1024 x 4096 with its factors (168 MB) 151.0 -> 146.4 us pass after pass, 768 x 768 in graphs 33.4 -> 31.2 us, 1000 x 333
// 37.4 -> 29.8, 10 x 32 14.9 -> 11.8; each launch is 2 us of the host's time besides (10 x 32: 33 -> 26 us).
struct CastJob {
  const float* src;
  __nv_bfloat16 *hi, *lo;
  long long lds, ldo, rows;
  int n, groups, lanes, across, first;   // blocks beside each other, first block
  bool vec;
};
template <int JOBS>
struct CastJobs {
  CastJob job[JOBS];
  int count, blocks;
  float scale;
};
template <int JOBS>
__global__ void __launch_bounds__(256) cast_jobs_kernel(const __grid_constant__ CastJobs<JOBS> t) {
  chain_next();
  int k = 0, past = t.count;   // the last job whose first block is not past this one
  while (past - k > 1) {
    const int mid = (k + past) / 2;
    (t.job[mid].first <= static_cast<int>(blockIdx.x) ? k : past) = mid;
  }
  const CastJob& j = t.job[k];
  const int end = k + 1 < t.count ? t.job[k + 1].first : t.blocks, block = blockIdx.x - j.first, down = (end - j.first) / j.across;
  const int lane = threadIdx.x / j.groups;
  const long long c0 = (static_cast<long long>(block % j.across) * j.groups + threadIdx.x % j.groups) * 8;
  if (lane >= j.lanes || c0 >= j.ldo) return;
  const long long first = static_cast<long long>(block / j.across) * j.lanes + lane, step = static_cast<long long>(down) * j.lanes;
  if (j.vec)
    cast_rows<float, 2, true>(j.src, j.lds, t.scale, j.hi, j.lo, nullptr, j.ldo, j.rows, j.n, c0, first, step);
  else
    cast_rows<float, 2, false>(j.src, j.lds, t.scale, j.hi, j.lo, nullptr, j.ldo, j.rows, j.n, c0, first, step);
}

static CastJob cast_job(const float* src, long long lds, int64_t rows, int64_t n, const at::Tensor& hi, const at::Tensor& lo) {
  TORCH_CHECK(hi.is_contiguous() && lo.is_contiguous() && hi.scalar_type() == at::kBFloat16 && lo.scalar_type() == at::kBFloat16 &&
                  hi.dim() == 2 && hi.size(1) % 8 == 0 && hi.size(1) < (1LL << 31) && hi.sizes() == lo.sizes() &&
                  hi.size(0) == rows && hi.size(1) >= n, "parts must match their matrix");
  CastJob j;
  j.src = src;
  j.hi = reinterpret_cast<__nv_bfloat16*>(hi.data_ptr());
  j.lo = reinterpret_cast<__nv_bfloat16*>(lo.data_ptr());
  TORCH_CHECK(((reinterpret_cast<uintptr_t>(j.hi) | reinterpret_cast<uintptr_t>(j.lo)) & 15) == 0, "parts must be 16-byte aligned");
  j.lds = lds, j.ldo = hi.size(1), j.rows = rows, j.n = static_cast<int>(n);
  j.vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0 && lds % 4 == 0;
  return j;
}
template <int JOBS>
static void launch_cast_jobs(CastJobs<JOBS>& t, double scale, cudaStream_t stream) {
  if (t.count == 0) return;
  double elements = 0;
  for (int i = 0; i < t.count; ++i) elements += static_cast<double>(t.job[i].rows) * t.job[i].ldo;
  t.blocks = 0, t.scale = static_cast<float>(scale);
  for (int i = 0; i < t.count; ++i) {
    CastJob& j = t.job[i];
    const Walk w = walk_plan(static_cast<int>(j.ldo / 8));
    j.groups = w.groups, j.lanes = w.lanes, j.across = w.chunks, j.first = t.blocks;
    const long long most = (j.rows + w.lanes - 1) / w.lanes;
    const long long share = static_cast<long long>(148 * 6 * (j.rows * j.ldo / elements) / w.chunks + 0.999);
    t.blocks += static_cast<int>(std::max(1LL, std::min(most, share))) * w.chunks;
  }
  cast_jobs_kernel<JOBS><<<t.blocks, 256, 0, stream>>>(t);
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
}

// src[i] -> hi[i], lo[i]: fp32 matrices with unit column stride, contiguous bf16 ones of a pitch that is a multiple of eight.
void cast_jobs(const std::vector<at::Tensor>& src, const std::vector<at::Tensor>& hi, const std::vector<at::Tensor>& lo) {
  TORCH_CHECK(src.size() == 3 && hi.size() == 3 && lo.size() == 3, "three matrices");
  CastJobs<3> t;
  t.count = 0;
  for (int i = 0; i < 3; ++i) {
    TORCH_CHECK(src[i].scalar_type() == at::kFloat && unit_columns(src[i]), "fp32 with unit column stride");
    if (hi[i].numel() > 0) t.job[t.count++] = cast_job(src[i].data_ptr<float>(), src[i].stride(0), src[i].size(0), src[i].size(1), hi[i], lo[i]);
  }
  launch_cast_jobs(t, 1.0, at::cuda::getCurrentCUDAStream(src[0].get_device()).stream());
}

// scale * grads[i] -> hi[i], lo[i].  staged[i] is the dense fp32 view, of the gradient's shape, whose memory is the matrix [rows, n]
// of the factor's order: a gradient of the same strides is read where it lies, another one is copied there first.  Up to 64
// gradients share a launch, whose table travels as an argument: they lie elsewhere in each step. Bound by memory: ResNet-50's
// 54 matrices (102 MB, 204 with the parts), two sets of them in turn in a graph, 97.0 us copied and split -> 38.2; the 18 of a
// bottleneck ResNet of four blocks (80 MB with the parts) 41.1 -> 16.7, and ten K-FAC steps of that one 24.13 -> 23.94 ms.
void stage_gradients(std::vector<at::Tensor> grads, std::vector<at::Tensor> staged, std::vector<at::Tensor> hi,
                     std::vector<at::Tensor> lo, double scale) {
  constexpr int JOBS = 64;
  TORCH_CHECK(grads.size() == staged.size() && grads.size() == hi.size() && grads.size() == lo.size(), "one of each per gradient");
  if (grads.empty()) return;
  const auto device = staged[0].device();
  TORCH_CHECK(device.is_cuda(), "CUDA gradients");
  c10::cuda::CUDAGuard guard(device);
  const cudaStream_t stream = at::cuda::getCurrentCUDAStream(device.index()).stream();
  CastJobs<JOBS> t;
  t.count = 0;
  for (size_t i = 0; i < grads.size(); ++i) {
    const at::Tensor &g = grads[i], &v = staged[i];
    TORCH_CHECK(v.scalar_type() == at::kFloat && v.is_non_overlapping_and_dense() && v.device() == device && hi[i].device() == device &&
                    lo[i].device() == device && v.dim() > 0, "dense fp32 matrices on one device");
    bool in_place = values_in_memory(g) && g.device() == device && g.scalar_type() == at::kFloat && g.sizes() == v.sizes();
    for (int64_t d = 0; in_place && d < v.dim(); ++d) in_place = v.size(d) == 1 || g.stride(d) == v.stride(d);
    if (!in_place) v.copy_(g);
    if (v.numel() == 0) continue;
    const int64_t rows = v.size(0), n = v.numel() / rows;
    TORCH_CHECK(rows == 1 || v.stride(0) == n, "rows of the matrix in the order of the first dimension");
    t.job[t.count++] = cast_job(in_place ? g.data_ptr<float>() : v.data_ptr<float>(), n, rows, n, hi[i], lo[i]);
    if (t.count == JOBS) {
      launch_cast_jobs(t, scale, stream);
      t.count = 0;
    }
  }
  launch_cast_jobs(t, scale, stream);
}

// The same for what the vector kernel does not take (launch_cast): one element per thread.
template <typename T, int PARTS>
__global__ void cast_parts_scalar_kernel(const T* __restrict__ src, long long lds, float scale,
                                         __nv_bfloat16* __restrict__ p0, __nv_bfloat16* __restrict__ p1,
                                         __nv_bfloat16* __restrict__ p2, long long ldo, long long rows, int n) {
  const long long total = rows * ldo;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / ldo;
    const int c = static_cast<int>(i - r * ldo);
    float v = (c < n) ? to_f32<T>(src[r * lds + c]) * scale : 0.f;
    __nv_bfloat16* const parts[3] = {p0, p1, p2};
#pragma unroll
    for (int part = 0; part < PARTS; ++part) {
      const __nv_bfloat16 h = __float2bfloat16_rn(v);
      parts[part][i] = h;
      v -= __bfloat162float(h);
    }
  }
}

template <typename T, int PARTS>
void launch_cast(const T* src, long long lds, float scale, __nv_bfloat16* p0, __nv_bfloat16* p1, __nv_bfloat16* p2,
                 long long ldo, long long rows, int n, cudaStream_t stream) {
  const uintptr_t outs = reinterpret_cast<uintptr_t>(p0) | (PARTS > 1 ? reinterpret_cast<uintptr_t>(p1) : 0) |
                         (PARTS > 2 ? reinterpret_cast<uintptr_t>(p2) : 0);
  // The vector kernel scales the zeros of the padding as well, which an infinite, NaN or negative scale does not leave +0.
  // (With the product next to the load the common casts took 5 to 15 % longer.)
  const bool zeros_stay = ldo == n || (std::isfinite(scale) && scale >= 0.f);
  // rows of more than 134 million columns have more CTAs across than a grid takes on y
  const bool vec_out = (ldo & 7) == 0 && (outs & 15) == 0 && zeros_stay;
  const Walk w = vec_out ? walk_plan(static_cast<int>(ldo / 8)) : Walk{};
  if (!vec_out || w.chunks > MAX_WALK_CHUNKS) {
    const int blocks = static_cast<int>(std::min<long long>((rows * ldo + 255) / 256, 148 * 16));
    cast_parts_scalar_kernel<T, PARTS><<<blocks, 256, 0, stream>>>(src, lds, scale, p0, p1, p2, ldo, rows, n);
  } else {
    const dim3 grid = walk_grid(w, rows, 6);
    const bool vec = (reinterpret_cast<uintptr_t>(src) & 15) == 0 && (lds * sizeof(T)) % 16 == 0;
    if (vec)
      cast_parts_kernel<T, PARTS, true><<<grid, 256, 0, stream>>>(src, lds, scale, p0, p1, p2, ldo, rows, n, w.groups, w.lanes);
    else
      cast_parts_kernel<T, PARTS, false><<<grid, 256, 0, stream>>>(src, lds, scale, p0, p1, p2, ldo, rows, n, w.groups, w.lanes);
  }
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
}

void cast_pad_bf16(at::Tensor src, at::Tensor hi, c10::optional<at::Tensor> lo, double scale) {
  TORCH_CHECK(src.is_cuda() && src.dim() == 2 && unit_columns(src), "src must be 2-D, unit col stride");
  TORCH_CHECK(hi.is_cuda() && hi.scalar_type() == at::kBFloat16 && hi.dim() == 2 &&
                  hi.is_contiguous() && hi.size(0) == src.size(0) && hi.size(1) >= src.size(1),
              "hi must be contiguous bf16 [rows, >= n]");
  __nv_bfloat16* lo_p = nullptr;
  if (lo.has_value()) {
    TORCH_CHECK(lo->sizes() == hi.sizes() && lo->is_contiguous() &&
                    lo->scalar_type() == at::kBFloat16, "lo must match hi");
    lo_p = reinterpret_cast<__nv_bfloat16*>(lo->data_ptr());
  }
  c10::cuda::CUDAGuard guard(src.get_device());
  const long long rows = src.size(0);
  const int n = static_cast<int>(src.size(1));
  const long long ldo = hi.size(1);
  const long long total = rows * ldo;
  if (total == 0) return;
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  auto* hi_p = reinterpret_cast<__nv_bfloat16*>(hi.data_ptr());
  const float s = static_cast<float>(scale);
  auto run = [&](auto* from) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(from)>>;
    if (lo_p != nullptr)
      launch_cast<T, 2>(from, src.stride(0), s, hi_p, lo_p, nullptr, ldo, rows, n, stream);
    else
      launch_cast<T, 1>(from, src.stride(0), s, hi_p, nullptr, nullptr, ldo, rows, n, stream);
  };
  if (src.scalar_type() == at::kFloat)
    run(static_cast<const float*>(src.data_ptr<float>()));
  else if (src.scalar_type() == at::kBFloat16)
    run(reinterpret_cast<const __nv_bfloat16*>(src.data_ptr()));
  else if (src.scalar_type() == at::kHalf)
    run(reinterpret_cast<const __half*>(src.data_ptr()));
  else
    TORCH_CHECK(false, "unsupported source dtype");
}

// Three-way split of an fp32 matrix: v = hi + mid + lo with every part a bf16 number, which carries
// the full 24-bit significand of v.  Six tensor-core products of such parts (hi*hi, hi*mid, mid*hi,
// hi*lo, mid*mid, lo*hi) reproduce an fp32 product to ~2^-24.
void cast_split3(at::Tensor src, at::Tensor hi, at::Tensor mid, at::Tensor lo) {
  TORCH_CHECK(src.is_cuda() && src.dim() == 2 && unit_columns(src) && src.scalar_type() == at::kFloat,
              "src must be a 2-D fp32 CUDA tensor with unit column stride");
  for (const at::Tensor* t : {&hi, &mid, &lo})
    TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kBFloat16 && t->dim() == 2 && t->is_contiguous() &&
                    t->size(0) == src.size(0) && t->size(1) >= src.size(1) && t->sizes() == hi.sizes(),
                "outputs must be contiguous bf16 [rows, >= n] tensors of one shape");
  c10::cuda::CUDAGuard guard(src.get_device());
  const long long rows = src.size(0);
  const long long ldo = hi.size(1);
  if (rows == 0) return;
  TORCH_CHECK(ldo > 0, "the outputs have no columns");
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  launch_cast<float, 3>(src.data_ptr<float>(), src.stride(0), 1.f, reinterpret_cast<__nv_bfloat16*>(hi.data_ptr()),
                        reinterpret_cast<__nv_bfloat16*>(mid.data_ptr()), reinterpret_cast<__nv_bfloat16*>(lo.data_ptr()),
                        ldo, rows, static_cast<int>(src.size(1)), stream);
}

// Grouped fp32 -> bf16 hi/lo staging: one launch converts many matrices.  Each table row holds
// (src fp32 ptr, hi ptr, lo ptr or 0, rows, n, src pitch, dst pitch) as int64.  blockIdx.y is the matrix;
// the grid is as wide as the largest matrix needs, so the CTAs of a small matrix past its end leave at once.
// Matrices whose rows are 16-byte aligned on both sides go eight elements per thread and trip (two 16-byte loads,
// one 16-byte store per part); the others one element at a time.
__global__ void __launch_bounds__(256) cast_pad_grouped_kernel(const long long* __restrict__ table) {
  const long long* e = table + static_cast<long long>(blockIdx.y) * 7;
  const float* src = reinterpret_cast<const float*>(e[0]);
  __nv_bfloat16* hi = reinterpret_cast<__nv_bfloat16*>(e[1]);
  __nv_bfloat16* lo = reinterpret_cast<__nv_bfloat16*>(e[2]);
  const long long rows = e[3], n = e[4], lds = e[5], ldo = e[6];
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  const long long first = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  const bool vec = ((n & 7) == 0) && ((ldo & 7) == 0) && ((lds & 3) == 0) &&
                   (((e[0] | e[1] | e[2]) & 15) == 0);
  if (vec) {
    const long long vpr = ldo >> 3, total = rows * vpr;
    for (long long v = first; v < total; v += step) {
      const long long r = v / vpr, c = (v - r * vpr) << 3;
      float x[8];
      if (c < n) {
        const float4 a = *reinterpret_cast<const float4*>(src + r * lds + c);
        const float4 b = *reinterpret_cast<const float4*>(src + r * lds + c + 4);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = 0.f;
      }
      uint32_t ph[4], pl[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const __nv_bfloat16 h0 = __float2bfloat16_rn(x[2 * k]), h1 = __float2bfloat16_rn(x[2 * k + 1]);
        const __nv_bfloat16 l0 = __float2bfloat16_rn(x[2 * k] - __bfloat162float(h0));
        const __nv_bfloat16 l1 = __float2bfloat16_rn(x[2 * k + 1] - __bfloat162float(h1));
        ph[k] = static_cast<uint32_t>(__bfloat16_as_ushort(h0)) | (static_cast<uint32_t>(__bfloat16_as_ushort(h1)) << 16);
        pl[k] = static_cast<uint32_t>(__bfloat16_as_ushort(l0)) | (static_cast<uint32_t>(__bfloat16_as_ushort(l1)) << 16);
      }
      *reinterpret_cast<uint4*>(hi + (v << 3)) = make_uint4(ph[0], ph[1], ph[2], ph[3]);
      if (lo != nullptr) *reinterpret_cast<uint4*>(lo + (v << 3)) = make_uint4(pl[0], pl[1], pl[2], pl[3]);
    }
    return;
  }
  const long long total = rows * ldo;
  for (long long i = first; i < total; i += step) {
    const long long r = i / ldo;
    const long long c = i - r * ldo;
    const float v = (c < n) ? src[r * lds + c] : 0.f;
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    hi[i] = h;
    if (lo != nullptr) lo[i] = __float2bfloat16_rn(v - __bfloat162float(h));
  }
}

// `max_elems`: rows x destination pitch of the largest matrix of the table (0: unknown, a narrow grid is used).
void cast_pad_bf16_grouped(at::Tensor table, int64_t count, int64_t max_elems) {
  TORCH_CHECK(table.is_cuda() && table.scalar_type() == at::kLong && table.is_contiguous() &&
                  table.numel() == count * 7, "table must be a CUDA int64 [count, 7] tensor");
  if (count == 0) return;
  c10::cuda::CUDAGuard guard(table.get_device());
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  // eight elements per thread and at least two trips per thread for the largest matrix, at most 512 CTAs per matrix
  int gx = 32;
  if (max_elems > 0) gx = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((max_elems / 8 + 511) / 512, 512)));
  cast_pad_grouped_kernel<<<dim3(gx, static_cast<unsigned>(count)), 256, 0, stream>>>(
      reinterpret_cast<const long long*>(table.data_ptr<int64_t>()));
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
}

// Casts of many tensors between fp32 and bf16 in one launch: the weights of a model and their gradients.  A block converts a piece of
// MC_PIECE elements, eight per thread and trip; which tensor it belongs to comes from a table in the kernel's parameters, so that a
// captured launch does not refer to host memory.  Bytes bound it: the weights of a bottleneck ResNet of four blocks
// (11 million) to bf16 and their gradients to fp32 24.0 + 21.7 us (PyTorch's copies of tensor lists) -> 11.8 + 14.5.
constexpr int MC_TENSORS = 128, MC_PIECE = 8192;
struct CastTable {
  const void* src[MC_TENSORS];
  void* dst[MC_TENSORS];
  long long count[MC_TENSORS];
  int first[MC_TENSORS + 1];   // block
  int tensors;
};
template <bool TO_BF16>
__global__ void __launch_bounds__(256) cast_many_kernel(const __grid_constant__ CastTable t) {
  int lo = 0, hi = t.tensors;   // the last tensor whose first block is not past this one
  while (hi - lo > 1) {
    const int mid = (lo + hi) / 2;
    (t.first[mid] <= static_cast<int>(blockIdx.x) ? lo : hi) = mid;
  }
  const long long begin = static_cast<long long>(blockIdx.x - t.first[lo]) * MC_PIECE, end = min(begin + MC_PIECE, t.count[lo]);
  using Src = std::conditional_t<TO_BF16, float, __nv_bfloat16>;
  using Dst = std::conditional_t<TO_BF16, __nv_bfloat16, float>;
  const Src* src = static_cast<const Src*>(t.src[lo]);
  Dst* dst = static_cast<Dst*>(t.dst[lo]);
  const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0;
  const long long whole = vec ? begin + (end - begin) / 8 * 8 : begin;
  if (vec) {
    constexpr int TRIPS = MC_PIECE / (256 * 8);
    uint4 a[TRIPS], b[TO_BF16 ? TRIPS : 1];
#pragma unroll
    for (int u = 0; u < TRIPS; ++u) {
      const long long at = begin + (u * 256 + threadIdx.x) * 8;
      if (at < whole) {
        const uint4* from = reinterpret_cast<const uint4*>(src + at);
        a[u] = from[0];
        if (TO_BF16) b[u] = from[1];
      }
    }
#pragma unroll
    for (int u = 0; u < TRIPS; ++u) {
      const long long at = begin + (u * 256 + threadIdx.x) * 8;
      if (at >= whole) break;
      const uint32_t w[4] = {a[u].x, a[u].y, a[u].z, a[u].w};
      uint4* to = reinterpret_cast<uint4*>(dst + at);
      if constexpr (TO_BF16) {
        const uint32_t v[8] = {w[0], w[1], w[2], w[3], b[u].x, b[u].y, b[u].z, b[u].w};
        uint32_t out[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
          out[k] = reinterpret_cast<const uint32_t&>(h);
        }
        to[0] = make_uint4(out[0], out[1], out[2], out[3]);
      } else {
        to[0] = make_uint4(w[0] << 16, w[0] & 0xffff0000u, w[1] << 16, w[1] & 0xffff0000u);
        to[1] = make_uint4(w[2] << 16, w[2] & 0xffff0000u, w[3] << 16, w[3] & 0xffff0000u);
      }
    }
  }
  for (long long at = whole + threadIdx.x; at < end; at += 256) {
    if constexpr (TO_BF16)
      dst[at] = __float2bfloat16_rn(src[at]);
    else
      dst[at] = __bfloat162float(src[at]);
  }
}

// dst[i] <- src[i].  Pairs of one memory layout and of fp32 and bf16 are converted together, the others one by one.
void cast_many(std::vector<at::Tensor> dst, std::vector<at::Tensor> src) {
  TORCH_CHECK(dst.size() == src.size(), "dst and src must have the same length");
  if (dst.empty()) return;
  const auto alike = [](const at::Tensor& a, const at::Tensor& b) {
    if (!values_in_memory(a) || !values_in_memory(b) || !a.is_cuda() || a.device() != b.device() || a.sizes() != b.sizes() || !a.is_non_overlapping_and_dense() || !b.is_non_overlapping_and_dense()) return false;
    for (int64_t k = 0; k < a.dim(); ++k)
      if (a.size(k) > 1 && a.stride(k) != b.stride(k)) return false;
    return true;
  };
  const at::Device device = dst[0].device();
  c10::cuda::OptionalCUDAGuard guard;
  if (device.is_cuda()) guard.set_device(device);
  for (const bool to_bf16 : {true, false}) {
    CastTable t;
    int blocks = 0;
    t.tensors = 0;
    const auto flush = [&] {
      if (t.tensors == 0) return;
      t.first[t.tensors] = blocks;
      auto kernel = to_bf16 ? cast_many_kernel<true> : cast_many_kernel<false>;
      kernel<<<blocks, 256, 0, at::cuda::getCurrentCUDAStream(device.index()).stream()>>>(t);
      B200_CUDA_CHECK(cudaGetLastError());
      count_launch();
      blocks = t.tensors = 0;
    };
    for (size_t i = 0; i < dst.size(); ++i) {
      const at::Tensor &d = dst[i], &s = src[i];
      const bool down = s.scalar_type() == at::kFloat && d.scalar_type() == at::kBFloat16;
      const bool up = s.scalar_type() == at::kBFloat16 && d.scalar_type() == at::kFloat;
      const bool together = (down || up) && s.device() == device && alike(d, s);
      if (!together) {
        if (!to_bf16) d.copy_(s);   // in the second round only
        continue;
      }
      if (down != to_bf16 || d.numel() == 0) continue;
      const long long pieces = (d.numel() + MC_PIECE - 1) / MC_PIECE;
      if (t.tensors == MC_TENSORS || blocks + pieces > (1 << 30)) flush();
      t.src[t.tensors] = s.data_ptr();
      t.dst[t.tensors] = d.data_ptr();
      t.count[t.tensors] = d.numel();
      t.first[t.tensors++] = blocks;
      blocks += static_cast<int>(pieces);
    }
    flush();
  }
}

// Transposing cast bf16 -> fp32: dst[i][j] = float(src[j * src_ld + i]) for i < rows, j < cols.
// Weight gradients of linear layers leave autograd as transposed (column-major) bf16 tensors; this
// brings one into the row-major fp32 layout of the parameter in one coalesced pass (32 x 32 tiles
// through shared memory).  All arguments are kernel parameters, so the launch can be captured in a
// CUDA graph.
__global__ void transpose_cast_kernel(const __nv_bfloat16* __restrict__ src, float* __restrict__ dst,
                                      long long rows, long long cols, long long lds, long long ldd) {
  __shared__ float tile[32][33];
  const long long tiles_r = (rows + 31) / 32, tiles_c = (cols + 31) / 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  for (long long t = blockIdx.x; t < tiles_r * tiles_c; t += gridDim.x) {
    const long long tr = t / tiles_c, tc = t - tr * tiles_c;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long j = tc * 32 + ty + 8 * k, i = tr * 32 + tx;
      tile[ty + 8 * k][tx] = (i < rows && j < cols) ? __bfloat162float(src[j * lds + i]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long i = tr * 32 + ty + 8 * k, j = tc * 32 + tx;
      if (i < rows && j < cols) dst[i * ldd + j] = tile[tx][ty + 8 * k];
    }
    __syncthreads();
  }
}

// src: bf16 [rows, cols] tensor with strides (1, ld) (a transposed matrix); dst: fp32 [rows, cols] row-major.
void transpose_cast(at::Tensor src, at::Tensor dst) {
  TORCH_CHECK(src.is_cuda() && dst.is_cuda() && src.dim() == 2 && dst.dim() == 2 && src.sizes() == dst.sizes(),
              "src and dst must be CUDA matrices of the same shape");
  TORCH_CHECK(src.scalar_type() == at::kBFloat16 && dst.scalar_type() == at::kFloat, "bf16 -> fp32 only");
  TORCH_CHECK(src.stride(0) == 1 && src.stride(1) >= src.size(0) && dst.stride(1) == 1 && dst.stride(0) >= dst.size(1),
              "src must be column-major and dst row-major");
  const long long rows = src.size(0), cols = src.size(1);
  if (rows == 0 || cols == 0) return;
  c10::cuda::CUDAGuard guard(src.get_device());
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  const long long tiles = ((rows + 31) / 32) * ((cols + 31) / 32);
  const int grid = static_cast<int>(std::min<long long>(tiles, 148LL * 8));
  transpose_cast_kernel<<<grid, 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(src.data_ptr()),
                                                  dst.data_ptr<float>(), rows, cols, src.stride(1), dst.stride(0));
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
}

struct Im2colParams {
  long long sN, sC, sH, sW;  // input strides in elements
  int N, C, H, W;
  int KH, KW, SH, SW, PH, PW, DH, DW;
  int Ho, Wo;
  long long ldo;   // output row pitch (elements), >= C*KH*KW
  int c_major;     // 1: columns ordered (c, kh, kw); 0: (kh, kw, c)
};

// Scalar path: one thread per output element (coalesced along the output row).
template <typename T>
__global__ void im2col_generic_kernel(const T* __restrict__ x, __nv_bfloat16* __restrict__ out,
                                      __nv_bfloat16* __restrict__ out_lo, Im2colParams p) {
  const long long rows = static_cast<long long>(p.N) * p.Ho * p.Wo;
  const long long total = rows * p.ldo;
  const int ncols = p.C * p.KH * p.KW;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long r = i / p.ldo;
    const int col = static_cast<int>(i - r * p.ldo);
    float v = 0.f;
    if (col < ncols) {
      int c, kh, kw;
      if (p.c_major) {
        c = col / (p.KH * p.KW);
        const int t = col - c * p.KH * p.KW;
        kh = t / p.KW;
        kw = t - kh * p.KW;
      } else {
        const int t = col / p.C;
        c = col - t * p.C;
        kh = t / p.KW;
        kw = t - kh * p.KW;
      }
      const int wo = static_cast<int>(r % p.Wo);
      const long long t2 = r / p.Wo;
      const int ho = static_cast<int>(t2 % p.Ho);
      const int n = static_cast<int>(t2 / p.Ho);
      const int hi = ho * p.SH - p.PH + kh * p.DH;
      const int wi = wo * p.SW - p.PW + kw * p.DW;
      if (hi >= 0 && hi < p.H && wi >= 0 && wi < p.W)
        v = to_f32<T>(x[n * p.sN + c * p.sC + hi * p.sH + wi * p.sW]);
    }
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    out[i] = h;
    if (out_lo != nullptr) out_lo[i] = __float2bfloat16_rn(v - __bfloat162float(h));
  }
}

// Output pixel -> (image, row, column), 32-bit (the host checks that the rows fit).
__device__ __forceinline__ void im2col_pixel(const Im2colParams& p, unsigned r, int& n, int& ho, int& wo) {
  const unsigned t = r / static_cast<unsigned>(p.Wo);
  wo = static_cast<int>(r - t * p.Wo);
  n = static_cast<int>(t / static_cast<unsigned>(p.Ho));
  ho = static_cast<int>(t - static_cast<unsigned>(n) * p.Ho);
}

// Vector path: channels_last bf16 input, C % 8 == 0, (kh, kw, c) column order.  One thread owns 8 channels (16 bytes)
// of one tap and walks down the output pixels (row_walk.h) with the loads of four in flight: the write of the patch
// matrix bounds it (14 x 14 x 256 channels, 32 images, 3 x 3: 28.9 MB).
__global__ void __launch_bounds__(256)
im2col_nhwc_vec8_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ out, Im2colParams p,
                        unsigned rows, int groups, int lanes) {
  constexpr int U = 4;
  const int c8n = p.C >> 3, lane = threadIdx.x / groups;
  const int v = blockIdx.y * groups + threadIdx.x % groups;
  if (lane >= lanes || v >= p.KH * p.KW * c8n) return;
  const int tap = v / c8n, c8 = v - tap * c8n;
  const int dh = (tap / p.KW) * p.DH - p.PH, dw = (tap % p.KW) * p.DW - p.PW;
  const __nv_bfloat16* base = x + c8 * 8;
  const unsigned step = gridDim.x * lanes;
  for (unsigned long long r = static_cast<unsigned long long>(blockIdx.x) * lanes + lane; r < rows;
       r += static_cast<unsigned long long>(U) * step) {
    uint4 val[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      val[u] = make_uint4(0, 0, 0, 0);
      const unsigned long long ru = r + static_cast<unsigned long long>(u) * step;
      if (ru < rows) {
        int n, ho, wo;
        im2col_pixel(p, static_cast<unsigned>(ru), n, ho, wo);
        const int hi = ho * p.SH + dh, wi = wo * p.SW + dw;
        if (hi >= 0 && hi < p.H && wi >= 0 && wi < p.W)
          val[u] = __ldg(reinterpret_cast<const uint4*>(base + n * p.sN + hi * p.sH + wi * p.sW));
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned long long ru = r + static_cast<unsigned long long>(u) * step;
      if (ru < rows) *reinterpret_cast<uint4*>(out + ru * p.ldo + static_cast<long long>(v) * 8) = val[u];
    }
  }
}

// Tile path (any dtype and strides): a CTA stages the input rows that one output row and `cc` channels need in shared
// memory, then every thread assembles eight consecutive columns of a patch from there (a table in shared memory maps
// column -> byte offset of the staged element) and writes 16 bytes per part.  Input is read once per filter row and
// coalesced along W (or along C for channels-innermost strides) with IM2COL_LOADS loads in flight per thread; padding is
// zeroed shared memory and the columns of the row pitch point at a zero row, so the assembly has no conditions.  What
// remains is the write of the patch matrix.  grid: (N * Ho, channel chunks).  c_major columns of a chunk are contiguous;
// (kh, kw, c) order needs all channels.
constexpr int IM2COL_LOADS = 8;
template <typename T, bool LO>
__global__ void __launch_bounds__(256)
im2col_tile_kernel(const T* __restrict__ x, __nv_bfloat16* __restrict__ out, __nv_bfloat16* __restrict__ out_lo,
                   Im2colParams p, int cc, int wp, int fast_lanes) {
  extern __shared__ float4 im2col_smem[];
  float* tile = reinterpret_cast<float*>(im2col_smem);   // [cc][KH][wp], a zero row [wp], then the column table
  const int taps = p.KH * p.KW, c_begin = blockIdx.y * cc, nc = min(cc, p.C - c_begin);
  const int elems = cc * p.KH * wp, cols = nc * taps, floats = (elems + wp + 3) / 4 * 4;
  const bool last = c_begin + nc == p.C;
  const long long col0 = static_cast<long long>(c_begin) * taps;
  const int width = last ? static_cast<int>(p.ldo - col0) : cols;   // with the zero padding of the row pitch
  unsigned short* table = reinterpret_cast<unsigned short*>(tile + floats);
  const int n = blockIdx.x / p.Ho, ho = blockIdx.x - n * p.Ho;
  for (int e = threadIdx.x; e < floats / 4; e += 256) im2col_smem[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int col = threadIdx.x; col < width; col += 256) {
    int at = elems;   // the zero row: padding columns
    if (col < cols) {
      const int c = p.c_major ? col / taps : col % p.C, t = p.c_major ? col - c * taps : col / p.C;
      at = (c * p.KH + t / p.KW) * wp + (t % p.KW) * p.DW;
    }
    table[col] = static_cast<unsigned short>(at * 4);
  }
  __syncthreads();
  // `fast_lanes` consecutive threads read consecutive elements of the dimension with the smaller stride (W, or C for
  // channels-innermost strides) of one row (c, kh), or (w, kh)
  const T* base = x + n * p.sN + c_begin * p.sC;
  const int h0 = ho * p.SH - p.PH, w_end = min(p.W, wp - p.PW);   // input columns that some output pixel reads
  const bool along_c = p.sC == 1;
  const int fast = along_c ? nc : w_end, slow = (along_c ? w_end : nc) * p.KH;
  const int f0 = threadIdx.x % fast_lanes, rows = 256 / fast_lanes;
  // FULL: all slots of the round have work.  The slots of other rounds are skipped by a branch: where the slow dimension is
  // short, most are empty, and their divisions bounded the kernel; in full rounds the branch keeps loads from overlapping.
  auto round = [&](auto full, int f, int t0) {
    constexpr bool FULL = decltype(full)::value;
    T v[IM2COL_LOADS];
    int to[IM2COL_LOADS];
#pragma unroll
    for (int u = 0; u < IM2COL_LOADS; ++u) {
      const int t = t0 + u * rows;
      to[u] = -1;
      if (!FULL && t >= slow) continue;
      const int s = t / p.KH, kh = t - s * p.KH, hi = h0 + kh * p.DH;
      const int c = along_c ? f : s, w = along_c ? s : f;
      if (hi >= 0 && hi < p.H) {
        to[u] = (c * p.KH + kh) * wp + w + p.PW;
        v[u] = __ldg(base + c * p.sC + hi * p.sH + w * p.sW);
      }
    }
#pragma unroll
    for (int u = 0; u < IM2COL_LOADS; ++u)
      if (to[u] >= 0) tile[to[u]] = to_f32<T>(v[u]);
  };
  for (int f = f0; f < fast; f += fast_lanes) {
    int t0 = threadIdx.x / fast_lanes;
    for (; t0 + (IM2COL_LOADS - 1) * rows < slow; t0 += IM2COL_LOADS * rows) round(std::true_type{}, f, t0);
    if (t0 < slow) round(std::false_type{}, f, t0);
  }
  __syncthreads();
  const int vecs = width / 8;
  __nv_bfloat16* const row0 = out + static_cast<long long>(blockIdx.x) * p.Wo * p.ldo + col0;
  __nv_bfloat16* const lo0 = LO ? out_lo + static_cast<long long>(blockIdx.x) * p.Wo * p.ldo + col0 : nullptr;
  const int step_wo = 256 / vecs, step_v = 256 - step_wo * vecs;
  int wo = threadIdx.x / vecs, v = threadIdx.x - wo * vecs;
  while (wo < p.Wo) {
    const uint4 raw = *reinterpret_cast<const uint4*>(table + v * 8);
    const uint32_t pairs[4] = {raw.x, raw.y, raw.z, raw.w};
    const char* from = reinterpret_cast<const char*>(tile + wo * p.SW);
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float a = *reinterpret_cast<const float*>(from + (pairs[k] & 0xffffu));
      const float b = *reinterpret_cast<const float*>(from + (pairs[k] >> 16));
      const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
      hi[k] = *reinterpret_cast<const uint32_t*>(&h);
      if (LO) {
        const __nv_bfloat162 l = __floats2bfloat162_rn(a - __low2float(h), b - __high2float(h));
        lo[k] = *reinterpret_cast<const uint32_t*>(&l);
      }
    }
    const long long at = static_cast<long long>(wo) * p.ldo + v * 8;
    *reinterpret_cast<uint4*>(row0 + at) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    if (LO) *reinterpret_cast<uint4*>(lo0 + at) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    wo += step_wo;
    v += step_v;
    if (v >= vecs) {
      v -= vecs;
      ++wo;
    }
  }
}

// Channels per CTA of the tile path, 0 if it does not apply: the staged rows and the column table fit `IM2COL_SMEM` (so a
// byte offset has 16 bits), each chunk starts on a multiple of eight columns, and it is expected to take less time than the
// element-wise kernel.
constexpr int IM2COL_SMEM = 44 * 1024;
struct Im2colTile {
  int cc, wp, smem, fast_lanes;
};

// Expected times in us, fitted to 480 shapes of 30 thousand to 58 million patch elements (5 % and 13 % off on average; the
// rule they give picks a kernel within 0.2 % of the better one on average).  The element-wise kernel is bound by its index
// divisions per element.  A CTA of the tile kernel goes through rounds of loads, the divisions of its column table and the
// assembly: one such chain where every SM has at most one CTA, the sum of their issue times where it has several.  Below
// 100 thousand elements, for images of one output pixel and for 1 x 1 filters over few pixels and many channels the former is
// faster (32 x 64 x 8 x 8 under an 8 x 8 filter: 3.6 and 7.6 us; 32 x 1024 x 14 x 14 channels_last fp32 under a strided
// 1 x 1 filter: 17 and 25 us).
inline float im2col_generic_us(const Im2colParams& p) {
  return 2.5f + 7.7e-6f * static_cast<float>(p.N) * p.Ho * p.Wo * p.ldo;
}
inline float im2col_tile_us(const Im2colParams& p, const Im2colTile& t) {
  auto up = [](long long a, long long b) { return static_cast<float>((a + b - 1) / b); };
  const long long w_end = std::min(p.W, t.wp), fast = p.sC == 1 ? t.cc : w_end, slow = (p.sC == 1 ? w_end : t.cc) * p.KH;
  const long long lane_rows = 256 / t.fast_lanes, cols = static_cast<long long>(t.cc) * p.KH * p.KW;
  const float rounds = up(fast, t.fast_lanes) * up(slow, lane_rows * IM2COL_LOADS);
  const float loads = up(fast, t.fast_lanes) * up(slow, lane_rows), table = up(cols, 256), pieces = up(cols * p.Wo, 8 * 256);
  const float ctas = static_cast<float>(p.N) * p.Ho * up(p.C, t.cc);
  return std::max(2.05f + 0.35f * rounds + 0.12f * loads + 0.18f * table + 0.15f * pieces,
                  2.f + ctas / 148 * (0.165f * rounds + 0.084f * loads + 0.173f * table + 0.081f * pieces));
}

Im2colTile im2col_tile_plan(const Im2colParams& p) {
  const Im2colTile none{0, 0, 0, 0};
  const long long taps = static_cast<long long>(p.KH) * p.KW;
  const long long wp = (static_cast<long long>(p.Wo - 1) * p.SW + static_cast<long long>(p.KW - 1) * p.DW + 1) | 1;
  auto smem = [&](long long cc) {
    return ((cc * p.KH * wp + wp + 3) / 4 * 4) * 4 + (cc * taps + 8) * 2 + (p.ldo - static_cast<long long>(p.C) * taps) * 2;
  };
  auto fits = [&](long long cc) { return smem(cc) <= IM2COL_SMEM; };
  if (p.ldo % 8 != 0 || p.PH < 0 || p.PW < 0 || static_cast<long long>(p.N) * p.Ho >= (1ll << 31)) return none;
  long long cc = p.C;
  if (!fits(cc)) {
    if (!p.c_major) return none;
    cc = p.C / 8 * 8;
    while (cc > 0 && !fits(cc)) cc -= 8;
    if (cc <= 0) return none;
    const long long chunks = (p.C + cc - 1) / cc;             // equal chunks
    cc = ((p.C + chunks - 1) / chunks + 7) / 8 * 8;
  }
  if ((p.C + cc - 1) / cc > 65535) return none;
  const long long fast = p.sC == 1 ? std::min<long long>(cc, p.C) : std::min<long long>(p.W, wp);
  int lanes = 4;
  while (lanes < fast && lanes < 32) lanes *= 2;
  const Im2colTile tile{static_cast<int>(cc), static_cast<int>(wp), static_cast<int>(smem(cc)), lanes};
  return im2col_tile_us(p, tile) < im2col_generic_us(p) ? tile : none;
}

// x: 4-D conv input [N, C, H, W] (logical), any memory format.  out: [N*Ho*Wo, ld] bf16, contiguous.
void im2col_bf16(at::Tensor x, at::Tensor out, c10::optional<at::Tensor> out_lo,
                 std::vector<int64_t> kernel, std::vector<int64_t> stride,
                 std::vector<int64_t> padding, std::vector<int64_t> dilation, bool c_major) {
  TORCH_CHECK(x.is_cuda() && x.dim() == 4, "x must be a 4-D CUDA tensor");
  TORCH_CHECK(out.is_cuda() && out.is_contiguous() && out.scalar_type() == at::kBFloat16 &&
                  out.dim() == 2, "out must be contiguous 2-D bf16");
  Im2colParams p;
  p.N = x.size(0); p.C = x.size(1); p.H = x.size(2); p.W = x.size(3);
  p.sN = x.stride(0); p.sC = x.stride(1); p.sH = x.stride(2); p.sW = x.stride(3);
  p.KH = kernel[0]; p.KW = kernel[1]; p.SH = stride[0]; p.SW = stride[1];
  p.PH = padding[0]; p.PW = padding[1]; p.DH = dilation[0]; p.DW = dilation[1];
  p.Ho = (p.H + 2 * p.PH - p.DH * (p.KH - 1) - 1) / p.SH + 1;
  p.Wo = (p.W + 2 * p.PW - p.DW * (p.KW - 1) - 1) / p.SW + 1;
  p.ldo = out.size(1);
  p.c_major = c_major ? 1 : 0;
  const long long rows = static_cast<long long>(p.N) * p.Ho * p.Wo;
  TORCH_CHECK(out.size(0) == rows && p.ldo >= static_cast<long long>(p.C) * p.KH * p.KW,
              "out has the wrong shape");
  if (rows == 0) return;
  TORCH_CHECK(p.ldo > 0, "the patch matrix has no columns");
  c10::cuda::CUDAGuard guard(x.get_device());
  auto stream = at::cuda::getCurrentCUDAStream().stream();
  auto* out_p = reinterpret_cast<__nv_bfloat16*>(out.data_ptr());
  __nv_bfloat16* lo_p = nullptr;
  if (out_lo.has_value()) {
    TORCH_CHECK(out_lo->sizes() == out.sizes() && out_lo->is_contiguous() &&
                    out_lo->scalar_type() == at::kBFloat16, "out_lo must match out");
    lo_p = reinterpret_cast<__nv_bfloat16*>(out_lo->data_ptr());
  }
  // with a single filter tap the (c, kh, kw) and (kh, kw, c) column orders are the same
  const bool vec = lo_p == nullptr && (!c_major || p.KH * p.KW == 1) && x.scalar_type() == at::kBFloat16 && p.sC == 1 && (p.C % 8) == 0 &&
                   p.ldo == static_cast<long long>(p.C) * p.KH * p.KW && (p.sW % 8) == 0 &&
                   (p.sH % 8) == 0 && (p.sN % 8) == 0 && rows < (1ll << 32) &&
                   ((reinterpret_cast<uintptr_t>(x.data_ptr()) | reinterpret_cast<uintptr_t>(out_p)) & 15) == 0 &&
                   p.ldo <= MAX_WALK_CHUNKS * 1024ll;   // below, a CTA covers half its vectors or more
  const bool aligned = ((reinterpret_cast<uintptr_t>(out_p) | reinterpret_cast<uintptr_t>(lo_p)) & 15) == 0;
  const Im2colTile tile = (vec || !aligned) ? Im2colTile{0, 0, 0, 0} : im2col_tile_plan(p);
  auto run = [&](auto* from) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(from)>>;
    if (tile.cc > 0) {
      const dim3 grid(static_cast<unsigned>(static_cast<long long>(p.N) * p.Ho), (p.C + tile.cc - 1) / tile.cc);
      if (lo_p != nullptr)
        im2col_tile_kernel<T, true><<<grid, 256, tile.smem, stream>>>(from, out_p, lo_p, p, tile.cc, tile.wp, tile.fast_lanes);
      else
        im2col_tile_kernel<T, false><<<grid, 256, tile.smem, stream>>>(from, out_p, nullptr, p, tile.cc, tile.wp, tile.fast_lanes);
    } else {
      const int blocks = static_cast<int>(std::min<long long>((rows * p.ldo + 255) / 256, 148 * 32));
      im2col_generic_kernel<T><<<blocks, 256, 0, stream>>>(from, out_p, lo_p, p);
    }
  };
  if (vec) {
    const Walk w = walk_plan(p.KH * p.KW * (p.C >> 3));
    // four pixels per thread; where that leaves SMs without a CTA, one (32 x 32 x 8 x 8, 3 x 3: 2.9 -> 2.4 us)
    dim3 grid = walk_grid(w, (rows + 3) / 4, 8);
    if (grid.x * grid.y < 148) grid = walk_grid(w, rows, 8);
    im2col_nhwc_vec8_kernel<<<grid, 256, 0, stream>>>(
        reinterpret_cast<const __nv_bfloat16*>(x.data_ptr()), out_p, p, static_cast<unsigned>(rows), w.groups, w.lanes);
  } else if (x.scalar_type() == at::kFloat) {
    run(static_cast<const float*>(x.data_ptr<float>()));
  } else if (x.scalar_type() == at::kBFloat16) {
    run(reinterpret_cast<const __nv_bfloat16*>(x.data_ptr()));
  } else if (x.scalar_type() == at::kHalf) {
    run(reinterpret_cast<const __half*>(x.data_ptr()));
  } else {
    TORCH_CHECK(false, "unsupported input dtype");
  }
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
}

}  // namespace b200
