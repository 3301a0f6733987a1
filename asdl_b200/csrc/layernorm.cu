// LayerNorm forward / backward over the last dimension for bf16 activations with fp32 parameters.
//
// A warp owns a row at a time; lane l holds the 8-element vectors l, l + 32, ... of the row in
// registers (VPL vectors per lane, so the feature size is 256 * VPL), which makes every global
// access a 16-byte load / store and the row statistics two warp reductions (mean first, then the
// centred sum of squares: no cancellation).  The backward pass produces the input gradient per
// row and accumulates the weight / bias gradients of the lane's own columns in registers over all
// rows of the warp; warps are combined through shared memory, CTAs through a [ctas, 2, d] partial
// buffer that a second kernel sums (one thread per column, coalesced over columns).
// Rows wider than 1024 elements are split over two or four warps (256 * VPL elements each, VPL <= 4), which
// meet at a named barrier for every row statistic: the backward kernel would otherwise need 40 registers
// per vector slot and spill from 1536 elements on.
//
// PyTorch's own kernels for the weight / bias gradient of LayerNorm take ~60 us per layer at
// d = 1024, 8192 rows on this GPU; these take the time of one pass over dy and x.
#include <cuda_bf16.h>

#include "host_utils.h"

namespace b200 {

namespace {

constexpr int LN_WARPS = 8;
constexpr int LN_THREADS = LN_WARPS * 32;
// CTAs of the backward kernel that an SM holds.  The row ahead takes it to 96 registers for VPL = 1, to the limit of 128 for
// VPL = 2 (48 bytes spilled) and to 218 - 255 for 3 and 4 (40 bytes spilled at <4, 2>): two CTAs up to VPL = 2, one above.
// Backward pass of 8192 rows without / with the row ahead: 256 columns 27 / 9 us, 512 33 / 15, 1024 44 / 19, 2048 57 / 27,
// 4096 93 / 45; of 64 rows 1.3 to 1.5 times as fast at every width.
constexpr int ln_bwd_ctas(int vpl) { return vpl <= 2 ? 2 : 1; }

__device__ __forceinline__ void ln_unpack8(const uint4& raw, float (&out)[8]) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    out[2 * i] = f.x;
    out[2 * i + 1] = f.y;
  }
}

__device__ __forceinline__ uint4 ln_pack8(const float (&v)[8]) {
  uint4 raw;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  return raw;
}

__device__ __forceinline__ float ln_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ void ln_load8(const float* p, float (&out)[8]) {
  const float4 lo = *reinterpret_cast<const float4*>(p), hi = *reinterpret_cast<const float4*>(p + 4);
  out[0] = lo.x; out[1] = lo.y; out[2] = lo.z; out[3] = lo.w;
  out[4] = hi.x; out[5] = hi.y; out[6] = hi.z; out[7] = hi.w;
}

// Sum over the SPLIT warps that share a row: every warp leaves its partial in shared memory, the group
// meets at a named barrier and every warp adds the SPLIT partials.  `slot` alternates so that one barrier
// per reduction is enough (a warp can only be one reduction ahead of the slowest warp of its group).
template <int SPLIT>
__device__ __forceinline__ float ln_group_sum(float v, float (*scratch)[LN_WARPS], int& slot, int warp) {
  v = ln_warp_sum(v);
  if constexpr (SPLIT == 1) return v;
  const int group = warp / SPLIT;
  if ((threadIdx.x & 31) == 0) scratch[slot][warp] = v;
  asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(SPLIT * 32) : "memory");
  float t = 0.f;
#pragma unroll
  for (int s = 0; s < SPLIT; ++s) t += scratch[slot][group * SPLIT + s];
  slot = (slot + 1) % 3;
  return t;
}

// A row of D = 256 * VPL * SPLIT elements is handled by SPLIT warps, each keeping 256 * VPL of it in
// registers (VPL 16-byte vectors per lane); SPLIT > 1 keeps the register need of wide rows at that of VPL <= 4.
template <int VPL, int SPLIT>
__global__ void __launch_bounds__(LN_THREADS)
ln_fwd_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ gamma,
              const float* __restrict__ beta, __nv_bfloat16* __restrict__ y, float* __restrict__ mean_out,
              float* __restrict__ rstd_out, long long rows, float eps) {
  constexpr int D = 256 * VPL * SPLIT;
  constexpr int GROUPS = LN_WARPS / SPLIT;
  __shared__ float scratch[3][LN_WARPS];
  int slot = 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group = warp / SPLIT, col0 = (warp % SPLIT) * 256 * VPL;
  float g[VPL][8], b[VPL][8];
#pragma unroll
  for (int v = 0; v < VPL; ++v) {
    ln_load8(gamma + col0 + (v * 32 + lane) * 8, g[v]);
    ln_load8(beta + col0 + (v * 32 + lane) * 8, b[v]);
  }
  for (long long r = static_cast<long long>(blockIdx.x) * GROUPS + group; r < rows;
       r += static_cast<long long>(gridDim.x) * GROUPS) {
    const __nv_bfloat16* xr = x + r * D + col0;
    float xv[VPL][8];
    float s = 0.f;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      ln_unpack8(__ldg(reinterpret_cast<const uint4*>(xr + (v * 32 + lane) * 8)), xv[v]);
#pragma unroll
      for (int i = 0; i < 8; ++i) s += xv[v][i];
    }
    const float mean = ln_group_sum<SPLIT>(s, scratch, slot, warp) * (1.f / D);
    float q = 0.f;
#pragma unroll
    for (int v = 0; v < VPL; ++v)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float c = xv[v][i] - mean;
        q = fmaf(c, c, q);
      }
    const float rstd = rsqrtf(ln_group_sum<SPLIT>(q, scratch, slot, warp) * (1.f / D) + eps);
    __nv_bfloat16* yr = y + r * D + col0;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      float out[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) out[i] = fmaf((xv[v][i] - mean) * rstd, g[v][i], b[v][i]);
      *reinterpret_cast<uint4*>(yr + (v * 32 + lane) * 8) = ln_pack8(out);
    }
    if (lane == 0 && col0 == 0) {
      mean_out[r] = mean;
      rstd_out[r] = rstd;
    }
  }
}

// The next row of x and dy is loaded while the current one is reduced: a warp has only a few rows, and each waited for its
// loads.  Rows are kept as the loaded bf16 vectors (half the registers of their fp32 values), unpacked once per use.
template <int VPL, int SPLIT>
__global__ void __launch_bounds__(LN_THREADS, ln_bwd_ctas(VPL))
ln_bwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ dy,
              const float* __restrict__ gamma, const float* __restrict__ mean, const float* __restrict__ rstd,
              __nv_bfloat16* __restrict__ dx, float* __restrict__ part, long long rows) {
  constexpr int D = 256 * VPL * SPLIT;
  constexpr int GROUPS = LN_WARPS / SPLIT;
  __shared__ float red[LN_WARPS][2][32 * 8 + 1];  // one vector slot (v) at a time
  __shared__ float scratch[3][LN_WARPS];
  int slot = 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int group = warp / SPLIT, col0 = (warp % SPLIT) * 256 * VPL;
  const long long step = static_cast<long long>(gridDim.x) * GROUPS;
  long long r = static_cast<long long>(blockIdx.x) * GROUPS + group;
  uint4 rx[VPL], rg[VPL];
  float mu = 0.f, rs = 0.f;
  auto load_row = [&](long long row, uint4 (&ax)[VPL], uint4 (&ag)[VPL], float& m, float& s) {
    const long long at = row * D + col0 + lane * 8;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      ax[v] = __ldg(reinterpret_cast<const uint4*>(x + at + v * 256));
      ag[v] = __ldg(reinterpret_cast<const uint4*>(dy + at + v * 256));
    }
    m = __ldg(mean + row);
    s = __ldg(rstd + row);
  };
  if (r < rows) load_row(r, rx, rg, mu, rs);
  float g[VPL][8], dg[VPL][8], db[VPL][8];
#pragma unroll
  for (int v = 0; v < VPL; ++v) {
    ln_load8(gamma + col0 + (v * 32 + lane) * 8, g[v]);
#pragma unroll
    for (int i = 0; i < 8; ++i) dg[v][i] = db[v][i] = 0.f;
  }
  for (; r < rows; r += step) {
    uint4 nx[VPL], ng[VPL];
    float nmu = 0.f, nrs = 0.f;
    const bool more = r + step < rows;
    if (more) load_row(r + step, nx, ng, nmu, nrs);
    float c1 = 0.f, c2 = 0.f;
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      float xv[8], dv[8];
      ln_unpack8(rx[v], xv);
      ln_unpack8(rg[v], dv);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float xh = (xv[i] - mu) * rs, gy = dv[i] * g[v][i];
        dg[v][i] = fmaf(dv[i], xh, dg[v][i]);
        db[v][i] += dv[i];
        c1 = fmaf(gy, xh, c1);
        c2 += gy;
      }
    }
    c1 = ln_group_sum<SPLIT>(c1, scratch, slot, warp) * (1.f / D);
    c2 = ln_group_sum<SPLIT>(c2, scratch, slot, warp) * (1.f / D);
#pragma unroll
    for (int v = 0; v < VPL; ++v) {
      float xv[8], dv[8], out[8];
      ln_unpack8(rx[v], xv);
      ln_unpack8(rg[v], dv);
#pragma unroll
      for (int i = 0; i < 8; ++i) out[i] = rs * (dv[i] * g[v][i] - c2 - (xv[i] - mu) * rs * c1);
      *reinterpret_cast<uint4*>(dx + r * D + col0 + (v * 32 + lane) * 8) = ln_pack8(out);
    }
    if (more) {
#pragma unroll
      for (int v = 0; v < VPL; ++v) {
        rx[v] = nx[v];
        rg[v] = ng[v];
      }
      mu = nmu;
      rs = nrs;
    }
  }
  // combine the warps of the CTA that hold the same columns, one vector slot at a time
  float* out = part + static_cast<size_t>(blockIdx.x) * 2 * D;
#pragma unroll
  for (int v = 0; v < VPL; ++v) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      red[warp][0][lane * 8 + i] = dg[v][i];
      red[warp][1][lane * 8 + i] = db[v][i];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 2 * 256 * SPLIT; e += LN_THREADS) {
      const int col = e & 255, which = (e >> 8) & 1, slice = e >> 9;
      float s = 0.f;
#pragma unroll
      for (int gi = 0; gi < GROUPS; ++gi) s += red[gi * SPLIT + slice][which][col];
      out[which * D + slice * 256 * VPL + v * 256 + col] = s;
    }
    __syncthreads();
  }
}

// dgamma[j] = sum over CTAs of part[c][0][j], dbeta[j] likewise.  A CTA takes 32 of the 2 d sums (one 128-byte line per
// part) with FIN_LANES parts in flight at a time: one thread per sum walked all parts alone, a chain of as many loads as
// there are CTAs on eight SMs.
constexpr int FIN_LANES = 16;
__global__ void __launch_bounds__(32 * FIN_LANES)
ln_bwd_finalize(const float* __restrict__ part, float* __restrict__ dgamma, float* __restrict__ dbeta, int ctas, int d) {
  __shared__ float red[FIN_LANES][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, j = blockIdx.x * 32 + tx;   // d is a multiple of 32
  const float* from = part + j;
  float s = 0.f;
#pragma unroll 4
  for (int c = ty; c < ctas; c += FIN_LANES) s += from[static_cast<size_t>(c) * 2 * d];
  red[ty][tx] = s;
  __syncthreads();
  if (ty != 0) return;
  s = 0.f;
#pragma unroll
  for (int k = 0; k < FIN_LANES; ++k) s += red[k][tx];
  if (j < d)
    dgamma[j] = s;
  else
    dbeta[j - d] = s;
}

int ln_grid(long long rows, int groups, int per_sm) {
  return static_cast<int>(std::max<long long>(1, std::min<long long>((rows + groups - 1) / groups, 148LL * per_sm)));
}

void ln_check(const at::Tensor& x, const at::Tensor& gamma, int& vpl, long long& rows) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.is_contiguous() && x.dim() >= 1,
              "x must be a contiguous bf16 CUDA tensor");
  const long long d = x.size(-1);
  TORCH_CHECK(d % 256 == 0 && d >= 256 && d <= 4096, "the normalised size must be a multiple of 256 up to 4096");
  vpl = static_cast<int>(d / 256);
  TORCH_CHECK(vpl == 1 || vpl == 2 || vpl == 3 || vpl == 4 || vpl == 6 || vpl == 8 || vpl == 12 || vpl == 16,
              "unsupported normalised size");
  rows = x.numel() / d;
  TORCH_CHECK(gamma.is_cuda() && gamma.scalar_type() == at::kFloat && gamma.is_contiguous() && gamma.numel() == d,
              "weight must be a contiguous fp32 vector of the normalised size");
  TORCH_CHECK((reinterpret_cast<uintptr_t>(x.data_ptr()) & 15) == 0, "16-byte alignment required");
}

template <int V, int S>
void launch_fwd(int grid, cudaStream_t stream, const __nv_bfloat16* x, const float* gamma, const float* beta,
                __nv_bfloat16* y, float* mean, float* rstd, long long rows, float eps) {
  ln_fwd_kernel<V, S><<<grid, LN_THREADS, 0, stream>>>(x, gamma, beta, y, mean, rstd, rows, eps);
}

template <int V, int S>
void launch_bwd(int grid, cudaStream_t stream, const __nv_bfloat16* x, const __nv_bfloat16* dy, const float* gamma,
                const float* mean, const float* rstd, __nv_bfloat16* dx, float* part, long long rows) {
  ln_bwd_kernel<V, S><<<grid, LN_THREADS, 0, stream>>>(x, dy, gamma, mean, rstd, dx, part, rows);
}

// rows of 256 * v elements: up to v = 4 one warp per row, wider rows split over 2 or 4 warps
#define LN_DISPATCH(VPL_VALUE, FN, ...)         \
  switch (VPL_VALUE) {                          \
    case 1: FN<1, 1>(__VA_ARGS__); break;       \
    case 2: FN<2, 1>(__VA_ARGS__); break;       \
    case 3: FN<3, 1>(__VA_ARGS__); break;       \
    case 4: FN<4, 1>(__VA_ARGS__); break;       \
    case 6: FN<3, 2>(__VA_ARGS__); break;       \
    case 8: FN<4, 2>(__VA_ARGS__); break;       \
    case 12: FN<3, 4>(__VA_ARGS__); break;      \
    default: FN<4, 4>(__VA_ARGS__); break;      \
  }

// warps of a CTA that work on different rows at a time
int ln_vpl_of_warp(int vpl) { return vpl <= 4 ? vpl : (vpl % 3 == 0 ? 3 : 4); }
int ln_groups(int vpl) { return vpl <= 4 ? LN_WARPS : (vpl <= 8 ? LN_WARPS / 2 : LN_WARPS / 4); }

}  // namespace

bool ln_supported_size(int64_t d) {
  if (d % 256 != 0) return false;
  const int64_t v = d / 256;
  return v == 1 || v == 2 || v == 3 || v == 4 || v == 6 || v == 8 || v == 12 || v == 16;
}

// Returns (y, mean, rstd); mean / rstd have one entry per row.
std::vector<at::Tensor> ln_forward(at::Tensor x, at::Tensor weight, at::Tensor bias, double eps) {
  int vpl;
  long long rows;
  ln_check(x, weight, vpl, rows);
  TORCH_CHECK(bias.is_cuda() && bias.scalar_type() == at::kFloat && bias.is_contiguous() &&
                  bias.numel() == weight.numel(), "bias must match weight");
  const int dev = x.get_device();
  c10::cuda::CUDAGuard guard(dev);
  auto stream = at::cuda::getCurrentCUDAStream(dev).stream();
  auto y = at::empty_like(x);
  auto mean = at::empty({rows}, weight.options()), rstd = at::empty({rows}, weight.options());
  if (rows == 0) return {y, mean, rstd};
  const int grid = ln_grid(rows, ln_groups(vpl), 2);
  const auto* xp = reinterpret_cast<const __nv_bfloat16*>(x.data_ptr());
  auto* yp = reinterpret_cast<__nv_bfloat16*>(y.data_ptr());
  LN_DISPATCH(vpl, launch_fwd, grid, stream, xp, weight.data_ptr<float>(), bias.data_ptr<float>(), yp,
              mean.data_ptr<float>(), rstd.data_ptr<float>(), rows, static_cast<float>(eps));
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch();
  return {y, mean, rstd};
}

// Returns (dx, dweight, dbias).
std::vector<at::Tensor> ln_backward(at::Tensor x, at::Tensor dy, at::Tensor weight, at::Tensor mean,
                                    at::Tensor rstd) {
  int vpl;
  long long rows;
  ln_check(x, weight, vpl, rows);
  TORCH_CHECK(dy.is_cuda() && dy.scalar_type() == at::kBFloat16 && dy.is_contiguous() && dy.sizes() == x.sizes() &&
                  (reinterpret_cast<uintptr_t>(dy.data_ptr()) & 15) == 0, "dy must match x");
  TORCH_CHECK(mean.is_cuda() && rstd.is_cuda() && mean.scalar_type() == at::kFloat && rstd.scalar_type() == at::kFloat &&
                  mean.numel() == rows && rstd.numel() == rows && mean.is_contiguous() && rstd.is_contiguous(),
              "mean / rstd must hold one fp32 value per row");
  const int dev = x.get_device();
  c10::cuda::CUDAGuard guard(dev);
  auto stream = at::cuda::getCurrentCUDAStream(dev).stream();
  const long long d = x.size(-1);
  auto dx = at::empty_like(x);
  if (rows == 0) return {dx, at::zeros({d}, weight.options()), at::zeros({d}, weight.options())};
  auto dweight = at::empty({d}, weight.options()), dbias = at::empty({d}, weight.options());
  const int grid = ln_grid(rows, ln_groups(vpl), ln_bwd_ctas(ln_vpl_of_warp(vpl)));
  auto part = at::empty({grid, 2, d}, weight.options());
  const auto* xp = reinterpret_cast<const __nv_bfloat16*>(x.data_ptr());
  const auto* gp = reinterpret_cast<const __nv_bfloat16*>(dy.data_ptr());
  auto* dxp = reinterpret_cast<__nv_bfloat16*>(dx.data_ptr());
  LN_DISPATCH(vpl, launch_bwd, grid, stream, xp, gp, weight.data_ptr<float>(), mean.data_ptr<float>(),
              rstd.data_ptr<float>(), dxp, part.data_ptr<float>(), rows);
  ln_bwd_finalize<<<static_cast<int>(2 * d / 32), 32 * FIN_LANES, 0, stream>>>(
      part.data_ptr<float>(), dweight.data_ptr<float>(), dbias.data_ptr<float>(), grid, static_cast<int>(d));
  B200_CUDA_CHECK(cudaGetLastError());
  count_launch(2);
  return {dx, dweight, dbias};
}

}  // namespace b200
