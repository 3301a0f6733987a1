// Max-pooling (3 x 3 windows, stride 2) of NHWC (channels_last) bf16 activations, forward and backward.
//
// A thread takes 8 channels (16 bytes) of one output pixel and loads its window at once; the position of the maximum inside the window
// is kept as one byte per value, where PyTorch keeps eight.  The backward pass gathers: a thread takes 8 channels of the 2 x 2 input
// pixels that begin one window and lie in at most four, and adds, in fp32 and window after window, the gradients of the windows whose
// maximum a pixel is, so that every value is written once and needs no zeros first.  Comparisons and selections work on two values at
// a time.  Values and gradients are PyTorch's: the first of equal values wins, a NaN wins over everything before it.
//
// Instruction issue bounds both (62 and 76 % of the slots busy): 70 MB (51 of activations, 13 pooled, 6 of positions) would take memory
// 11 us, and a pass over 32 x 64 x 112 x 112 runs at half that rate.  In graphs: forward 112.7 (PyTorch's kernels) -> 20.2 us, backward 237.3 -> 19.4; 24 x 32 x 96 x 96 45.1 -> 7.0 and 107.4 -> 8.2, 4 x 16 x 32 x 32 9.8 -> 3.7 and 8.4 -> 2.0.  With
// a thread per input pixel, one window loaded after the other, the backward pass took 58.6.
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <cuda_bf16.h>
#include <torch/extension.h>

#include "host_utils.h"

namespace b200 {

namespace {

constexpr int POOL_THREADS = 256;

constexpr int K = 3, S = 2;
struct Pool {
  int vecs, h, w, oh, ow, pad;
};

// 0xffff in each half where `value` takes the place of `best`: greater, or a NaN
__device__ __forceinline__ uint32_t wins(uint32_t value, uint32_t best) {
  const __nv_bfloat162 v = reinterpret_cast<const __nv_bfloat162&>(value), b = reinterpret_cast<const __nv_bfloat162&>(best);
  return __hgt2_mask(v, b) | __hneu2_mask(v, v);
}

// One row of output pixels per blockIdx.y; the threads of a CTA are consecutive vectors of the row.
__global__ void __launch_bounds__(POOL_THREADS)
max_pool_forward_kernel(const uint4* __restrict__ x, uint4* __restrict__ y, uint2* __restrict__ code, const Pool s) {
  const int at = blockIdx.x * POOL_THREADS + threadIdx.x;
  if (at >= s.ow * s.vecs) return;
  const int ox = at / s.vecs, v = at - ox * s.vecs, left = ox * S - s.pad;
  const long long image = blockIdx.z;
  for (int oy = blockIdx.y; oy < s.oh; oy += gridDim.y) {
    const int top = oy * S - s.pad;
    const uint4* corner = x + ((image * s.h + top) * s.w + left) * s.vecs + v;
    uint4 raw[K * K];
#pragma unroll
    for (int i = 0; i < K; ++i)
#pragma unroll
      for (int j = 0; j < K; ++j)
        raw[i * K + j] = top + i >= 0 && top + i < s.h && left + j >= 0 && left + j < s.w
                             ? __ldg(corner + (static_cast<long long>(i) * s.w + j) * s.vecs)
                             : make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);   // -infinity
    // a window without a value above -infinity names the first pixel of the image, as PyTorch's indices do, or no pixel of its own
    const uint32_t first = (top <= 0 && left <= 0 ? -top * K - left : 0xff) * 0x00010001u;
    uint32_t best[4], where[4];   // two values each
#pragma unroll
    for (int i = 0; i < 4; ++i) best[i] = 0xff80ff80u, where[i] = first;
#pragma unroll
    for (int k = 0; k < K * K; ++k) {
      const uint32_t value[4] = {raw[k].x, raw[k].y, raw[k].z, raw[k].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t m = wins(value[i], best[i]);
        best[i] = (value[i] & m) | (best[i] & ~m);
        where[i] = (k * 0x00010001u & m) | (where[i] & ~m);
      }
    }
    const long long to = ((image * s.oh + oy) * s.ow + ox) * s.vecs + v;
    y[to] = make_uint4(best[0], best[1], best[2], best[3]);
    code[to] = make_uint2(__byte_perm(where[0], where[1], 0x6420), __byte_perm(where[2], where[3], 0x6420));
  }
}

// Pixels (2 by - pad + i, 2 bx - pad + j), i, j < 2: position (i + 2 m, j + 2 n) of window (by - m, bx - n), where that is inside of it.
__global__ void __launch_bounds__(POOL_THREADS)
max_pool_backward_kernel(const uint4* __restrict__ dy, const uint2* __restrict__ code, uint4* __restrict__ dx, const Pool s, int blocks_x, int blocks_y) {
  const int at = blockIdx.x * POOL_THREADS + threadIdx.x;
  if (at >= blocks_x * s.vecs) return;
  const int bx = at / s.vecs, v = at - bx * s.vecs;
  const long long image = blockIdx.z;
  for (int by = blockIdx.y; by < blocks_y; by += gridDim.y) {
    uint4 raw[4];
    uint2 c[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {   // window after window
      const int wy = by - 1 + q / 2, wx = bx - 1 + q % 2;
      const bool there = wy >= 0 && wy < s.oh && wx >= 0 && wx < s.ow;
      const long long from = ((image * s.oh + wy) * s.ow + wx) * s.vecs + v;
      raw[q] = there ? __ldg(dy + from) : make_uint4(0, 0, 0, 0);
      c[q] = there ? __ldg(code + from) : make_uint2(~0u, ~0u);
    }
#pragma unroll
    for (int i = 0; i < S; ++i) {
#pragma unroll
      for (int j = 0; j < S; ++j) {
        float sum[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) sum[k] = 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int py = i + S * (1 - q / 2), px = j + S * (1 - q % 2);
          if (py >= K || px >= K) continue;
          const uint32_t here = (py * K + px) * 0x01010101u, lo = __vcmpeq4(c[q].x, here), hi = __vcmpeq4(c[q].y, here);
          const uint32_t w[4] = {raw[q].x, raw[q].y, raw[q].z, raw[q].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t g = w[k] & __byte_perm(k < 2 ? lo : hi, 0, k & 1 ? 0x3322 : 0x1100);
            sum[2 * k] += __uint_as_float(g << 16);
            sum[2 * k + 1] += __uint_as_float(g & 0xffff0000u);
          }
        }
        uint4 out;
        __nv_bfloat162* half = reinterpret_cast<__nv_bfloat162*>(&out);
#pragma unroll
        for (int k = 0; k < 4; ++k) half[k] = __floats2bfloat162_rn(sum[2 * k], sum[2 * k + 1]);
        const int iy = by * S - s.pad + i, ix = bx * S - s.pad + j;
        if (iy >= 0 && iy < s.h && ix >= 0 && ix < s.w) dx[((image * s.h + iy) * s.w + ix) * s.vecs + v] = out;
      }
    }
  }
}

bool plain(const at::Tensor& t) {
  return t.is_cuda() && t.dim() == 4 && t.scalar_type() == at::kBFloat16 && t.is_contiguous(at::MemoryFormat::ChannelsLast) &&
         (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0;
}

Pool shape(const at::Tensor& x, int64_t pad) {
  TORCH_CHECK(plain(x) && x.numel() > 0 && x.size(1) % 8 == 0, "x must be a channels_last bf16 CUDA tensor with a multiple of 8 channels");
  TORCH_CHECK(pad == 0 || pad == 1, "padding of 0 or 1");
  TORCH_CHECK(x.size(0) <= 65535 && x.size(2) + 2 * pad >= K && x.size(3) + 2 * pad >= K && x.size(2) < (1LL << 30) &&
                  (x.size(3) + 2) * (x.size(1) / 8) < (1LL << 31) - POOL_THREADS, "size out of range");
  Pool s;
  s.vecs = static_cast<int>(x.size(1) / 8), s.h = static_cast<int>(x.size(2)), s.w = static_cast<int>(x.size(3)), s.pad = static_cast<int>(pad);
  s.oh = (s.h + 2 * s.pad - K) / S + 1, s.ow = (s.w + 2 * s.pad - K) / S + 1;
  return s;
}

dim3 pool_grid(int width, int height, int vecs, int64_t images) {
  return dim3(static_cast<unsigned>((static_cast<long long>(width) * vecs + POOL_THREADS - 1) / POOL_THREADS), std::min(height, 65535),
              static_cast<unsigned>(images));
}

// The backward pass in operations of PyTorch, on its indices: where it is differentiated again, by dy or (a derivative of zeros) by x, for a
// gradient with a tangent, that is a batch (is_grads_batched) or a subclass, or while operations are recorded.
bool needs_operations(const at::Tensor& dy, const at::Tensor& x) {
  return (at::GradMode::is_enabled() && (dy.requires_grad() || x.requires_grad())) || c10::impl::TorchDispatchModeTLS::any_modes_set() || !values_in_memory(dy) ||
         dy._fw_grad(0).defined();
}
at::Tensor backward_operations(const at::Tensor& dy, const at::Tensor& x, const at::Tensor& code, int64_t pad) {
  const auto place = code.view({dy.size(0), dy.size(2), dy.size(3), dy.size(1)}).permute({0, 3, 1, 2}).to(at::kLong);
  const auto options = place.options();
  const auto top = (at::arange(dy.size(2), options) * S - pad).view({-1, 1}), left = at::arange(dy.size(3), options) * S - pad;
  const auto indices = ((place.floor_divide(K) + top) * x.size(3) + place.remainder(K) + left).masked_fill(place == 0xff, 0);
  return at::max_pool2d_with_indices_backward(dy, x, {K, K}, {S, S}, {pad, pad}, {1, 1},
                                              false, indices.contiguous(at::MemoryFormat::ChannelsLast));
}

struct MaxPool : torch::autograd::Function<MaxPool> {
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& x, int64_t pad) {
    const Pool s = shape(x, pad);
    c10::cuda::CUDAGuard guard(x.get_device());
    auto y = at::empty({x.size(0), x.size(1), s.oh, s.ow}, x.options(), at::MemoryFormat::ChannelsLast);
    auto code = at::empty({y.numel()}, x.options().dtype(at::kByte));
    max_pool_forward_kernel<<<pool_grid(s.ow, s.oh, s.vecs, x.size(0)), POOL_THREADS, 0, at::cuda::getCurrentCUDAStream(x.get_device()).stream()>>>(
        reinterpret_cast<const uint4*>(x.data_ptr()), reinterpret_cast<uint4*>(y.data_ptr()), reinterpret_cast<uint2*>(code.data_ptr()), s);
    B200_CUDA_CHECK(cudaGetLastError());
    count_launch();
    ctx->save_for_backward({x, code});
    ctx->saved_data["pad"] = pad;
    return y;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const at::Tensor &x = saved[0], &code = saved[1];
    at::Tensor dy = grads[0];
    const int64_t pad = ctx->saved_data["pad"].toInt();
    c10::cuda::CUDAGuard guard(dy.get_device());
    if (needs_operations(dy, x)) return {backward_operations(dy, x, code, pad), at::Tensor()};
    dy = dy.contiguous(at::MemoryFormat::ChannelsLast);
    if ((reinterpret_cast<uintptr_t>(dy.data_ptr()) & 15) != 0) dy = dy.clone();   // a view into another gradient
    auto dx = at::empty(x.sizes(), dy.options(), at::MemoryFormat::ChannelsLast);
    const Pool s = shape(dx, pad);
    TORCH_CHECK(plain(dy) && dy.size(2) == s.oh && dy.size(3) == s.ow && code.is_cuda() && code.get_device() == dy.get_device() &&
                    code.is_contiguous() && code.numel() == dy.numel(), "dy must match the output");
    const int blocks_x = (s.w + s.pad + S - 1) / S, blocks_y = (s.h + s.pad + S - 1) / S;
    max_pool_backward_kernel<<<pool_grid(blocks_x, blocks_y, s.vecs, dx.size(0)), POOL_THREADS, 0,
                               at::cuda::getCurrentCUDAStream(dy.get_device()).stream()>>>(
        reinterpret_cast<const uint4*>(dy.data_ptr()), reinterpret_cast<const uint2*>(code.data_ptr()), reinterpret_cast<uint4*>(dx.data_ptr()), s, blocks_x, blocks_y);
    B200_CUDA_CHECK(cudaGetLastError());
    count_launch();
    return {dx, at::Tensor()};
  }
};

}  // namespace

at::Tensor max_pool_autograd(at::Tensor x, int64_t pad) { return MaxPool::apply(x, pad); }

}  // namespace b200
