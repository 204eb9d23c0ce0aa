// Element-wise work of the UNet between its convolutions and INT8 layers, over channels-last activations of a
// 16-bit type: one pass over memory where separate ops took two or three, with the roundings those would have
// made, so the bits are the same.
//
//   add_bias    y = round(round(x + bx) + round(h + bh)): a residual sum whose two sides come from convolutions
//               that left their bias to it (torch adds a convolution's bias in a pass of its own, and not a
//               vectorised one: 19 us for 12 x 320 x 64 x 64).  Any of bx, h, bh may be absent.
//   concat      channels of a, then of b, per pixel
//   upsample2x  nearest-neighbour, twice the height and width
//
// All of them are bound by HBM: 16-byte vectors, several independent ones per thread in flight.
// Nothing here has a counterpart in the reference, whose UNet is stock PyTorch / diffusers.
#include "common.cuh"

namespace hy3d {
int device_sm_count();
namespace nhwc {
namespace {

constexpr int kThreads = 256;
constexpr int kUnroll = 4;      // vectors a thread has in flight

// A block takes kUnroll * kThreads adjacent vectors; the column of a vector (its place in the bias) comes from
// one 32-bit division per thread and additions from there on.
template <bool kBf16>
__global__ void __launch_bounds__(kThreads)
add_bias_kernel(const uint4* x, const uint4* __restrict__ bx, const uint4* h, const uint4* __restrict__ bh, uint4* y,
                int64_t total, int vec_cols) {          // y may be x or h: a thread has read its vectors before it writes
  pdl_launch_dependents();
  const int64_t first = static_cast<int64_t>(blockIdx.x) * (kUnroll * kThreads);
  int col = static_cast<int>((first + threadIdx.x) % vec_cols);
  const int step = kThreads % vec_cols;
  pdl_wait();
  uint4 vx[kUnroll], vh[kUnroll];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t at = first + u * kThreads + threadIdx.x;
    if (at < total) {
      vx[u] = __ldcs(x + at);
      if (h) vh[u] = __ldcs(h + at);
    }
  }
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t at = first + u * kThreads + threadIdx.x;
    if (at < total) {
      uint4 v = vx[u];
      if (bx) v = add8_16<kBf16>(v, __ldg(bx + col));
      if (h) v = add8_16<kBf16>(v, bh ? add8_16<kBf16>(vh[u], __ldg(bh + col)) : vh[u]);
      y[at] = v;
    }
    col += step;
    if (col >= vec_cols) col -= vec_cols;
  }
}

__global__ void __launch_bounds__(kThreads)
concat_kernel(const uint4* __restrict__ a, int va, const uint4* __restrict__ b, int vb, uint4* __restrict__ y, int64_t total) {
  pdl_launch_dependents();
  const int64_t first = static_cast<int64_t>(blockIdx.x) * (kUnroll * kThreads);
  const int vy = va + vb;
  int64_t row = (first + threadIdx.x) / vy;
  int col = static_cast<int>((first + threadIdx.x) - row * vy);
  const int step_row = kThreads / vy, step_col = kThreads - step_row * vy;
  pdl_wait();
  uint4 v[kUnroll];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t at = first + u * kThreads + threadIdx.x;
    if (at < total) v[u] = col < va ? __ldcs(a + row * va + col) : __ldcs(b + row * vb + (col - va));
    row += step_row;
    col += step_col;
    if (col >= vy) { col -= vy; ++row; }
  }
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t at = first + u * kThreads + threadIdx.x;
    if (at < total) y[at] = v[u];
  }
}

// One thread per input vector and kUnroll of them: read once, written to the four output pixels.
__global__ void __launch_bounds__(kThreads)
upsample2x_kernel(const uint4* __restrict__ x, uint4* __restrict__ y, int64_t total, int W, int vec_cols) {
  pdl_launch_dependents();
  const int64_t first = static_cast<int64_t>(blockIdx.x) * (kUnroll * kThreads);
  pdl_wait();
  uint4 v[kUnroll];
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t at = first + u * kThreads + threadIdx.x;
    if (at < total) v[u] = __ldcs(x + at);
  }
#pragma unroll
  for (int u = 0; u < kUnroll; ++u) {
    const int64_t at = first + u * kThreads + threadIdx.x;
    if (at >= total) break;
    const int64_t pixel = at / vec_cols, line = pixel / W;              // line = sample * H + row
    const int c = static_cast<int>(at - pixel * vec_cols), col = static_cast<int>(pixel - line * W);
    uint4* out = y + (4 * line * W + 2 * col) * vec_cols + c;
    out[0] = v[u];
    out[vec_cols] = v[u];
    out[2 * static_cast<int64_t>(W) * vec_cols] = v[u];
    out[(2 * static_cast<int64_t>(W) + 1) * vec_cols] = v[u];
  }
}

template <typename... Params, typename... Args>
int launch(void (*kernel)(Params...), int64_t vectors, cudaStream_t stream, Args... args) {
  const int64_t blocks = (vectors + kUnroll * kThreads - 1) / (kUnroll * kThreads);
  if (blocks > 0x7FFFFFFF) return HY3D_ERR_SHAPE;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(kThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2] = {pdl_attribute(), carveout_attribute(2048 / kThreads, 0)};
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...) != cudaSuccess) {
    cudaGetLastError();
    return HY3D_ERR_CUDA;
  }
  return HY3D_OK;
}

bool misaligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) != 0; }

}  // namespace

int add_bias(const void* x, const void* bias_x, const void* h, const void* bias_h, int dtype, void* y, int64_t rows,
             int64_t C, cudaStream_t stream) {
  if (dtype != HY3D_F16 && dtype != HY3D_BF16) return HY3D_ERR_ARG;
  if (rows < 0 || C <= 0 || (C & 7) || C > (1 << 24)) return HY3D_ERR_SHAPE;
  if (rows == 0) return HY3D_OK;
  if (!x || !y || (bias_h && !h)) return HY3D_ERR_ARG;
  if (misaligned(x) || misaligned(y) || misaligned(h) || misaligned(bias_x) || misaligned(bias_h)) return HY3D_ERR_SHAPE;
  const int vec_cols = static_cast<int>(C >> 3);
  const int64_t total = rows * vec_cols;
  auto v = [](const void* p) { return static_cast<const uint4*>(p); };
  return dtype == HY3D_BF16 ? launch(add_bias_kernel<true>, total, stream, v(x), v(bias_x), v(h), v(bias_h), static_cast<uint4*>(y), total, vec_cols)
                            : launch(add_bias_kernel<false>, total, stream, v(x), v(bias_x), v(h), v(bias_h), static_cast<uint4*>(y), total, vec_cols);
}

int concat(const void* a, int64_t Ca, const void* b, int64_t Cb, void* y, int64_t rows, cudaStream_t stream) {
  if (rows < 0 || Ca <= 0 || Cb <= 0 || (Ca & 7) || (Cb & 7) || Ca + Cb > (1 << 24)) return HY3D_ERR_SHAPE;
  if (rows == 0) return HY3D_OK;
  if (!a || !b || !y) return HY3D_ERR_ARG;
  if (misaligned(a) || misaligned(b) || misaligned(y)) return HY3D_ERR_SHAPE;
  const int64_t total = rows * ((Ca + Cb) >> 3);
  return launch(concat_kernel, total, stream, static_cast<const uint4*>(a), static_cast<int>(Ca >> 3), static_cast<const uint4*>(b),
                static_cast<int>(Cb >> 3), static_cast<uint4*>(y), total);
}

int upsample2x(const void* x, void* y, int64_t B, int64_t H, int64_t W, int64_t C, cudaStream_t stream) {
  if (B < 0 || H <= 0 || W <= 0 || C <= 0 || (C & 7) || W > (1 << 24) || C > (1 << 24)) return HY3D_ERR_SHAPE;
  if (B == 0) return HY3D_OK;
  if (!x || !y) return HY3D_ERR_ARG;
  if (misaligned(x) || misaligned(y)) return HY3D_ERR_SHAPE;
  const int vec_cols = static_cast<int>(C >> 3);
  const int64_t total = B * H * W * vec_cols;
  return launch(upsample2x_kernel, total, stream, static_cast<const uint4*>(x), static_cast<uint4*>(y), total, static_cast<int>(W), vec_cols);
}

}  // namespace nhwc
}  // namespace hy3d
