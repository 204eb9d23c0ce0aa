// GroupNorm (+ optional SiLU) over channels-last activations, for the UNet that surrounds the
// INT8 linear layers: x is (B, H*W, C) with C contiguous (torch's channels_last NCHW tensor),
// groups are runs of C / groups adjacent channels, statistics run over H*W x (C / groups)
// elements per (sample, group).  torch's own GroupNorm kernel takes NCHW only, so a model whose
// convolutions run NHWC pays two layout copies around every normalisation.
//
// One launch: a cluster of up to eight CTAs owns one sample's slab of whole groups, each CTA a range of
// its rows.
//   pass 1  per-channel sum and sum of squares in fp32 registers, folded into per-group partials in a
//           fixed order and exchanged through distributed shared memory (no atomics: results do not
//           depend on timing)
//   pass 2  mean / rstd per group, then y = x * (rstd * gamma[c]) + (beta[c] - mean * rstd * gamma[c]) on
//           the rows read again (from L2, where pass 1 left them), rounded to the activation type; with
//           silu the rounded value goes through v / (1 + exp(-v)) and is rounded again (the two roundings
//           of GroupNorm followed by SiLU as separate ops)
// Bound by HBM at the large sizes (2 x 31.5 MB for 12 x 320 x 64 x 64: 9.7 us) beside two special-function
// instructions per element of the SiLU (7 us), by latency at the small ones.  Two grid-wide launches with
// partials in global memory took 27.1 us there and 11.5 us for 12 x 1280 x 8 x 8.
// Nothing here has a counterpart in the reference, whose UNet is stock PyTorch / diffusers.
#include "common.cuh"

namespace hy3d {
int device_sm_count();
namespace gnorm {
namespace {

constexpr int kMaxThreads = 384;
constexpr int kTargetThreads = 384;
constexpr int kMaxRanks = 8;          // portable cluster size

template <bool kBf16>
__device__ __forceinline__ float2 unpack2f(uint32_t w) {
  if (kBf16) return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <bool kBf16>
__device__ __forceinline__ void unpack8f(const uint4& v, float2 (&f)[4]) {
  f[0] = unpack2f<kBf16>(v.x);
  f[1] = unpack2f<kBf16>(v.y);
  f[2] = unpack2f<kBf16>(v.z);
  f[3] = unpack2f<kBf16>(v.w);
}

// x + add[b, c], rounded to the activation type as a separate broadcast add would have stored it.
template <bool kBf16>
__device__ __forceinline__ void add_round8(float2 (&f)[4], const float2 (&a)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 t = __fadd2_rn(f[j], a[j]);
    f[j] = unpack2f<kBf16>(pack2(t.x, t.y, kBf16 ? HY3D_BF16 : HY3D_F16));
  }
}

__device__ __forceinline__ float rcp_approx(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

__device__ __forceinline__ void cluster_sync_release() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Threads are laid out as (row lane ty, vector column tx): tx = tid % (slab / 8) owns 8 adjacent
// channels, ty = tid / (slab / 8) walks rows ty, ty + k, ...  blockDim.x = (slab / 8) * k.
// grid.x = S (the cluster: row ranges), grid.y = slabs, grid.z = samples.
template <bool kBf16, bool kAdd, bool kSilu>
__global__ void __launch_bounds__(kMaxThreads, 3)
groupnorm_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ add, int64_t HW, int C, int cpg,
                 int slab_groups, int rows_per_cta, const void* __restrict__ gamma, const void* __restrict__ beta,
                 int gb_dtype, float eps, uint16_t* __restrict__ y) {
  // [S][2 * slab_groups] group partials of every rank, then the fold's [k][2][slab] per-channel sums (the
  // first slice later holds every channel's scale and shift)
  extern __shared__ float smem[];
  const int slab = slab_groups * cpg;
  const int vec_cols = slab >> 3, row_vecs = C >> 3;
  const int k = blockDim.x / vec_cols;
  const int tx = threadIdx.x % vec_cols, ty = threadIdx.x / vec_cols;
  const int S = gridDim.x, rank = blockIdx.x, b = blockIdx.z;
  const int c0 = static_cast<int>(blockIdx.y) * slab + 8 * tx;      // this thread's first channel
  float* s_part = smem;
  float* s_acc = s_part + (S * 2 * slab_groups + 3) / 4 * 4;
  pdl_launch_dependents();
  if (S > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  pdl_wait();
  const int64_t r0 = static_cast<int64_t>(rank) * rows_per_cta;
  const int64_t r1 = r0 + rows_per_cta < HW ? r0 + rows_per_cta : HW;
  const int64_t base = static_cast<int64_t>(b) * HW * C + c0;
  const uint4* src = reinterpret_cast<const uint4*>(x + base);
  float2 av[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) av[j] = make_float2(0.0f, 0.0f);
  if (kAdd) unpack8f<kBf16>(__ldcs(reinterpret_cast<const uint4*>(add + static_cast<int64_t>(b) * C + c0)), av);

  float2 s2[4], q2[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) { s2[j] = make_float2(0.0f, 0.0f); q2[j] = make_float2(0.0f, 0.0f); }
  auto accumulate = [&](const uint4& v) {
    float2 f[4];
    unpack8f<kBf16>(v, f);
    if (kAdd) add_round8<kBf16>(f, av);
#pragma unroll
    for (int j = 0; j < 4; ++j) { s2[j] = __fadd2_rn(s2[j], f[j]); q2[j] = __ffma2_rn(f[j], f[j], q2[j]); }
  };
  const int64_t step = static_cast<int64_t>(k) * row_vecs, at0 = (r0 + ty) * row_vecs;
  int left = static_cast<int>((r1 - r0 - ty + k - 1) / k);          // rows of this thread (may be < 1)
  const uint4* in = src + at0;
  for (; left >= 4; left -= 4, in += 4 * step) {                    // four rows in flight per thread
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = in[u * step];
#pragma unroll
    for (int u = 0; u < 4; ++u) accumulate(v[u]);
  }
  for (; left > 0; --left, in += step) accumulate(*in);

  // Every row lane parks its sums in its own slice, channel c adds the k slices in order, group g its
  // channels in order; the group sums go to every rank of the cluster.
  float* mine = s_acc + static_cast<size_t>(ty) * 2 * slab + 8 * tx;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    *reinterpret_cast<float2*>(mine + 2 * j) = s2[j];
    *reinterpret_cast<float2*>(mine + slab + 2 * j) = q2[j];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < 2 * slab; c += blockDim.x) {
    float a = s_acc[c];
#pragma unroll 4
    for (int lane = 1; lane < k; ++lane) a += s_acc[static_cast<size_t>(lane) * 2 * slab + c];
    s_acc[c] = a;
  }
  if (S > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // the peers run
  __syncthreads();
  for (int g = threadIdx.x; g < 2 * slab_groups; g += blockDim.x) {   // sums, then sums of squares
    const float* p = s_acc + g * cpg;
    float a = 0.0f;
#pragma unroll 4
    for (int c = 0; c < cpg; ++c) a += p[c];
    const uint32_t at = smem_u32(s_part + rank * 2 * slab_groups + g);
    for (int peer = 0; peer < S; ++peer)
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(map_to_cta(at, static_cast<uint32_t>(peer))), "f"(a) : "memory");
  }
  __syncwarp();
  if (S > 1) cluster_sync_release(); else __syncthreads();
  // One thread per channel of the slab turns the partials into scale and shift.
  const float inv_n = 1.0f / (static_cast<float>(HW) * static_cast<float>(cpg));
  for (int c = threadIdx.x; c < slab; c += blockDim.x) {
    const int g = c / cpg;
    float a = 0.0f, q = 0.0f;
    for (int peer = 0; peer < S; ++peer) {
      a += s_part[peer * 2 * slab_groups + g];
      q += s_part[peer * 2 * slab_groups + slab_groups + g];
    }
    const float mean = a * inv_n;
    const float rstd = rsqrtf(fmaxf(fmaf(-mean, mean, q * inv_n), 0.0f) + eps);
    const int ch = static_cast<int>(blockIdx.y) * slab + c;
    const float ga = gamma ? load_scalar(gamma, gb_dtype, ch) : 1.0f;
    const float be = beta ? load_scalar(beta, gb_dtype, ch) : 0.0f;
    s_acc[c] = rstd * ga;
    s_acc[slab + c] = fmaf(-mean, rstd * ga, be);
  }
  __syncthreads();

  float2 sc[4], sh[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    sc[j] = *reinterpret_cast<const float2*>(s_acc + 8 * tx + 2 * j);
    sh[j] = *reinterpret_cast<const float2*>(s_acc + slab + 8 * tx + 2 * j);
  }
  uint4* dst = reinterpret_cast<uint4*>(y + base);
  auto transform = [&](const uint4& v) {
    float2 f[4];
    unpack8f<kBf16>(v, f);
    if (kAdd) add_round8<kBf16>(f, av);
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 t = __ffma2_rn(f[j], sc[j], sh[j]);
      if (kSilu) {
        t = unpack2f<kBf16>(pack2(t.x, t.y, kBf16 ? HY3D_BF16 : HY3D_F16));
        // t / (1 + 2^(-t log2 e)): exponential and reciprocal approximations whose error is far below half
        // a unit of the 16-bit result
        const float2 n = __fmul2_rn(t, make_float2(-1.4426950408889634f, -1.4426950408889634f));
        const float2 d = __fadd2_rn(make_float2(ex2_approx(n.x), ex2_approx(n.y)), make_float2(1.0f, 1.0f));
        t = __fmul2_rn(t, make_float2(rcp_approx(d.x), rcp_approx(d.y)));
      }
      w[j] = pack2(t.x, t.y, kBf16 ? HY3D_BF16 : HY3D_F16);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  };
  left = static_cast<int>((r1 - r0 - ty + k - 1) / k);
  in = src + at0;
  uint4* out = dst + at0;
  for (; left >= 4; left -= 4, in += 4 * step, out += 4 * step) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = __ldcs(in + u * step);
#pragma unroll
    for (int u = 0; u < 4; ++u) out[u * step] = transform(v[u]);
  }
  for (; left > 0; --left, in += step, out += step) *out = transform(__ldcs(in));
}

}  // namespace

// Nothing needs global scratch any more; callers of the C ABI still pass a workspace of this size.
int64_t workspace_floats(int64_t B, int64_t HW, int groups) {
  (void)HW;
  return B * groups * 2;
}

int groupnorm_nhwc(const void* x, const void* add, int x_dtype, int64_t B, int64_t HW, int64_t C, int groups,
                   const void* gamma, const void* beta, int gb_dtype, float eps, int silu,
                   void* y, float* workspace, cudaStream_t stream) {
  if (x_dtype != HY3D_F16 && x_dtype != HY3D_BF16) return HY3D_ERR_ARG;
  if ((gamma || beta) && (gb_dtype < HY3D_F16 || gb_dtype > HY3D_F32)) return HY3D_ERR_ARG;
  if (B < 0 || HW <= 0 || C <= 0 || groups <= 0 || (C & 7) || C % groups) return HY3D_ERR_SHAPE;
  if (C > 2560 || B > 65535 || HW > (1ll << 31)) return HY3D_ERR_SHAPE;
  if (B == 0) return HY3D_OK;
  if (!x || !y || !workspace) return HY3D_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(add)) & 15)
    return HY3D_ERR_SHAPE;
  const int cpg = static_cast<int>(C / groups);
  // Slab: the widest run of whole groups (a multiple of 8 channels, so that 16-byte vectors stay inside
  // it) that still gives two CTAs per SM with clusters of eight; narrower than 32 channels only where
  // nothing else divides, since a row of a slab is one contiguous piece.
  const int sms = device_sm_count() > 0 ? device_sm_count() : 148;
  int slab_groups = 0;
  for (int g = groups; g >= 1; --g) {
    if (groups % g || (g * cpg) % 8 || g * cpg > 2560) continue;
    if (slab_groups && g * cpg < 32) break;
    slab_groups = g;
    if (B * (groups / g) * kMaxRanks >= 2 * sms) break;
  }
  if (!slab_groups) return HY3D_ERR_SHAPE;
  const int slab = slab_groups * cpg, vec_cols = slab >> 3;
  // Rank count: up to eight, while every row lane keeps at least four rows.
  int k = kTargetThreads / vec_cols > 0 ? kTargetThreads / vec_cols : 1;
  int ranks = kMaxRanks;
  while (ranks > 1 && HW < static_cast<int64_t>(4) * k * ranks && HW < static_cast<int64_t>(32) * ranks) ranks >>= 1;
  const int64_t rows_per_cta = (HW + ranks - 1) / ranks;
  if (rows_per_cta < k) k = static_cast<int>(rows_per_cta);
  const size_t smem = (static_cast<size_t>(ranks * 2 * slab_groups + 3) + static_cast<size_t>(k) * 2 * slab) * sizeof(float);
  if (rows_per_cta > 0x7FFFFFFF || B > 65535 || groups / slab_groups > 65535) return HY3D_ERR_SHAPE;
  (void)workspace;

  using KernelFn = void (*)(const uint16_t*, const uint16_t*, int64_t, int, int, int, int, const void*, const void*, int,
                            float, uint16_t*);
  static const KernelFn kernels[2][2][2] = {
      {{groupnorm_kernel<false, false, false>, groupnorm_kernel<false, false, true>},
       {groupnorm_kernel<false, true, false>, groupnorm_kernel<false, true, true>}},
      {{groupnorm_kernel<true, false, false>, groupnorm_kernel<true, false, true>},
       {groupnorm_kernel<true, true, false>, groupnorm_kernel<true, true, true>}}};
  const KernelFn kernel = kernels[x_dtype == HY3D_BF16 ? 1 : 0][add ? 1 : 0][silu ? 1 : 0];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ranks), static_cast<unsigned>(groups / slab_groups), static_cast<unsigned>(B));
  cfg.blockDim = dim3(static_cast<unsigned>(vec_cols * k));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0] = pdl_attribute();
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(ranks);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t err = cudaLaunchKernelEx(
      &cfg, kernel, static_cast<const uint16_t*>(x), static_cast<const uint16_t*>(add), HW, static_cast<int>(C), cpg,
      slab_groups, static_cast<int>(rows_per_cta), gamma, beta, gb_dtype, eps, static_cast<uint16_t*>(y));
  if (err != cudaSuccess) {
    cudaGetLastError();
    return HY3D_ERR_CUDA;
  }
  return HY3D_OK;
}

}  // namespace gnorm
}  // namespace hy3d
