// Per-token absmax activation quantiser and the stand-alone dequant+bias epilogue kernel.
//
// Quantiser arithmetic (bit-exact contract, checked against the CPU oracle):
//     amax  = max_k |x[m,k]|                       (fp32)
//     scale = max(amax, 1e-8f) / 127.0f            (IEEE division)
//     q     = clamp(rint(x / scale), -128, 127)    (IEEE division, round-half-even)
// The row is read ONCE with 16-byte loads and kept in registers between the absmax reduction and the
// rounding pass, so the kernel moves 2*K + K + 4/M bytes per row.
//
// The rounding costs one fused multiply-add per value, fma(x, mul, 1.5 * 2^23), with a multiplier that is
// 1 / scale nudged by two units in the last place.  Why that is exact: x and amax carry at most 11 significant
// bits, and x / amax = (2 k + 1) / 254 needs 127 to divide 2 k + 1 or the significand of amax (127 is prime).
// So unless it divides the latter -- then scale * 127 == amax exactly and several ties exist -- the only tie is
// x = amax / 2, between 63 and 64; every other quotient is at least 2.4e-4 away from one, far more than the
// nudge (6e-5) and scale's own rounding move it.  At that tie the IEEE quotient of the rounded scale is 63.5 or
// above (code 64, the even one) or below it (63); amax / scale, its double, tells which, and the nudge goes the
// same way.  Rows whose scale is exact refine their quotient instead: q0 = x * rcp(scale), one residual
// correction q = fma(fma(-q0, scale, x), rcp, q0).  A device-side enumeration of every pair of 16-bit patterns
// (amax, x) with |x| <= amax -- 1.0e9 pairs for fp16, 1.07e9 for bf16, i.e. every input this kernel can see --
// found rint(q) == rint(__fdiv_rn(x, scale)) for all of them.
#include "common.cuh"

namespace hy3d {
int device_sm_count();
namespace quant {
namespace {

int sm_count() { return device_sm_count() > 0 ? device_sm_count() : 148; }

constexpr int kQuantThreads = 256;
struct True { static constexpr bool value = true; };
struct False { static constexpr bool value = false; };

template <bool kBf16>
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (kBf16) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    } else {
      __half2 h = *reinterpret_cast<const __half2*>(&w[i]);
      float2 t = __half22float2(h);
      f[2 * i] = t.x;
      f[2 * i + 1] = t.y;
    }
  }
}

// Folds the eight 16-bit values of a 16-byte vector into a running packed maximum of |x| (two lanes per
// register), without widening them first.  The signs of the result mean nothing.
template <bool kBf16>
__device__ __forceinline__ void absmax8(const uint4& v, uint32_t& acc) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (kBf16) asm("max.xorsign.abs.bf16x2 %0, %0, %1;" : "+r"(acc) : "r"(w[i]));
    else asm("max.xorsign.abs.f16x2 %0, %0, %1;" : "+r"(acc) : "r"(w[i]));
  }
}
template <bool kBf16>
__device__ __forceinline__ float absmax_to_float(uint32_t acc) {
  acc &= 0x7FFF7FFFu;
  if (kBf16) {
    return fmaxf(__uint_as_float(acc << 16), __uint_as_float(acc & 0xFFFF0000u));
  }
  const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&acc));
  return fmaxf(t.x, t.y);
}

// What a row's values are quantised with (see the file header).
struct RowQuant {
  float scale, mul, inv;
  bool exact;      // scale * 127 == amax: refine the quotients
};
__device__ __forceinline__ RowQuant row_quant(float amax) {
  RowQuant r;
  const float a = fmaxf(amax, 1e-8f);
  r.scale = __fdiv_rn(a, 127.0f);
  r.inv = __frcp_rn(r.scale);
  // The division's residual a - 127 scale is representable, so its sign and zero are the true ones; the IEEE
  // quotient a / scale is 127 or more from half a unit in the last place (2^-18) below it on.
  const float rest = fmaf(r.scale, -127.0f, a);
  r.exact = rest == 0.0f;
  r.mul = __int_as_float(__float_as_int(r.inv) + (fmaf(r.scale, 3.814697265625e-6f, rest) >= 0.0f ? 2 : -2));
  return r;
}

// Quantises eight values to eight int8 codes (two words).  Float <-> int conversion instructions run at half
// the FMA rate or less, so the rounding uses the 1.5 * 2^23 trick: adding that constant rounds |t| < 2^22 to
// the nearest integer (ties to even, the FPU's own rounding) and leaves the two's-complement code in the low
// mantissa byte, which a byte permute then gathers.  No clamp is needed: scale = max|x| / 127 bounds
// |x / scale| by 127 (+ one rounding).  Packed fp32x2 instructions: two IEEE operations per issue slot.
__device__ __forceinline__ float2 fast_code2(float2 x, float mul) {
  return __ffma2_rn(x, make_float2(mul, mul), make_float2(12582912.0f, 12582912.0f));
}
__device__ __forceinline__ float2 refined_code2(float2 x, float scale, float inv) {
  const float2 inv2 = make_float2(inv, inv), nscale2 = make_float2(-scale, -scale);
  const float2 q0 = __fmul2_rn(x, inv2);
  const float2 r = __ffma2_rn(q0, nscale2, x);
  const float2 q = __ffma2_rn(r, inv2, q0);
  return __fadd2_rn(q, make_float2(12582912.0f, 12582912.0f));
}
template <bool kExact>
__device__ __forceinline__ uint2 quant8(const float (&f)[8], const RowQuant& r) {
  uint32_t b[8];
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    const float2 x = make_float2(f[j], f[j + 1]);
    const float2 t = kExact ? refined_code2(x, r.scale, r.inv) : fast_code2(x, r.mul);
    b[j] = __float_as_uint(t.x);
    b[j + 1] = __float_as_uint(t.y);
  }
  const uint32_t p01 = __byte_perm(b[0], b[1], 0x0040), p23 = __byte_perm(b[2], b[3], 0x0040);
  const uint32_t p45 = __byte_perm(b[4], b[5], 0x0040), p67 = __byte_perm(b[6], b[7], 0x0040);
  return make_uint2(__byte_perm(p01, p23, 0x5410), __byte_perm(p45, p67, 0x5410));
}
__device__ __forceinline__ uint2 quant8(const float (&f)[8], const RowQuant& r) {
  return r.exact ? quant8<true>(f, r) : quant8<false>(f, r);
}

// 2^lg threads cooperate on one row; each holds up to kMaxV 16-byte vectors.  A block of 256 threads covers
// 256 >> lg rows; threads past the last row repeat it (same values to the same places).  kFull: every thread
// has exactly kMaxV vectors.  Bound by HBM reads (the codes stay in L2 for the GEMM) and by issue slots:
// about 35 instructions per 8 values.
// kAdd: the rows are x + add, rounded to the 16-bit type and not stored.
template <bool kBf16, int kMaxV, bool kFull, bool kAdd>
__global__ void __launch_bounds__(kQuantThreads, kAdd ? 3 : kMaxV <= 6 ? 5 : 4)
quantize_rows_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ add, int64_t ldx, int8_t* __restrict__ q,
                     float* __restrict__ scale_out, int64_t M, int K, int lg) {
  __shared__ float s_part[kQuantThreads / 32];
  pdl_launch_dependents();
  const int tid = threadIdx.x, G = 1 << lg;
  const int sub = tid & (G - 1);  // position within the row group
  int64_t row = static_cast<int64_t>(blockIdx.x) * (kQuantThreads >> lg) + (tid >> lg);
  if (row >= M) row = M - 1;
  const int nvec = K >> 3;
  const uint4* src = reinterpret_cast<const uint4*>(x + row * ldx) + sub;
  uint2* dst = reinterpret_cast<uint2*>(q + row * static_cast<int64_t>(K)) + sub;
  pdl_wait();   // x comes from the previous kernel in the stream

  uint4 v[kMaxV];
#pragma unroll
  for (int i = 0; i < kMaxV; ++i)
    v[i] = kFull || sub + i * G < nvec ? __ldcs(src + i * G) : make_uint4(0, 0, 0, 0);
  if (kAdd) {
    const uint4* other = reinterpret_cast<const uint4*>(add + row * ldx) + sub;
    uint4 w[kMaxV];
#pragma unroll
    for (int i = 0; i < kMaxV; ++i)
      w[i] = kFull || sub + i * G < nvec ? __ldcs(other + i * G) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int i = 0; i < kMaxV; ++i) v[i] = add8_16<kBf16>(v[i], w[i]);
  }
  uint32_t amax2 = 0;
#pragma unroll
  for (int i = 0; i < kMaxV; ++i) absmax8<kBf16>(v[i], amax2);
  float amax = absmax_to_float<kBf16>(amax2);
  // Reduce over the threads of the row.
  for (int off = (G < 32 ? G : 32) >> 1; off > 0; off >>= 1)
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  if (G > 32) {
    const int warp = tid >> 5;
    if ((tid & 31) == 0) s_part[warp] = amax;
    __syncthreads();
    const int warps_per_row = G >> 5;
    const int first = warp & ~(warps_per_row - 1);
    amax = s_part[first];
    for (int i = 1; i < warps_per_row; ++i) amax = fmaxf(amax, s_part[first + i]);
  }
  const RowQuant rq = row_quant(amax);
  if (sub == 0) scale_out[row] = rq.scale;
  auto write = [&](auto exact) {
#pragma unroll
    for (int i = 0; i < kMaxV; ++i) {
      if (kFull || sub + i * G < nvec) {
        float f[8];
        unpack8<kBf16>(v[i], f);
        dst[i * G] = quant8<decltype(exact)::value>(f, rq);
      }
    }
  };
  if (rq.exact) write(True{}); else write(False{});
}

template <bool kBf16>
int launch_quantize(const void* x, const void* add, int64_t M, int64_t K, int64_t ldx, int8_t* q, float* scale, bool l1,
                    cudaStream_t stream) {
  const int nvec = static_cast<int>(K >> 3);
  // Power-of-two group size and vectors per thread (<= 10) that cover the row with the fewest idle slots;
  // among equals the fewest threads per row, since the row's reductions and divisions are repeated by every
  // warp that holds a part of it -- unless the rows are too few to fill the chip that way.
  int lg = -1, maxv = 0;
  int64_t best = INT64_MAX;
  const int64_t fill = static_cast<int64_t>(sm_count()) * 4 * kQuantThreads;
  for (int l = 0; l <= 8; ++l) {
    const int64_t g = int64_t{1} << l;
    const int64_t v = (nvec + g - 1) / g;
    if (v > 10) continue;
    const int64_t idle = (g * v - nvec) * 64 / nvec;
    const int64_t few = M * g < fill && l < 5 ? fill / (M * g + 1) : 0;     // a warp per row at most
    const int64_t score = idle * 8 + few * 8 + l + (l > 5 ? 4 : 0);
    if (score < best) { best = score; lg = l; maxv = static_cast<int>(v); }
  }
  if (lg < 0) return HY3D_ERR_SHAPE;
  const int rows_per_block = kQuantThreads >> lg;
  const int64_t blocks = (M + rows_per_block - 1) / rows_per_block;
  if (blocks > 0x7FFFFFFF) return HY3D_ERR_SHAPE;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(kQuantThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2] = {pdl_attribute(), carveout_attribute(2048 / kQuantThreads, 32)};
  cfg.attrs = attr;
  cfg.numAttrs = l1 ? 2 : 1;
  using KernelFn = void (*)(const uint16_t*, const uint16_t*, int64_t, int8_t*, float*, int64_t, int, int);
#define HY3D_Q(V)                                                                                      \
  {{quantize_rows_kernel<kBf16, V, false, false>, quantize_rows_kernel<kBf16, V, true, false>},        \
   {quantize_rows_kernel<kBf16, V, false, true>, quantize_rows_kernel<kBf16, V, true, true>}}
  static const KernelFn kernels[10][2][2] = {HY3D_Q(1), HY3D_Q(2), HY3D_Q(3), HY3D_Q(4), HY3D_Q(5),
                                          HY3D_Q(6), HY3D_Q(7), HY3D_Q(8), HY3D_Q(9), HY3D_Q(10)};
#undef HY3D_Q
  const KernelFn kernel = kernels[maxv - 1][add ? 1 : 0][(maxv << lg) == nvec ? 1 : 0];
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, reinterpret_cast<const uint16_t*>(x),
                                             reinterpret_cast<const uint16_t*>(add), ldx, q, scale, M,
                                             static_cast<int>(K), lg);
  if (err != cudaSuccess) {
    cudaGetLastError();
    return HY3D_ERR_CUDA;
  }
  return HY3D_OK;
}

// LayerNorm fused with the per-token quantiser: the row is normalised in registers, rounded to
// the 16-bit activation type exactly as a stand-alone LayerNorm would store it, and those
// rounded values are quantised with the arithmetic above -- so the codes and scales equal
// quantize_rows(LayerNorm(x)) bit for bit while the normalised activations never go to memory
// (x is read once: 2*K bytes in, K + 4 bytes out per row, instead of 2K + 2K for the LayerNorm
// and 2K + K for the quantiser).  Arithmetic, all fp32, fixed reduction order:
//     mean = sum(x) / K;  var = sum((x - mean)^2) / K;  rstd = 1 / sqrt(var + eps)  (IEEE)
//     y    = round16( fma((x - mean) * rstd, gamma, beta) )
// 2^lg <= 32 lanes share a row (shuffle reductions), each with up to kMaxV vectors; gamma / beta are staged
// once per block in shared memory as fp32 and the block walks rows with a grid-stride loop, the next row's
// vectors requested before the current row is worked on.  Issue-bound.  Everything that can be is decided at
// compile time (kFull: no lane has a vector too few; kOut 1: the normalised row is stored too; kOut 2: the rows
// are x + add, rounded to the 16-bit type, and that sum is stored -- a transformer block's residual stream).
__host__ __device__ constexpr int ln_blocks(int maxv, int out) { return maxv <= 2 ? 4 : maxv <= 5 && out < 2 ? 3 : 2; }
template <bool kBf16, int kMaxV, bool kFull, int kOut>
__global__ void __launch_bounds__(kQuantThreads, ln_blocks(kMaxV, kOut))
layernorm_quantize_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ add, int64_t ldx, const void* __restrict__ gamma,
                          const void* __restrict__ beta, int gb_dtype, float eps,
                          int8_t* __restrict__ q, float* __restrict__ scale_out,
                          uint16_t* __restrict__ y_out, int64_t M, int K, int lg) {
  extern __shared__ float s_gb[];            // gamma and beta as fp32, 2 * K floats in planes
  pdl_launch_dependents();
  // Four planes of K/8 float4 each: [gamma 0-3 | gamma 4-7 | beta 0-3 | beta 4-7] of every
  // 8-element vector, so that the 16-byte loads of neighbouring lanes (neighbouring vectors)
  // are contiguous and conflict-free.
  const int plane = (K >> 3) * 4;
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const int at = ((k >> 2) & 1) * plane + (k >> 3) * 4 + (k & 3);
    s_gb[at] = gamma ? load_scalar(gamma, gb_dtype, k) : 1.0f;
    s_gb[2 * plane + at] = beta ? load_scalar(beta, gb_dtype, k) : 0.0f;
  }
  const int tid = threadIdx.x, G = 1 << lg;
  const int sub = tid & (G - 1);
  const int nvec = K >> 3;
  const float inv_k = 1.0f / static_cast<float>(K);
  const float* gb = s_gb + 4 * sub;
  const int rows_per_block = kQuantThreads >> lg;
  const int64_t row_step = static_cast<int64_t>(gridDim.x) * rows_per_block;
  int64_t row = static_cast<int64_t>(blockIdx.x) * rows_per_block + (tid >> lg);
  // The trip count is the block's: a thread past the last row repeats that row (same values, same places).
  const int trips = static_cast<int>((M - static_cast<int64_t>(blockIdx.x) * rows_per_block + row_step - 1) / row_step);
  pdl_wait();   // x comes from the previous kernel in the stream; gamma / beta are parameters
  __syncthreads();
  uint4 vn[kMaxV], an[kOut == 2 ? kMaxV : 1];
  auto fetch = [&](int64_t r) {
    const int64_t off = (r < M ? r : M - 1) * ldx;
    const uint4* src = reinterpret_cast<const uint4*>(x + off) + sub;
    if (kOut == 2) {
      const uint4* other = reinterpret_cast<const uint4*>(add + off) + sub;
#pragma unroll
      for (int i = 0; i < kMaxV; ++i)
        an[kOut == 2 ? i : 0] = kFull || sub + i * G < nvec ? __ldcs(other + i * G) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int i = 0; i < kMaxV; ++i)
      vn[i] = kFull || sub + i * G < nvec ? __ldcs(src + i * G) : make_uint4(0, 0, 0, 0);
  };
  fetch(row);
  for (int trip = 0; trip < trips; ++trip, row += row_step) {
    const int64_t at_row = row < M ? row : M - 1;
    // The row lives in registers as pairs; every step below is a packed fp32x2 instruction
    // (two IEEE single-precision operations per issue slot).
    float2 f[kMaxV][4];
    float2 sum2 = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < kMaxV; ++i) {
      float t[8];
      if (kOut == 2) {
        vn[i] = add8_16<kBf16>(vn[i], an[kOut == 2 ? i : 0]);
        if (kFull || sub + i * G < nvec)
          (reinterpret_cast<uint4*>(y_out + at_row * static_cast<int64_t>(K)) + sub)[i * G] = vn[i];
      }
      unpack8<kBf16>(vn[i], t);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        f[i][j] = make_float2(t[2 * j], t[2 * j + 1]);
        sum2 = __fadd2_rn(sum2, f[i][j]);
      }
    }
    if (trip + 1 < trips) fetch(row + row_step);
    float sum = sum2.x + sum2.y;
    for (int off = G >> 1; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const float mean = sum * inv_k;
    const float2 nmean2 = make_float2(-mean, -mean);
    float2 ss2 = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < kMaxV; ++i) {
      if (kFull || sub + i * G < nvec) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          f[i][j] = __fadd2_rn(f[i][j], nmean2);          // centred from here on
          ss2 = __ffma2_rn(f[i][j], f[i][j], ss2);
        }
      }
    }
    float ss = ss2.x + ss2.y;
    for (int off = G >> 1; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
    const float rstd = __frcp_rn(__fsqrt_rn(fmaf(ss, inv_k, eps)));
    const float2 rstd2 = make_float2(rstd, rstd);
    // normalise, round to the activation type, keep the rounded values for the quantiser
    uint32_t amax2 = 0;
    uint4 yv[kMaxV];
#pragma unroll
    for (int i = 0; i < kMaxV; ++i) {
      yv[i] = make_uint4(0, 0, 0, 0);
      if (kFull || sub + i * G < nvec) {
        const float* g = gb + 4 * i * G;
        const float4 g0 = *reinterpret_cast<const float4*>(g);
        const float4 g1 = *reinterpret_cast<const float4*>(g + plane);
        const float4 b0 = *reinterpret_cast<const float4*>(g + 2 * plane);
        const float4 b1 = *reinterpret_cast<const float4*>(g + 3 * plane);
        const float2 gg[4] = {make_float2(g0.x, g0.y), make_float2(g0.z, g0.w),
                              make_float2(g1.x, g1.y), make_float2(g1.z, g1.w)};
        const float2 bb[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w),
                              make_float2(b1.x, b1.y), make_float2(b1.z, b1.w)};
        uint32_t w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 y = __ffma2_rn(__fmul2_rn(f[i][j], rstd2), gg[j], bb[j]);
          w[j] = pack2(y.x, y.y, kBf16 ? HY3D_BF16 : HY3D_F16);
        }
        yv[i] = make_uint4(w[0], w[1], w[2], w[3]);
        absmax8<kBf16>(yv[i], amax2);
      }
    }
    float amax = absmax_to_float<kBf16>(amax2);
    for (int off = G >> 1; off > 0; off >>= 1)
      amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    const RowQuant rq = row_quant(amax);
    if (sub == 0) scale_out[at_row] = rq.scale;
    uint2* dst = reinterpret_cast<uint2*>(q + at_row * static_cast<int64_t>(K)) + sub;
    auto write = [&](auto exact) {
#pragma unroll
      for (int i = 0; i < kMaxV; ++i) {
        if (kFull || sub + i * G < nvec) {
          float fy[8];
          unpack8<kBf16>(yv[i], fy);
          dst[i * G] = quant8<decltype(exact)::value>(fy, rq);
        }
      }
    };
    if (rq.exact) write(True{}); else write(False{});
    if (kOut == 1) {
      uint4* ydst = reinterpret_cast<uint4*>(y_out + at_row * static_cast<int64_t>(K)) + sub;
#pragma unroll
      for (int i = 0; i < kMaxV; ++i)
        if (kFull || sub + i * G < nvec) ydst[i * G] = yv[i];
    }
  }
}

template <bool kBf16>
int launch_layernorm_quantize(const void* x, const void* add, int64_t M, int64_t K, int64_t ldx, const void* gamma,
                              const void* beta, int gb_dtype, float eps, int8_t* q, float* scale,
                              void* y_out, cudaStream_t stream) {
  const int nvec = static_cast<int>(K >> 3);
  // lanes per row: the power of two (<= 32) that leaves at most 5 vectors per lane.  (The number of lanes
  // also fixes the order of the row's sums, hence their last bits.)
  int lg = 0;
  while (lg < 5 && ((nvec + (1 << lg) - 1) >> lg) > 5) ++lg;
  const int maxv = (nvec + (1 << lg) - 1) >> lg;
  if (maxv > 8) return HY3D_ERR_SHAPE;
  const int rows_per_block = kQuantThreads >> lg;
  const int64_t batches = (M + rows_per_block - 1) / rows_per_block;
  using KernelFn = void (*)(const uint16_t*, const uint16_t*, int64_t, const void*, const void*, int, float, int8_t*,
                            float*, uint16_t*, int64_t, int, int);
#define HY3D_LNQ(V)                                                                                          \
  {{layernorm_quantize_kernel<kBf16, V, false, 0>, layernorm_quantize_kernel<kBf16, V, false, 1>,            \
    layernorm_quantize_kernel<kBf16, V, false, 2>},                                                          \
   {layernorm_quantize_kernel<kBf16, V, true, 0>, layernorm_quantize_kernel<kBf16, V, true, 1>,              \
    layernorm_quantize_kernel<kBf16, V, true, 2>}}
  static const KernelFn kernels[6][2][3] = {HY3D_LNQ(1), HY3D_LNQ(2), HY3D_LNQ(3), HY3D_LNQ(4), HY3D_LNQ(5), HY3D_LNQ(8)};
#undef HY3D_LNQ
  const int v = maxv <= 5 ? maxv : 8, out = add ? 2 : y_out ? 1 : 0;
  const KernelFn kernel = kernels[maxv <= 5 ? maxv - 1 : 5][(v << lg) == nvec ? 1 : 0][out];
  // One full wave of resident blocks: the first few take a row batch more.  As few blocks as take no more trips left SMs
  // a block short: 49152 x 320 12.4 us, as here 11.5; 5000 x 2048 10.3 and 9.1, with the GEMM behind it (-> 512) 20.2 and 18.0.
  const int64_t wave = static_cast<int64_t>(sm_count()) * ln_blocks(v, out);
  const int64_t blocks = batches < wave ? batches : wave;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(blocks));
  cfg.blockDim = dim3(kQuantThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(2 * K) * sizeof(float);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2] = {pdl_attribute(), carveout_attribute(ln_blocks(v, out), 8 * K)};
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, reinterpret_cast<const uint16_t*>(x),
                                             reinterpret_cast<const uint16_t*>(add), ldx, gamma, beta, gb_dtype, eps, q, scale, reinterpret_cast<uint16_t*>(y_out), M, static_cast<int>(K), lg);
  if (err != cudaSuccess) {
    cudaGetLastError();
    return HY3D_ERR_CUDA;
  }
  return HY3D_OK;
}

// Enumeration behind the quantiser's exactness claim: block a takes the 16-bit pattern a as
// amax, its threads walk all 65536 patterns x with |x| <= amax and compare the code the
// quantiser's arithmetic produces with (int8) rint(x / scale) computed by IEEE division.
__device__ unsigned long long g_enum_counts[2];   // [0] pairs checked, [1] codes that differ

template <bool kBf16>
__global__ void __launch_bounds__(256) quotient_enum_kernel() {
  const uint32_t a_bits = blockIdx.x;
  const float amax = kBf16 ? __uint_as_float(a_bits << 16)
                           : __half2float(__ushort_as_half(static_cast<unsigned short>(a_bits)));
  if (!(amax == amax) || isinf(amax)) return;
  const RowQuant rq = row_quant(amax);
  unsigned long long pairs = 0, bad = 0;
  // Two patterns per step, through the packed arithmetic the quantiser kernels run.
  for (uint32_t xb = 2 * threadIdx.x; xb < 65536u; xb += 2 * blockDim.x) {
    float x[2];
#pragma unroll
    for (int h = 0; h < 2; ++h)
      x[h] = kBf16 ? __uint_as_float((xb + h) << 16)
                   : __half2float(__ushort_as_half(static_cast<unsigned short>(xb + h)));
    const float2 t = rq.exact ? refined_code2(make_float2(x[0], x[1]), rq.scale, rq.inv) : fast_code2(make_float2(x[0], x[1]), rq.mul);
    const uint32_t b[2] = {__float_as_uint(t.x), __float_as_uint(t.y)};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (!(fabsf(x[h]) <= amax)) continue;
      const int code = static_cast<int>(static_cast<signed char>(b[h] & 0xFFu));
      const int ref = static_cast<int>(rintf(__fdiv_rn(x[h], rq.scale)));
      ++pairs;
      if (code != ref) ++bad;
    }
  }
  atomicAdd(&g_enum_counts[0], pairs);
  atomicAdd(&g_enum_counts[1], bad);
}

// out[m,n] = acc[m,n] * (act_scale[m] * w_scale[n]) + bias[n]; 8 columns per thread.
__global__ void __launch_bounds__(256)
dequant_bias_kernel(const int32_t* __restrict__ acc, const float* __restrict__ act_scale,
                    const void* __restrict__ w_scale, int ws_dtype, const void* __restrict__ bias,
                    int bias_dtype, void* __restrict__ out, int out_dtype, int64_t M, int64_t N) {
  const int64_t nchunk = N >> 3;
  const int64_t total = M * nchunk;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t m = i / nchunk;
    const int64_t n0 = (i - m * nchunk) << 3;
    const int4* src = reinterpret_cast<const int4*>(acc + m * N + n0);
    const int4 a0 = src[0], a1 = src[1];
    const int a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    const float as = act_scale[m];
    float y[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float s = as * load_scalar(w_scale, ws_dtype, n0 + j);
      const float b = bias ? load_scalar(bias, bias_dtype, n0 + j) : 0.0f;
      y[j] = fmaf(static_cast<float>(a[j]), s, b);
    }
    uint4 o;
    o.x = pack2(y[0], y[1], out_dtype);
    o.y = pack2(y[2], y[3], out_dtype);
    o.z = pack2(y[4], y[5], out_dtype);
    o.w = pack2(y[6], y[7], out_dtype);
    *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(out) + m * N + n0) = o;
  }
}

}  // namespace

// Elements from which the quantiser asks for L1.  It gains by it where the loads in flight bound it, and the GEMM behind
// it may start later, since the SMs change their split in between.  Dense layers, time with it over time without, inputs
// from HBM / from L2: 0.6 to 1 million elements 0.99 / 1.00, 2 to 4 million 0.97 / 0.99, from 8 million on 0.94 / 0.95;
// fewer 1.00, up to 1.05.  (2:4-sparse layers: sparse_l1_elements.)
constexpr double kL1Elements = 6e5;

int quantize_rows(const void* x, const void* add, int x_dtype, int64_t M, int64_t K, int64_t ldx, int8_t* q,
                  float* scale, cudaStream_t stream, double l1_elements = kL1Elements) {
  if (x_dtype != HY3D_F16 && x_dtype != HY3D_BF16) return HY3D_ERR_ARG;
  if (M < 0 || K <= 0 || (K & 7) || K > 16384 || ldx < K || (ldx & 7)) return HY3D_ERR_SHAPE;
  if (M == 0) return HY3D_OK;
  if (!x || !q || !scale) return HY3D_ERR_ARG;
  if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(add)) & 15) || (reinterpret_cast<uintptr_t>(q) & 7))
    return HY3D_ERR_SHAPE;
  if (M == 0) return HY3D_OK;
  const bool l1 = static_cast<double>(M) * static_cast<double>(K) >= l1_elements;
  return x_dtype == HY3D_BF16 ? launch_quantize<true>(x, add, M, K, ldx, q, scale, l1, stream)
                              : launch_quantize<false>(x, add, M, K, ldx, q, scale, l1, stream);
}

int layernorm_quantize(const void* x, const void* add, int x_dtype, int64_t M, int64_t K, int64_t ldx, const void* gamma,
                       const void* beta, int gb_dtype, float eps, int8_t* q, float* scale, void* y_out,
                       cudaStream_t stream) {
  if (x_dtype != HY3D_F16 && x_dtype != HY3D_BF16) return HY3D_ERR_ARG;
  if ((gamma || beta) && (gb_dtype < HY3D_F16 || gb_dtype > HY3D_F32)) return HY3D_ERR_ARG;
  if (M < 0 || K <= 0 || (K & 7) || K > 2048 || ldx < K || (ldx & 7)) return HY3D_ERR_SHAPE;
  if (!(eps >= 0.0f)) return HY3D_ERR_ARG;
  if (M == 0) return HY3D_OK;
  if (!x || !q || !scale || (add && !y_out)) return HY3D_ERR_ARG;
  if (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(add)) & 15) || (reinterpret_cast<uintptr_t>(q) & 7) ||
      (reinterpret_cast<uintptr_t>(y_out) & 15))
    return HY3D_ERR_SHAPE;
  return x_dtype == HY3D_BF16
             ? launch_layernorm_quantize<true>(x, add, M, K, ldx, gamma, beta, gb_dtype, eps, q, scale, y_out, stream)
             : launch_layernorm_quantize<false>(x, add, M, K, ldx, gamma, beta, gb_dtype, eps, q, scale, y_out, stream);
}

int quantizer_enum_check(int x_dtype, unsigned long long* pairs, unsigned long long* mismatches,
                         cudaStream_t stream) {
  if (x_dtype != HY3D_F16 && x_dtype != HY3D_BF16) return HY3D_ERR_ARG;
  if (!pairs || !mismatches) return HY3D_ERR_ARG;
  void* counts = nullptr;
  if (cudaGetSymbolAddress(&counts, g_enum_counts) != cudaSuccess) return HY3D_ERR_CUDA;
  if (cudaMemsetAsync(counts, 0, 2 * sizeof(unsigned long long), stream) != cudaSuccess)
    return HY3D_ERR_CUDA;
  if (x_dtype == HY3D_BF16) quotient_enum_kernel<true><<<32768, 256, 0, stream>>>();
  else quotient_enum_kernel<false><<<32768, 256, 0, stream>>>();
  if (cudaGetLastError() != cudaSuccess) return HY3D_ERR_CUDA;
  unsigned long long h[2] = {0, 0};
  if (cudaMemcpyAsync(h, counts, sizeof(h), cudaMemcpyDeviceToHost, stream) != cudaSuccess)
    return HY3D_ERR_CUDA;
  if (cudaStreamSynchronize(stream) != cudaSuccess) return HY3D_ERR_CUDA;
  *pairs = h[0];
  *mismatches = h[1];
  return HY3D_OK;
}

int dequant_bias(const int32_t* acc, const float* act_scale, const void* w_scale, int ws_dtype,
                 const void* bias, int bias_dtype, void* out, int out_dtype, int64_t M, int64_t N,
                 cudaStream_t stream) {
  if (!acc || !act_scale || !w_scale || !out) return HY3D_ERR_ARG;
  if (out_dtype != HY3D_F16 && out_dtype != HY3D_BF16) return HY3D_ERR_ARG;
  if (M < 0 || N <= 0 || (N & 7)) return HY3D_ERR_SHAPE;
  if (M == 0) return HY3D_OK;
  const int64_t total = M * (N >> 3);
  int64_t blocks = (total + 255) / 256;
  if (blocks > sm_count() * 16) blocks = sm_count() * 16;
  dequant_bias_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
      acc, act_scale, w_scale, ws_dtype, bias, bias_dtype, out, out_dtype, M, N);
  return cudaGetLastError() == cudaSuccess ? HY3D_OK : HY3D_ERR_CUDA;
}

}  // namespace quant

using quant::kL1Elements;
using quant::quantize_rows;
using quant::layernorm_quantize;
using quant::dequant_bias;
using quant::quantizer_enum_check;

}  // namespace hy3d
