// Offline 2:4 magnitude prune + compress + metadata pack for int8 weights, in one pass.
//
// Per group of four consecutive K elements the two smallest magnitudes are dropped with the
// reference's tie rule (strict comparisons, so on ties the later element survives) and the
// survivors are written in ascending index order together with the nibble idx0 | idx1<<2.
// One thread handles 32 consecutive K elements of one row: two 16-byte loads, one 16-byte
// store of compressed values, one 32-bit metadata word (8 nibbles, least-significant first)
// and optionally 8 raw nibble bytes.  Traffic: N*K read, N*K/2 + N*K/8 written.
#include "common.cuh"

#include <type_traits>

namespace hy3d {
namespace prune {
namespace {

// Returns the nibble; writes the two survivors to k0,k1.
__device__ __forceinline__ uint32_t prune_group(const int (&v)[4], int& k0, int& k1) {
  int a[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) a[i] = v[i] < 0 ? -v[i] : v[i];
  int min1 = 0, min2 = 1;
  if (a[0] > a[1]) { min1 = 1; min2 = 0; }
#pragma unroll
  for (int i = 2; i < 4; ++i) {
    if (a[i] < a[min1]) { min2 = min1; min1 = i; }
    else if (a[i] < a[min2]) { min2 = i; }
  }
  int idx0 = -1, idx1 = -1;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (i != min1 && i != min2) {
      if (idx0 < 0) idx0 = i; else idx1 = i;
    }
  }
  k0 = v[idx0];
  k1 = v[idx1];
  return static_cast<uint32_t>(idx0 | (idx1 << 2));
}

// The same selection without branches or indexed arrays, on the four bytes of one word.  The strict
// comparisons above keep the later element on ties, i.e. order equal magnitudes by index, so the two
// survivors are the two largest keys 4 * |v| + index.  Keys sit in 16-bit halves ((k0, k2) and (k1, k3))
// and a three-level min / max network on both halves at once finds them: 24 instructions a group, 38
// with six pairwise comparisons and ranks.  Returns the nibble; `two` receives the survivors (ascending
// index) in its low 16 bits.
__device__ __forceinline__ uint32_t max_u16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t min_u16x2(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t prune_word(uint32_t w, uint32_t& two) {
  const uint32_t neg = (w >> 7) & 0x01010101u;                       // 1 in the bytes below zero
  const uint32_t a = (w ^ (neg * 0xFFu)) + neg;                      // |v| per byte (|-128| = 128)
  const uint32_t x = (a & 0x00FF00FFu) * 4u + 0x00020000u;           // keys of elements 0 and 2
  const uint32_t y = ((a >> 8) & 0x00FF00FFu) * 4u + 0x00030001u;    // keys of elements 1 and 3
  const uint32_t hi = max_u16x2(x, y), lo = min_u16x2(x, y);
  const uint32_t his = __byte_perm(hi, 0u, 0x1032), los = __byte_perm(lo, 0u, 0x1032);
  const uint32_t top = max_u16x2(hi, his);
  const uint32_t second = max_u16x2(min_u16x2(hi, his), max_u16x2(lo, los));
  const uint32_t i = top & 3u, j = second & 3u;
  const uint32_t idx0 = min(i, j), idx1 = max(i, j);
  two = __byte_perm(w, 0u, 0x4400u + idx0 + idx1 * 16u);             // bytes 2, 3 of the result: zero
  return idx0 + idx1 * 4u;
}

__device__ __forceinline__ void unpack4(uint32_t w, int (&v)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = static_cast<int>(static_cast<int8_t>((w >> (8 * i)) & 0xFF));
}

__global__ void __launch_bounds__(256)
prune_pack_kernel(const int8_t* __restrict__ w, int64_t N, int K, int8_t* __restrict__ comp,
                  uint8_t* __restrict__ meta_raw, uint32_t* __restrict__ meta_packed, int meta_ld) {
  const int chunks = K >> 5;                       // 32-wide K chunks that hold data
  const int per_row = meta_packed ? meta_ld : chunks;
  const int64_t total = N * per_row;
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const int64_t row = idx / per_row;
  const int chunk = static_cast<int>(idx - row * per_row);
  if (chunk >= chunks) {  // padding word: any valid 2:4 pattern (indices 0,1)
    meta_packed[row * meta_ld + chunk] = 0x44444444u;
    return;
  }
  const uint4* src = reinterpret_cast<const uint4*>(w + row * K + (chunk << 5));
  const uint4 lo = __ldcs(src), hi = __ldcs(src + 1);
  const uint32_t words[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  uint32_t packed = 0;
  uint32_t out[4] = {0, 0, 0, 0};
  uint32_t raw[2] = {0, 0};
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    uint32_t two;
    const uint32_t nib = prune_word(words[g], two);
    packed |= nib << (4 * g);
    raw[g >> 2] |= nib << (8 * (g & 3));
    out[g >> 1] |= two << (16 * (g & 1));
  }
  *reinterpret_cast<uint4*>(comp + row * (K >> 1) + (chunk << 4)) =
      make_uint4(out[0], out[1], out[2], out[3]);
  if (meta_packed) meta_packed[row * meta_ld + chunk] = packed;
  if (meta_raw)
    *reinterpret_cast<uint2*>(meta_raw + row * (K >> 2) + (chunk << 3)) = make_uint2(raw[0], raw[1]);
}

// Largest |w| with NaN carried through, as torch's amax does.
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// The same for two 16-bit values at once, into a running pair of maxima whose signs mean nothing.
template <int kType>
__device__ __forceinline__ void absmax_nan2(uint32_t w, uint32_t& acc) {
  if (kType == HY3D_BF16) asm("max.NaN.xorsign.abs.bf16x2 %0, %0, %1;" : "+r"(acc) : "r"(w));
  else asm("max.NaN.xorsign.abs.f16x2 %0, %0, %1;" : "+r"(acc) : "r"(w));
}

// Sixteen bytes of weights as floats: 8 values of a 16-bit type, 4 of fp32.
template <int kType>
__device__ __forceinline__ void widen16(const uint4& v, float (&f)[kType == HY3D_F32 ? 4 : 8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if constexpr (kType == HY3D_F32) {
      f[i] = __uint_as_float(w[i]);
    } else if constexpr (kType == HY3D_BF16) {
      f[2 * i] = __uint_as_float(w[i] << 16);
      f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
    } else {
      const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
      f[2 * i] = t.x;
      f[2 * i + 1] = t.y;
    }
  }
}

// Correctly rounded w / scale of two weights, rounded to integers (ties to even) that are left in the low
// byte of a and b by adding 1.5 * 2^23.
__device__ __forceinline__ void quotient2(float2 w, float scale, float inv, uint32_t& a, uint32_t& b) {
  const float2 inv2 = make_float2(inv, inv), nscale2 = make_float2(-scale, -scale);
  float2 q = __fmul2_rn(w, inv2);
  q = __ffma2_rn(__ffma2_rn(q, nscale2, w), inv2, q);
  q = __ffma2_rn(__ffma2_rn(q, nscale2, w), inv2, q);
  q = __fadd2_rn(q, make_float2(12582912.0f, 12582912.0f));
  a = __float_as_uint(q.x);
  b = __float_as_uint(q.y);
}

// Per-output-channel quantisation of a weight matrix, optionally 2:4 pruned and packed, in one pass
// over HBM.  G threads share a row: 16-byte loads for the row's absmax (two 16-bit values an instruction), then every
// thread quantises eight adjacent K elements at a time and writes 8 codes, or 4 survivors and the byte of
// metadata that belongs to them.  Neighbouring lanes take neighbouring elements: loads and
// stores are contiguous, and a row of 1280 fills a warp five times (in pieces of 32 elements a thread it was two
// rounds, the second a quarter full).  The arithmetic is torch's, operation by operation, so the buffers equal those of the torch
// expressions: |w| max; dense: max(amax * (1/127), 1e-8), sparse: max(amax, 1e-8) * (1/127) (torch on
// CUDA multiplies by the reciprocal of a Python divisor); rint of the IEEE quotient w / scale.
// 16-bit weights take one fused multiply-add, w * mul + 1.5 * 2^23, with the nudged reciprocal of the activation
// quantiser: the argument in quantize.cu's header holds for this scale too, which is within 1.3e-7 of amax / 127 (w / amax
// times 127 is at least 1.9e-6 of itself away from a half-integer, 11 significant bits each, unless it is one; scale,
// reciprocal and nudge move it by 4.2e-7).  Half-integers at w = amax / 2 are told by the nudge; there are others where 127
// divides the significand of amax, and where the scale comes from the floor of 1e-8 nothing says how near a quotient lies to
// one: such rows, and fp32 weights, divide.
// Their quotient comes from the correctly rounded reciprocal and two residual corrections, two values per
// instruction: the first makes it faithful, and by Markstein's theorem ("Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990) the second then gives the correctly rounded
// one.  |w| <= amax keeps the code within +-127.  Rows whose scale is not finite (a NaN or an infinity
// among the weights) divide one by one in a loop of their own; a NaN quotient becomes 0 as in torch's cast.
// Bound by instruction issue, most of it the pruning network on the half-rate ALU pipe.  10240 x 1280 bf16 with pruning:
// the torch form, 11 launches over fp32 temporaries, took 160 us, this kernel 10.7 (without pruning 7.3), of which 6 are
// HBM time; with the corrected quotient for every weight, six packed instructions a pair instead of one, 11.6 and 8.9
// (8192 x 2048 14.3 and 10.2, now 12.7 and 8.4).  Pieces of 32 elements a thread took 16.1; four lanes that shuffle a metadata
// word together, and the question whether the row is finite at every four elements, 13.2 (both with that quotient).
// kKeep > 0 (16-bit types): a thread has at most that many vectors of its row and keeps them in registers between the
// two passes (five fill five blocks an SM, eight leave four); otherwise (fp32, rows of more than 16384) the second pass
// reads them again, which costs more than the fifth block brings (10240 x 4096 46.5 us against 35.5).
enum { kNudged, kDivided, kNotFinite };      // how a row's codes are found
template <int kType, bool kSparse, int kKeep>
__global__ void __launch_bounds__(256, kKeep > 5 ? 4 : 5)
quantize_weight_kernel(const void* __restrict__ w, int64_t N, int K, int8_t* __restrict__ codes,
                       uint32_t* __restrict__ meta, int meta_ld, void* __restrict__ scale_out, int scale_dtype, int G) {
  constexpr int kPer = kType == HY3D_F32 ? 4 : 8;       // elements of a 16-byte vector
  __shared__ float s_part[8];
  const int sub = threadIdx.x % G;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (256 / G) + threadIdx.x / G;
  const bool ok = row < N;
  const uint4* src = reinterpret_cast<const uint4*>(w) + (ok ? row : 0) * (K / kPer);
  float amax = 0.0f;
  uint4 kept[kKeep > 0 ? kKeep : 1];
  if (ok) {
    if constexpr (kType == HY3D_F32) {
#pragma unroll 4
      for (int c = sub; c < K / kPer; c += G) {
        float f[kPer];
        widen16<kType>(__ldg(src + c), f);
#pragma unroll
        for (int j = 0; j < kPer; ++j) amax = max_nan(amax, fabsf(f[j]));
      }
    } else {
      uint32_t acc = 0;
      auto fold = [&](const uint4& v) {
        absmax_nan2<kType>(v.x, acc);
        absmax_nan2<kType>(v.y, acc);
        absmax_nan2<kType>(v.z, acc);
        absmax_nan2<kType>(v.w, acc);
      };
      if constexpr (kKeep > 0) {
#pragma unroll
        for (int i = 0; i < kKeep; ++i)
          kept[i] = sub + i * G < K / kPer ? __ldcs(src + sub + i * G) : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int i = 0; i < kKeep; ++i) fold(kept[i]);
      } else {
#pragma unroll 4
        for (int c = sub; c < K / kPer; c += G) fold(__ldg(src + c));
      }
      acc &= 0x7FFF7FFFu;
      if constexpr (kType == HY3D_BF16) {
        amax = max_nan(__uint_as_float(acc << 16), __uint_as_float(acc & 0xFFFF0000u));
      } else {
        const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&acc));
        amax = max_nan(t.x, t.y);
      }
    }
  }
  for (int off = 16; off > 0; off >>= 1) amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, off));
  if (G > 32) {
    const int warp = threadIdx.x >> 5, per_row = G >> 5;
    if ((threadIdx.x & 31) == 0) s_part[warp] = amax;
    __syncthreads();
    const int first = warp / per_row * per_row;
    for (int i = 0; i < per_row; ++i) amax = max_nan(amax, s_part[first + i]);
  }
  if (!ok) return;
  const float inv127 = 1.0f / 127.0f;
  const float scale = kSparse ? __fmul_rn(amax != amax ? amax : fmaxf(amax, 1e-8f), inv127)
                              : (amax != amax ? amax : fmaxf(__fmul_rn(amax, inv127), 1e-8f));
  if (sub == 0) {
    if (scale_dtype == HY3D_BF16) static_cast<__nv_bfloat16*>(scale_out)[row] = __float2bfloat16_rn(scale);
    else static_cast<__half*>(scale_out)[row] = __float2half_rn(scale);
  }
  const bool finite = scale < __int_as_float(0x7F800000);   // false for NaN too
  const float inv = __frcp_rn(scale);
  float mul = inv;
  bool divide = kType == HY3D_F32;
  if constexpr (kType != HY3D_F32) {
    const float rest = fmaf(scale, -127.0f, amax);      // exact: a few units in the scale's last place, times 127
    mul = __int_as_float(__float_as_int(inv) + (fmaf(scale, 3.814697265625e-6f, rest) >= 0.0f ? 2 : -2));
    const bool floored = kSparse ? amax < 1e-8f : __fmul_rn(amax, inv127) < 1e-8f;
    divide = floored || fmaf(__fdiv_rn(amax, 127.0f), -127.0f, amax) == 0.0f;
  }
  const int units = K >> 3;
  auto work = [&](int u, auto how, auto vector) {
    const bool in = u < units;
    uint32_t words[2] = {0, 0};
    if (in) {
#pragma unroll
      for (int v = 0; v < 8 / kPer; ++v) {
        float f[kPer];
        widen16<kType>(vector(v), f);
#pragma unroll
        for (int j = 0; j < kPer; j += 4) {
          uint32_t b[4];
          if constexpr (how.value == kNudged) {
            const float2 t0 = quant::fast_code2(make_float2(f[j], f[j + 1]), mul), t1 = quant::fast_code2(make_float2(f[j + 2], f[j + 3]), mul);
            b[0] = __float_as_uint(t0.x); b[1] = __float_as_uint(t0.y); b[2] = __float_as_uint(t1.x); b[3] = __float_as_uint(t1.y);
          } else if constexpr (how.value == kDivided) {
            quotient2(make_float2(f[j], f[j + 1]), scale, inv, b[0], b[1]);
            quotient2(make_float2(f[j + 2], f[j + 3]), scale, inv, b[2], b[3]);
          } else {
#pragma unroll
            for (int t = 0; t < 4; ++t)
              b[t] = static_cast<uint32_t>(max(-128, min(127, __float2int_rn(__fdiv_rn(f[j + t], scale)))));
          }
          words[(v * kPer + j) >> 2] = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410);
        }
      }
    }
    if constexpr (kSparse) {
      uint32_t two0, two1;
      const uint32_t n0 = prune_word(words[0], two0), n1 = prune_word(words[1], two1);
      if (in) {
        *reinterpret_cast<uint32_t*>(codes + row * (K >> 1) + 4 * u) = two0 | two1 << 16;
        reinterpret_cast<uint8_t*>(meta + row * meta_ld)[u] = static_cast<uint8_t>(n0 | n1 << 4);
      }
    } else if (in) {
      *reinterpret_cast<uint2*>(codes + row * static_cast<int64_t>(K) + 8 * u) = make_uint2(words[0], words[1]);
    }
  };
  using Nudged = std::integral_constant<int, kNudged>;
  using Divided = std::integral_constant<int, kDivided>;
  auto again = [&](int first) { return [=](int v) { return __ldg(src + (first + sub) * (8 / kPer) + v); }; };
  if (!finite) {
#pragma unroll 1
    for (int first = 0; first < units; first += G) work(first + sub, std::integral_constant<int, kNotFinite>{}, again(first));
  } else if (divide) {
#pragma unroll 2
    for (int first = 0; first < units; first += G) work(first + sub, Divided{}, again(first));
  } else if constexpr (kKeep > 0) {
#pragma unroll
    for (int i = 0; i < kKeep; ++i)
      if (i * G < units) work(sub + i * G, Nudged{}, [&](int) { return kept[i]; });
  } else if constexpr (kType != HY3D_F32) {
#pragma unroll 2
    for (int first = 0; first < units; first += G) work(first + sub, Nudged{}, again(first));
  }
  if constexpr (kSparse)                    // padding words: any valid 2:4 pattern (indices 0,1)
    for (int c = (K >> 5) + sub; c < meta_ld; c += G) meta[row * meta_ld + c] = 0x44444444u;
}

// Any K % 4 == 0: one thread per group, byte accesses (small / odd matrices only).
__global__ void __launch_bounds__(256)
prune_compress_generic_kernel(const int8_t* __restrict__ w, int64_t N, int K,
                              int8_t* __restrict__ comp, uint8_t* __restrict__ meta_raw) {
  const int groups = K >> 2;
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= N * groups) return;
  const int8_t* p = w + idx * 4;
  int v[4] = {p[0], p[1], p[2], p[3]}, k0, k1;
  const uint32_t nib = prune_group(v, k0, k1);
  comp[idx * 2] = static_cast<int8_t>(k0);
  comp[idx * 2 + 1] = static_cast<int8_t>(k1);
  if (meta_raw) meta_raw[idx] = static_cast<uint8_t>(nib);
}

}  // namespace

int prune_pack_24(const int8_t* w, int64_t N, int64_t K, int8_t* comp, uint8_t* meta_raw,
                  uint32_t* meta_packed, int64_t meta_ld, cudaStream_t stream) {
  if (!w || !comp) return HY3D_ERR_ARG;
  if (N < 0 || K <= 0 || (K & 3) || K > (1 << 20)) return HY3D_ERR_SHAPE;
  if (N == 0) return HY3D_OK;
  const bool fast = (K & 31) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0 &&
                    (reinterpret_cast<uintptr_t>(comp) & 15) == 0 &&
                    (!meta_raw || (reinterpret_cast<uintptr_t>(meta_raw) & 7) == 0);
  if (meta_packed) {
    if (!fast) return HY3D_ERR_SHAPE;
    if (meta_ld < (K >> 5)) return HY3D_ERR_SHAPE;
  }
  if (fast) {
    const int64_t per_row = meta_packed ? meta_ld : (K >> 5);
    const int64_t blocks = (N * per_row + 255) / 256;
    if (blocks > 0x7FFFFFFF) return HY3D_ERR_SHAPE;
    prune_pack_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
        w, N, static_cast<int>(K), comp, meta_raw, meta_packed, static_cast<int>(meta_ld));
  } else {
    const int64_t blocks = (N * (K >> 2) + 255) / 256;
    if (blocks > 0x7FFFFFFF) return HY3D_ERR_SHAPE;
    prune_compress_generic_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(
        w, N, static_cast<int>(K), comp, meta_raw);
  }
  return cudaGetLastError() == cudaSuccess ? HY3D_OK : HY3D_ERR_CUDA;
}

int quantize_weight(const void* w, int w_dtype, int64_t N, int64_t K, int8_t* codes, uint32_t* meta, int64_t meta_ld,
                    void* scale, int scale_dtype, cudaStream_t stream) {
  if (w_dtype < HY3D_F16 || w_dtype > HY3D_F32) return HY3D_ERR_ARG;
  if (scale_dtype != HY3D_F16 && scale_dtype != HY3D_BF16) return HY3D_ERR_ARG;
  if (N < 0 || K <= 0 || (K & 31) || K > (1 << 20) || (meta && meta_ld < (K >> 5)) || meta_ld > (1 << 20)) return HY3D_ERR_SHAPE;
  if (N == 0) return HY3D_OK;
  if (!w || !codes || !scale) return HY3D_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(codes)) & 15) return HY3D_ERR_SHAPE;
  // Threads per row: a warp while that is at most eight rounds of eight elements a thread, then up to the block, so
  // that long rows of few channels still spread over the chip.
  int G = 32;
  while (G < 256 && (K >> 3) > 8 * G) G <<= 1;
  const int64_t blocks = (N + 256 / G - 1) / (256 / G);
  if (blocks > 0x7FFFFFFF) return HY3D_ERR_SHAPE;
  using KernelFn = void (*)(const void*, int64_t, int, int8_t*, uint32_t*, int, void*, int, int);
  // Vectors a thread keeps, by the rounds that a row takes: two (rows up to 512), five (1280 and its doublings), eight.
#define HY3D_QW(T) {{quantize_weight_kernel<T, false, 2>, quantize_weight_kernel<T, true, 2>},  \
                    {quantize_weight_kernel<T, false, 5>, quantize_weight_kernel<T, true, 5>},  \
                    {quantize_weight_kernel<T, false, 8>, quantize_weight_kernel<T, true, 8>},  \
                    {quantize_weight_kernel<T, false, 0>, quantize_weight_kernel<T, true, 0>}}
  static const KernelFn kernels[2][4][2] = {HY3D_QW(HY3D_F16), HY3D_QW(HY3D_BF16)};
#undef HY3D_QW
  static const KernelFn wide[2] = {quantize_weight_kernel<HY3D_F32, false, 0>, quantize_weight_kernel<HY3D_F32, true, 0>};
  const int64_t rounds = ((K >> 3) + G - 1) / G;
  const int sp = meta ? 1 : 0;
  const KernelFn kernel = w_dtype == HY3D_F32 ? wide[sp]
                                              : kernels[w_dtype == HY3D_BF16][rounds <= 2 ? 0 : rounds <= 5 ? 1 : rounds <= 8 ? 2 : 3][sp];
  kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(w, N, static_cast<int>(K), codes, meta,
                                                            static_cast<int>(meta_ld), scale, scale_dtype, G);
  return cudaGetLastError() == cudaSuccess ? HY3D_OK : HY3D_ERR_CUDA;
}

}  // namespace prune

using prune::prune_pack_24;
using prune::quantize_weight;

}  // namespace hy3d
