// GroupNorm (+ optional SiLU) over channels-last activations, for the UNet that surrounds the
// INT8 linear layers: x is (B, H*W, C) with C contiguous (torch's channels_last NCHW tensor),
// groups are runs of C / groups adjacent channels, statistics run over H*W x (C / groups)
// elements per (sample, group).  torch's own GroupNorm kernel takes NCHW only, so a model whose
// convolutions run NHWC pays two layout copies around every normalisation.
//
// One launch: a cluster of up to eight CTAs owns one sample's slab of whole groups.
//   pass 1  per-channel sum and sum of squares in fp32 registers, chunk of rows by chunk, folded into
//           per-group partials and exchanged through distributed shared memory
//   pass 2  mean / rstd per group, then y = x * (rstd * gamma[c]) + (beta[c] - mean * rstd * gamma[c]) on
//           the rows read again (from L2, where pass 1 left them), rounded to the activation type; with
//           silu the rounded value goes through v / (1 + exp(-v)) and is rounded again (the two roundings
//           of GroupNorm followed by SiLU as separate ops)
// Results must not depend on how the work is spread: a statistic that moves in its last place changes some
// rounding of the output, and behind an int8 quantiser a deep network turns that into 2 % of its result.  So
// the order of every sum is a function of (B, HW, C, groups) and the device's SM count alone -- row chunks, row
// lanes within a chunk, channels within a group, chunk classes -- and slabs, ranks and sets only say who adds
// which part.
// Bound by HBM at the large sizes (2 x 31.5 MB for 12 x 320 x 64 x 64: 9.7 us) beside two special-function
// instructions per element of the SiLU (7 us), by latency at the small ones.  Two grid-wide launches with
// partials in global memory took 27.1 us there and 11.5 us for 12 x 1280 x 8 x 8.
// Nothing here has a counterpart in the reference, whose UNet is stock PyTorch / diffusers.
#include "common.cuh"

namespace hy3d {
int planned_sms();
int resident_clusters(int ranks, int per_sm);
int ensure_max_smem(const void* kernel, int bytes);
namespace gnorm {
namespace {

// Three CTAs per SM: 56 registers a thread, 64 with terms to add, which would spill otherwise.
__host__ __device__ constexpr int narrow_threads(bool add) { return add ? 320 : 384; }
constexpr int kWideThreads = 1024;
// Registers that the launch bounds leave a thread: 56, 64 with terms to add, 64 in a wide CTA.  The compiler cannot use
// more, so at least this many CTAs of `warps` warps are resident on an SM (64 K registers, 64 warps, 32 CTAs).
constexpr int bounded_registers(bool wide, bool add) { return 65536 / (wide ? kWideThreads : 3 * narrow_threads(add)) / 8 * 8; }
static_assert(bounded_registers(false, false) == 56 && bounded_registers(true, false) == 64, "");
int64_t resident_ctas(bool wide, bool add, int64_t warps) {
  int64_t n = 65536 / (bounded_registers(wide, add) * 32 * warps);
  if (n > 64 / warps) n = 64 / warps;
  return n < 32 ? n : 32;
}
constexpr int kOrderThreads = 320;    // lanes of a chunk: what 320 threads over whole rows make
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

__device__ __forceinline__ float rcp_approx(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

__device__ __forceinline__ void cluster_sync_release() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Floats of a chunk's per-channel sums in shared memory.  Padded, so that chunks start in different banks: the threads that
// add a group's channels take one chunk each, and with slices of 160 floats sixteen of them met in one bank (12 x 1280 x 16 x 16
// 12.3 -> 11.2 us, 12 x 2560 x 16 x 16 17.0 -> 13.6, 12 x 1280 x 8 x 8 7.3 -> 6.7, 12 x 640 x 32 x 32 17.7 -> 17.4).
__host__ __device__ constexpr int slice_floats(int lanes, int slab) { return (lanes * 2 * slab + 31) / 32 * 32 + 2; }

// How a sample's sums are ordered: `chunks` ranges of `rows` rows; `lanes` row lanes walk a chunk with a
// stride of `lanes`; lanes, then the channels of a group are added in order; a group's chunk sums go to
// `classes` running sums (chunk modulo classes), added in order last.
struct Order {
  int chunks, rows, lanes, classes;
};

// Sets that work side by side when `most` could: evened out over the rounds that a rank's chunks take.
int even_sets(int chunks, int ranks, int most) {
  const int per_rank = (chunks + ranks - 1) / ranks, rounds = (per_rank + most - 1) / most;
  return (per_rank + rounds - 1) / rounds;
}

// i / by for 0 <= i and i * by < 2^31 (after Granlund and Montgomery, "Division by invariant integers using multiplication",
// 1994): a multiplication by ceil(2^31 / by), which is above 2^31 / by by less than one, so
// that the product errs by less than i / 2^31 < 1 / by.  The indices divided here are below 2^15 and `by` is at most 5120.
// Integer division takes some twenty instructions in a row, and every phase of the kernel began with one or two: with
// these and loops that count rows, 12 x 320 x 64 x 64 25.3 -> 24.3 us, 12 x 1280 x 16 x 16 11.2 -> 9.8, 4 x 128 x 11 x 12
// 4.6 -> 4.2.
struct Divisor {
  uint32_t magic;
  explicit Divisor(int by) : magic(static_cast<uint32_t>(((1ll << 31) + by - 1) / by)) {}
  __device__ int operator()(int i) const { return static_cast<int>(__umulhi(2u * static_cast<uint32_t>(i), magic)); }
};

// What the cut into slabs, ranks and sets gives every thread to know.
struct Cut {
  int sets;                 // chunks that a CTA works on at a time
  float inv_n;              // 1 / elements of a group
  Divisor vec_cols, lanes, width, pairs, cpg;       // vectors of a slab's row, order.lanes, 2 * slab, 2 * slab_groups
};

// Threads are laid out as (row lane ty, vector column tx): tx = tid % (slab / 8) owns 8 adjacent channels.
// In pass 1 every `order.lanes` lanes form a set that works on a chunk at a time, `reps` of them before the
// CTA folds; in pass 2 all lanes walk the rank's rows.  grid.x = S (the cluster), grid.y = slabs, grid.z =
// samples.
// kWide: up to 1024 threads, one CTA per SM, for grids that do not fill the chip.
// kAdd: 0 nothing, 1 a (B, C) term, 2 a (C) term and then the (B, C) one is added to x first, each rounded as
// a separate broadcast add would have stored it.
template <bool kBf16, int kAdd, bool kSilu, bool kWide>
__global__ void __launch_bounds__(kWide ? kWideThreads : narrow_threads(kAdd > 0), kWide ? 1 : 3)
groupnorm_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ pre, const uint16_t* __restrict__ add,
                 int64_t add_ld, int64_t HW, int C, int cpg,
                 int slab_groups, int rows_per_cta, int chunks_per_rank, int reps, Order order, Cut cut,
                 const void* __restrict__ gamma, const void* __restrict__ beta, int gb_dtype, float eps,
                 uint16_t* __restrict__ y) {
  // [chunks][2 * slab_groups] group partials, [classes][2 * slab_groups] their class sums, then the fold's
  // [sets * reps][lanes][2][slab] per-channel sums (the first slice later holds every channel's scale and shift)
  extern __shared__ float smem[];
  const int slab = slab_groups * cpg;
  const int vec_cols = slab >> 3, row_vecs = C >> 3;
  const int sets = cut.sets, k = sets * order.lanes;
  const int ty = cut.vec_cols(threadIdx.x), tx = threadIdx.x - ty * vec_cols;
  const int set = cut.lanes(ty), lane = ty - set * order.lanes;
  const int S = gridDim.x, rank = blockIdx.x, b = blockIdx.z;
  const int c0 = static_cast<int>(blockIdx.y) * slab + 8 * tx;      // this thread's first channel
  float* s_part = smem;
  float* s_class = s_part + order.chunks * 2 * slab_groups;
  float* s_acc = smem + ((order.chunks + order.classes) * 2 * slab_groups + 3) / 4 * 4;
  pdl_launch_dependents();
  if (S > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  pdl_wait();
  const int64_t base = static_cast<int64_t>(b) * HW * C + c0;
  const uint4* src = reinterpret_cast<const uint4*>(x + base);
  uint4 pv = make_uint4(0, 0, 0, 0), av = pv;
  if (kAdd == 2) pv = __ldg(reinterpret_cast<const uint4*>(pre + c0));
  if (kAdd) av = __ldcs(reinterpret_cast<const uint4*>(add + b * add_ld + c0));
  auto with_terms = [&](uint4 v) {
    if (kAdd == 2) v = add8_16<kBf16>(v, pv);
    return kAdd ? add8_16<kBf16>(v, av) : v;
  };

  bool peers_run = S == 1;
  const int set_floats = slice_floats(order.lanes, slab);
  const int last_chunk = min(order.chunks, (rank + 1) * chunks_per_rank);
  for (int first = rank * chunks_per_rank; first < last_chunk; first += sets * reps) {
    const int here = min(sets * reps, last_chunk - first);       // chunks of this batch
    for (int slot = set; slot < here; slot += sets) {
      float2 s2[4], q2[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) { s2[j] = make_float2(0.0f, 0.0f); q2[j] = make_float2(0.0f, 0.0f); }
      auto accumulate = [&](const uint4& v) {
        float2 f[4];
        unpack8f<kBf16>(with_terms(v), f);
#pragma unroll
        for (int j = 0; j < 4; ++j) { s2[j] = __fadd2_rn(s2[j], f[j]); q2[j] = __ffma2_rn(f[j], f[j], q2[j]); }
      };
      const int64_t r0 = static_cast<int64_t>(first + slot) * order.rows;
      const int rows = static_cast<int>(r0 + order.rows < HW ? order.rows : HW - r0);
      const int step = order.lanes * row_vecs;                        // at most 320 vectors and a row
      int left = rows - lane;                                         // rows from this lane's on (may be < 1)
      const uint4* in = src + (r0 + lane) * row_vecs;
      for (; left > 0; left -= 4 * order.lanes, in += 4 * step) {    // four rows in flight per thread, to the last
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u * order.lanes < left) v[u] = in[u * step];
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (u * order.lanes < left) accumulate(v[u]);
      }
      // every row lane parks its sums in its own slice
      float* mine = s_acc + slot * set_floats + lane * 2 * slab + 8 * tx;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        *reinterpret_cast<float2*>(mine + 2 * j) = s2[j];
        *reinterpret_cast<float2*>(mine + slab + 2 * j) = q2[j];
      }
    }
    __syncthreads();
    // Channel c adds the lanes of its chunk in order, group g its channels in order; the group sums of the
    // chunk go to every rank of the cluster.
    if (order.lanes > 1) {
      for (int i = threadIdx.x; i < here * 2 * slab; i += blockDim.x) {
        const int slot = cut.width(i);
        float* p = s_acc + slot * set_floats + i - slot * 2 * slab;
        float a = *p;
#pragma unroll 4
        for (int l = 1; l < order.lanes; ++l) a += p[l * 2 * slab];
        *p = a;
      }
    }
    __syncwarp();          // the fold's trip counts differ by thread; the barrier is for converged warps
    if (!peers_run) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    peers_run = true;
    __syncthreads();
    for (int i = threadIdx.x; i < here * 2 * slab_groups; i += blockDim.x) {    // sums, then sums of squares
      const int slot = cut.pairs(i), g = i - slot * 2 * slab_groups;
      const float* p = s_acc + slot * set_floats + g * cpg;
      float a = 0.0f;
#pragma unroll 4
      for (int c = 0; c < cpg; ++c) a += p[c];
      const uint32_t at = smem_u32(s_part + (first + slot) * 2 * slab_groups + g);
      for (int peer = 0; peer < S; ++peer)
        asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(map_to_cta(at, static_cast<uint32_t>(peer))), "f"(a) : "memory");
    }
    __syncthreads();       // the slices are free again
  }
  if (!peers_run) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // a rank without chunks
  if (S > 1) cluster_sync_release(); else __syncthreads();
  for (int i = threadIdx.x; i < order.classes * 2 * slab_groups; i += blockDim.x) {
    const int cls = cut.pairs(i), g = i - cls * 2 * slab_groups;
    float a = 0.0f;
#pragma unroll 4
    for (int ch = cls; ch < order.chunks; ch += order.classes) a += s_part[ch * 2 * slab_groups + g];
    s_class[i] = a;
  }
  __syncthreads();
  // One thread per channel of the slab turns the class sums into scale and shift.
  for (int c = threadIdx.x; c < slab; c += blockDim.x) {
    const int g = cut.cpg(c);
    float a = 0.0f, q = 0.0f;
    for (int cls = 0; cls < order.classes; ++cls) {
      a += s_class[cls * 2 * slab_groups + g];
      q += s_class[cls * 2 * slab_groups + slab_groups + g];
    }
    const float mean = a * cut.inv_n;
    const float rstd = rsqrtf(fmaxf(fmaf(-mean, mean, q * cut.inv_n), 0.0f) + eps);
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
    unpack8f<kBf16>(with_terms(v), f);
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
  const int64_t r0 = static_cast<int64_t>(rank) * rows_per_cta;
  const int rows = static_cast<int>(r0 + rows_per_cta < HW ? rows_per_cta : HW - r0);
  const int64_t at0 = (r0 + ty) * row_vecs;
  const int step = k * row_vecs;
  int left = rows - ty;                                               // may be < 1
  const uint4* in = src + at0;
  uint4* out = dst + at0;
  for (; left > 0; left -= 4 * k, in += 4 * step, out += 4 * step) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (u * k < left) v[u] = __ldcs(in + u * step);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (u * k < left) out[u * step] = transform(v[u]);
  }
}

// How a call is spread over the device: slabs of whole groups, ranks of a cluster, chunks that a CTA could work on at a time.
struct Spread {
  Order order;
  int slab_groups = 0, ranks = 0, sets = 0;
  bool wide = false;
};
bool spread_call(int64_t B, int64_t HW, int64_t C, int groups, bool add, int sms, Spread* spread) {
  const int cpg = static_cast<int>(C / groups);
  // The order of the sums (see Order), fixed by the shape: chunks so that 320-thread blocks of whole rows
  // would fill four per SM, at least eight rows each.
  Order& order = spread->order;
  {
    int64_t want = static_cast<int64_t>(sms) * 4 / B;
    want = want < 1 ? 1 : want > 64 ? 64 : want;
    int64_t rows = (HW + want - 1) / want;
    if (rows < 8) rows = 8;
    order.chunks = static_cast<int>((HW + rows - 1) / rows);
    order.rows = static_cast<int>((HW + order.chunks - 1) / order.chunks);
    const int full_cols = static_cast<int>(C >> 3);
    order.lanes = kOrderThreads / full_cols > 0 ? kOrderThreads / full_cols : 1;
    order.classes = order.lanes * full_cols / groups > 0 ? order.lanes * full_cols / groups : 1;
    if (order.lanes > order.rows) order.lanes = order.rows;     // the others would add zeros
  }
  // A slab is a run of whole groups, a multiple of 8 channels (so that 16-byte vectors stay inside it) and,
  // where the groups allow, at least 32 channels (one contiguous piece of a row); its partials take at most
  // 32 KB.
  int slab_groups = 0, ranks = 0, sets = 0;
  bool wide = false;
  auto slab_fits = [&](int g) {
    return groups % g == 0 && (g * cpg) % 8 == 0 && static_cast<int64_t>(order.chunks) * g <= 4096;
  };
  // One round, one wave: the narrowest slab, and the fewest ranks (at best one: no exchange) with which every
  // chunk has a set of its own and all CTAs are resident, as long as 64 CTAs remain; else the most ranks that
  // do.  Against the rule below, 12 x 2560 x 8 x 8: 7.8 us for 11.2, 12 x 1920 x 32 x 32: 32.3 for 41.8,
  // 4 x 96 x 96 x 96 (wide): 11.5 for 14.2.
  {
    int g = 1;
    while (g < groups && !(slab_fits(g) && g * cpg >= 32)) ++g;
    const int vec = g * cpg >> 3;
    for (int w = 0; w < 2 && !ranks && slab_fits(g); ++w) {
      for (int r = 1; r <= kMaxRanks; ++r) {
        const int per_rank = (order.chunks + r - 1) / r;
        if (r > 1 && (r - 1) * per_rank >= order.chunks) continue;      // a rank without chunks
        const int64_t threads = static_cast<int64_t>(per_rank) * order.lanes * vec;
        if (threads > (w ? kWideThreads : narrow_threads(add))) continue;
        const int64_t warps = (threads + 31) / 32;
        const int64_t resident = resident_ctas(w != 0, add, warps);
        const int64_t ctas = static_cast<int64_t>(r) * (groups / g) * B;
        if (ctas * 20 > sms * resident * 19) continue;                  // clusters leave a few slots empty
        slab_groups = g; ranks = r; sets = per_rank; wide = w != 0;
        if (ctas >= 64) break;
      }
    }
  }
  // Otherwise the widest slab that still gives two CTAs per SM with clusters of eight; up to eight ranks
  // while each has at least 16 rows and a chunk of its own; as many chunks at once as threads allow, evened
  // out over the rounds.
  if (!ranks) {
    for (int g = groups; g >= 1; --g) {
      if (!slab_fits(g)) continue;
      if (slab_groups && g * cpg < 32) break;
      slab_groups = g;
      if (B * (groups / g) * kMaxRanks >= 2 * sms) break;
    }
    ranks = kMaxRanks;
    while (ranks > 1 && (order.chunks < ranks || HW < static_cast<int64_t>(16) * ranks)) ranks >>= 1;
    wide = static_cast<int64_t>(ranks) * (groups / slab_groups) * B <= sms;
    sets = (wide ? kWideThreads : narrow_threads(add)) / ((slab_groups * cpg >> 3) * order.lanes);
    if (sets < 1) return false;
    // Clusters that do not all run at the same time make a second wave: as many ranks as prevent it, if any number does.
    // 8 x 96 x 89 x 86 (16 wide clusters of eight, 15 run) 24.6 us, with six ranks 16.4; 8 x 640 x 40 x 40 20.3 and 17.0
    // (seven).  Narrow CTAs with much to read hide the second wave and lose by the lanes that fewer ranks leave, the more so
    // the fewer clusters are left for it: 9 x 1920 x 65 x 34 (72 clusters, 71 run) 57.3 us, with six ranks 71.3.  260 sizes
    // that it concerns, time with a second wave over time without: wide 1.54 on average, 1.46 at least; narrow below 16 million
    // elements 1.26, 0.99 at least (below 8 million where at most a twentieth of the clusters is left over); the other narrow
    // ones 1.00, 41 of 94 below 0.985 and down to 0.80.
    const int64_t clusters = B * (groups / slab_groups), elements = B * HW * C;
    auto running = [&](int r) {
      const int64_t warps = (((slab_groups * cpg >> 3) * order.lanes * even_sets(order.chunks, r, sets)) + 31) / 32;
      const int64_t most = resident_ctas(wide, add, warps);
      const int n = resident_clusters(r, static_cast<int>(most < 8 ? most : 8));
      return n == 0 ? clusters : static_cast<int64_t>(n);
    };
    const int64_t first_wave = running(ranks);
    if (wide || elements < (clusters * 20 <= first_wave * 21 ? 8000000 : 16000000))
      for (int r = ranks; r >= 1; --r)
        if (clusters <= running(r)) { ranks = r; break; }
  }
  spread->slab_groups = slab_groups; spread->ranks = ranks; spread->sets = sets; spread->wide = wide;
  return true;
}

}  // namespace

// Nothing needs global scratch any more; callers of the C ABI still pass a workspace of this size.
int64_t workspace_floats(int64_t B, int64_t HW, int groups) {
  (void)HW;
  return B * groups * 2;
}

// Ranks of the clusters of a call (hy3d_groupnorm_ranks), 0 where it is refused.
int ranks_of(int64_t B, int64_t HW, int64_t C, int groups, bool add) {
  if (B <= 0 || HW <= 0 || C <= 0 || groups <= 0 || (C & 7) || C % groups || C > 2560 || B > 65535 || HW > (1ll << 31)) return 0;
  Spread spread;
  return spread_call(B, HW, C, groups, add, planned_sms(), &spread) ? spread.ranks : 0;
}

int groupnorm_nhwc(const void* x, const void* pre, const void* add, int64_t add_ld, int x_dtype, int64_t B, int64_t HW,
                   int64_t C, int groups, const void* gamma, const void* beta, int gb_dtype, float eps, int silu,
                   void* y, cudaStream_t stream) {
  if (x_dtype != HY3D_F16 && x_dtype != HY3D_BF16) return HY3D_ERR_ARG;
  if ((gamma || beta) && (gb_dtype < HY3D_F16 || gb_dtype > HY3D_F32)) return HY3D_ERR_ARG;
  if (B < 0 || HW <= 0 || C <= 0 || groups <= 0 || (C & 7) || C % groups) return HY3D_ERR_SHAPE;
  if (C > 2560 || B > 65535 || HW > (1ll << 31)) return HY3D_ERR_SHAPE;
  if (B == 0) return HY3D_OK;
  if (!x || !y || (pre && !add)) return HY3D_ERR_ARG;
  if (add && (add_ld < C || (add_ld & 7))) return HY3D_ERR_SHAPE;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(add) | reinterpret_cast<uintptr_t>(pre)) & 15)
    return HY3D_ERR_SHAPE;
  const int cpg = static_cast<int>(C / groups);
  const int sms = planned_sms();
  Spread spread;
  if (!spread_call(B, HW, C, groups, add != nullptr, sms, &spread)) return HY3D_ERR_SHAPE;
  const Order& order = spread.order;
  const int slab_groups = spread.slab_groups, ranks = spread.ranks;
  int sets = spread.sets;
  const bool wide = spread.wide;
  const int slab = slab_groups * cpg, vec_cols = slab >> 3;
  // As many rounds as 42 KB of slices hold between two folds.  Over 150 sizes, with and without a term, 40 KB, which the
  // padding just fills with one round less at times, take 0.7 % longer on average and up to 9 % (10 x 256 x 13 x 55 8.9 -> 9.7
  // us), 36 KB 1.1 % and up to 19 %; 46 KB are no faster.
  const int chunks_per_rank = (order.chunks + ranks - 1) / ranks;
  const int rounds = (chunks_per_rank + sets - 1) / sets;
  sets = even_sets(order.chunks, ranks, sets);
  const int k = sets * order.lanes;
  int reps = 42 * 1024 / (sets * slice_floats(order.lanes, slab) * 4);
  reps = reps < 1 ? 1 : reps > rounds ? rounds : reps;
  const int64_t rows_per_cta = (HW + ranks - 1) / ranks;
  const size_t smem = (static_cast<size_t>(order.chunks + order.classes) * 2 * slab_groups + 3 +
                       static_cast<size_t>(reps) * sets * slice_floats(order.lanes, slab)) * sizeof(float);
  if (rows_per_cta > 0x7FFFFFFF || B > 65535 || groups / slab_groups > 65535) return HY3D_ERR_SHAPE;

  using KernelFn = void (*)(const uint16_t*, const uint16_t*, const uint16_t*, int64_t, int64_t, int, int, int, int, int, int, Order, Cut, const void*,
                            const void*, int, float, uint16_t*);
#define HY3D_GN_ADD(BF, A, W) {groupnorm_kernel<BF, A, false, W>, groupnorm_kernel<BF, A, true, W>}
#define HY3D_GN_ROW(W)                                                                    \
  {{HY3D_GN_ADD(false, 0, W), HY3D_GN_ADD(false, 1, W), HY3D_GN_ADD(false, 2, W)},        \
   {HY3D_GN_ADD(true, 0, W), HY3D_GN_ADD(true, 1, W), HY3D_GN_ADD(true, 2, W)}}
  static const KernelFn kernels[2][2][3][2] = {HY3D_GN_ROW(false), HY3D_GN_ROW(true)};
#undef HY3D_GN_ROW
#undef HY3D_GN_ADD
  const KernelFn kernel = kernels[wide ? 1 : 0][x_dtype == HY3D_BF16 ? 1 : 0][pre ? 2 : add ? 1 : 0][silu ? 1 : 0];
  if (smem > 48 * 1024) {          // few samples of many chunks and narrow groups
    const int rc = ensure_max_smem(reinterpret_cast<const void*>(kernel), 116 * 1024);
    if (rc != HY3D_OK) return rc;
    if (smem > 116 * 1024) return HY3D_ERR_SHAPE;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(ranks), static_cast<unsigned>(groups / slab_groups), static_cast<unsigned>(B));
  cfg.blockDim = dim3(static_cast<unsigned>(vec_cols * k));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  // Shared memory for as few CTAs an SM as run all clusters at the same time, L1 with what is left: 12 x 320 x 64 x 64 with
  // room for one CTA fewer 35.6 us, with all of it shared 30.6, as here 25.1 (24.3 since).  Clusters leave SMs of a GPC empty, so an
  // even share of the CTAs is not always enough: 6 x 960 x 64 x 64 (48 clusters of six) 42.4 us with room for two CTAs, 30.5
  // for three, 2 x 320 x 32 x 32 (16 of eight) 10.8 for one, 6.8 for two.  From two CTAs on the scheduler leaves a few more.
  const int64_t clusters = static_cast<int64_t>(groups / slab_groups) * B;
  const int64_t most = resident_ctas(wide, add != nullptr, (vec_cols * k + 31) / 32);
  int64_t room = (clusters * ranks + sms - 1) / sms;
  auto holds = [&](int64_t per_sm) {
    const int64_t n = resident_clusters(ranks, static_cast<int>(per_sm));
    return n == 0 || (per_sm == 1 ? clusters <= n : clusters * 20 <= n * 19);
  };
  while (room < most && !holds(room)) ++room;
  const Cut cut{sets, 1.0f / (static_cast<float>(HW) * static_cast<float>(cpg)), Divisor(vec_cols), Divisor(order.lanes),
                Divisor(2 * slab), Divisor(2 * slab_groups), Divisor(cpg)};
  cudaLaunchAttribute attr[3];
  attr[0] = pdl_attribute();
  attr[2] = carveout_attribute(room < most ? room : most, static_cast<int64_t>(smem));
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(ranks);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 3;
  const cudaError_t err = cudaLaunchKernelEx(
      &cfg, kernel, static_cast<const uint16_t*>(x), static_cast<const uint16_t*>(pre), static_cast<const uint16_t*>(add), add_ld, HW, static_cast<int>(C), cpg,
      slab_groups, static_cast<int>(rows_per_cta), chunks_per_rank, reps, order, cut, gamma, beta, gb_dtype, eps, static_cast<uint16_t*>(y));
  if (err != cudaSuccess) {
    cudaGetLastError();
    return HY3D_ERR_CUDA;
  }
  return HY3D_OK;
}

}  // namespace gnorm
}  // namespace hy3d
