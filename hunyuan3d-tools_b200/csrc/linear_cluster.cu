// Whole W8A8 linear layer in one launch for problems of about one wave of small tiles, dense or 2:4 sparse:
//     out(M tokens, N) = epilogue( quantise_rows(x(M,K)) * W(N,K)^T )
//
// What bounds a program of such layers is the host: a launch costs 2.0-2.4 us there, and quantiser plus
// GEMM are two of them for 6-8 us of device time.  Here every CTA owns 128 weight rows and a block of
// tokens, quantises that block itself (redundantly over the weight tiles, which is cheap while it is
// small) and multiplies it; a cluster of ks CTAs shares a tile by ranges of K.  Every CTA
//   1  starts the TMA loads of its weights,
//   2  reads the block's rows over its K range, reduces each row's absmax, exchanging partial maxima between
//      the ks ranges through distributed shared memory,
//   3  quantises them (the arithmetic of quantize.cu, so the codes are the same bits) straight into the
//      128-byte-swizzled operand tiles,
//   4  runs tcgen05.mma kind::i8 (or mma.sp) with the weights as the 128-row A operand and the token block
//      as B, so that a handful of tokens costs a narrow instruction instead of a padded 128-row tile,
//   5  with ks > 1 sends its int32 accumulators to the CTA that owns each 32 x 32 unit of the tile, which
//      adds them (exactly), and
//   6  applies rescale / bias / GELU / GEGLU in accumulator-fragment order and stores the transposed
//      slabs by TMA.
// The CTAs of a cluster wait for one another only at hardware cluster barriers; every mbarrier wait is
// bounded as in the other kernels.
#include "common.cuh"
#include <cstdlib>

namespace hy3d {
int resident_clusters(int ranks, int per_sm);   // in capi.cu
namespace lincl {
namespace {

constexpr int kWarps = 16;
constexpr int kThreads = kWarps * 32;
constexpr int kTileW = 128;                       // weight rows per CTA
constexpr int kMaxTok = 256;                      // tokens per block (columns of the MMA)
constexpr int kMaxStages = 8;
constexpr int kMaxRanks = 8;                      // portable cluster size
constexpr int kSlab = 32;                         // tokens x weight rows of one epilogue unit
constexpr int kSlabBytes = kSlab * kSlab * 2;
constexpr int kUnitBytes = kSlab * kSlab * 4;     // int32 partials of one unit
constexpr int kSmemLimit = 227 * 1024;

// Bytes of one pipeline stage: dense 128 K elements; sparse 256 (compressed values + two metadata tiles).
constexpr int kDenseStage = kTileW * 128;
constexpr int kSparseStage = kTileW * 128 + kTileW * 32;

struct Args {
  const uint16_t* x;
  int64_t ldx;
  const void* w_scale;
  const void* bias;
  int ws_dtype, bias_dtype;
  int M, N, K;
  int block_t, ks, ku_per, num_ku, stages, w_tiles, tmem_cols;
  int q_lanes;        // lanes that share a row while it is quantised
  int red_bytes;      // exchange buffer of the partial accumulators (0 when ks == 1)
};

struct __align__(16) Ctrl {
  float amax[kMaxRanks][kMaxTok];   // partial row maxima by K range
  float scale[kMaxTok];
  float slab_scale[kWarps][kSlab];
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t tmem_full;
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void st_cluster_f32(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// Read twice by the same thread: kept in L1.
__device__ __forceinline__ uint4 ld_l1(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.ca.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}

template <bool kSparse, bool kBf16, int kEpi>
__global__ void __launch_bounds__(kThreads, 1)
linear_cluster_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_e,
                      const __grid_constant__ CUtensorMap tm_o, const Args p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t smem_base = smem_u32(smem_raw);
  if (smem_base & 1023u) {   // the swizzled tiles need a 1024-byte aligned base
    if (threadIdx.x == 0) atomicCAS(&g_device_status, 0, static_cast<int>(kDevBadAlignment));
    return;
  }
  constexpr int kUnitK = kSparse ? 256 : 128;          // K elements of a pipeline stage
  constexpr int kTokAtoms = kUnitK / 128;              // 128-byte token tiles of a stage
  constexpr uint32_t kStage = kSparse ? kSparseStage : kDenseStage;
  constexpr int kOutDtype = kBf16 ? HY3D_BF16 : HY3D_F16;

  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const int k_rank = p.ks > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
  const int tile = static_cast<int>(blockIdx.x) / p.ks;
  const int w0 = (tile % p.w_tiles) * kTileW;
  const int t0 = (tile / p.w_tiles) * p.block_t;
  const int rows = min(p.block_t, p.M - t0);
  const int ku0 = k_rank * p.ku_per;
  const int nku = min(p.ku_per, p.num_ku - ku0);       // at least 1 (the plan leaves no range empty)
  const int k0 = ku0 * kUnitK;
  const int klen = min(nku * kUnitK, p.K - k0);

  // Shared memory: [token tiles][weight stages, later the store staging][partials][control]
  const uint32_t tok_atom = static_cast<uint32_t>(p.block_t) * 128u;
  const uint32_t ring = smem_base + static_cast<uint32_t>(p.ku_per * kTokAtoms) * tok_atom;
  const uint32_t red = ring + static_cast<uint32_t>(p.stages) * kStage;
  Ctrl* ctrl = reinterpret_cast<Ctrl*>(smem_raw + (red - smem_base) + p.red_bytes);
  volatile int* abort_flag = &ctrl->abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(smem_u32(&ctrl->full[s]), 1);
      mbar_init(smem_u32(&ctrl->empty[s]), 1);
    }
    mbar_init(smem_u32(&ctrl->tmem_full), 1);
    ctrl->abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_w);
    if (kSparse) tma_prefetch_desc(&tm_e);
    tma_prefetch_desc(&tm_o);
  }
  if (warp == 1) {
    tmem_alloc_1cta(smem_u32(&ctrl->tmem_base), static_cast<uint32_t>(p.tmem_cols));
    tmem_relinquish_1cta();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (p.ks > 1) cluster_arrive();     // waited for before the first access to a peer's shared memory
  tc_fence_after_sync();
  const uint32_t tmem_base = ctrl->tmem_base;
  pdl_launch_dependents();
  pdl_wait();

  auto load_stage = [&](int u) {       // unit u of this CTA's K range into its stage
    const int s = u % p.stages;
    const uint32_t full = smem_u32(&ctrl->full[s]);
    const uint32_t sa = ring + static_cast<uint32_t>(s) * kStage;
    mbar_arrive_expect_tx(full, kStage);
    tma_load_2d(sa, &tm_w, full, (ku0 + u) * 128, w0);
    if (kSparse) {
      tma_load_2d(sa + kTileW * 128, &tm_e, full, (ku0 + u) * 32, w0);
      tma_load_2d(sa + kTileW * 144, &tm_e, full, (ku0 + u) * 32 + 16, w0);
    }
  };
  if (warp == 0 && elect_one()) {
    for (int u = 0; u < nku && u < p.stages; ++u) load_stage(u);
  }

  // ---------------- quantise the token block over this CTA's K range ----------------
  // q_lanes lanes share a row, as many as let every lane of the block work.  Both passes are short loops
  // and the second reads its values again (from L1): this code runs once per launch, so its instructions
  // are fetched cold, and an unrolled form that kept the row in registers spent twice the time on them.
  {
    const int nvec = klen >> 3;
    const int sub = lane & (p.q_lanes - 1);
    const int per = 32 / p.q_lanes, step = kWarps * per;
    const int rounds = (rows + step - 1) / step;             // the same for every warp: shuffles stay whole
    const uint16_t* xk = p.x + static_cast<int64_t>(t0) * p.ldx + k0;
    const int first = warp * per + lane / p.q_lanes;
    auto row_src = [&](int r) { return reinterpret_cast<const uint4*>(xk + static_cast<int64_t>(r) * p.ldx); };
    auto row_amax = [&](int r) {
      uint32_t acc = 0;
      if (r < rows) {
        const uint4* src = row_src(r);
#pragma unroll 4
        for (int c = sub; c < nvec; c += p.q_lanes) quant::absmax8<kBf16>(ld_l1(src + c), acc);
      }
      float a = quant::absmax_to_float<kBf16>(acc);
#pragma unroll 1
      for (int off = p.q_lanes >> 1; off > 0; off >>= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, off));
      return a;
    };
    auto write_row = [&](int r, float amax) {
      if (r >= rows) return;
      const quant::RowQuant rq = quant::row_quant(amax);
      if (sub == 0) ctrl->scale[r] = rq.scale;
      const uint4* src = row_src(r);
      const uint32_t row_at = smem_base + static_cast<uint32_t>(r >> 3) * 1024u + static_cast<uint32_t>(r & 7) * 128u;
#pragma unroll 2
      for (int c = sub; c < nvec; c += p.q_lanes) {
        float f[8];
        quant::unpack8<kBf16>(ld_l1(src + c), f);
        const uint2 q = quant::quant8(f, rq);
        // eight codes = half a 16-byte chunk of row r in token tile c / 16
        const uint32_t at = row_at + static_cast<uint32_t>(c >> 4) * tok_atom +
                            ((((static_cast<uint32_t>(c) >> 1) & 7u) ^ (static_cast<uint32_t>(r) & 7u)) << 4) +
                            (static_cast<uint32_t>(c) & 1u) * 8u;
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(q.x), "r"(q.y) : "memory");
      }
    };
    if (p.ks > 1) {
      // partial maxima of every row to the ks CTAs of the cluster
      bool waited = false;
#pragma unroll 1
      for (int i = 0; i < rounds; ++i) {
        const int r = first + i * step;
        const float a = row_amax(r);
        __syncwarp();                          // row_amax's trip counts differ by lane
        if (!waited) cluster_wait();           // the peers run: their shared memory may be written
        waited = true;
        if (r < rows && sub == 0)
          for (int kk = 0; kk < p.ks; ++kk)
            st_cluster_f32(map_to_cta(smem_u32(&ctrl->amax[k_rank][r]), static_cast<uint32_t>(kk)), a);
      }
      __syncwarp();
      cluster_arrive();
      cluster_wait();
    }
#pragma unroll 1
    for (int i = 0; i < rounds; ++i) {
      const int r = first + i * step;
      float a = 0.0f;
      if (p.ks == 1) a = row_amax(r);
      else if (r < rows)
        for (int kk = 0; kk < p.ks; ++kk) a = fmaxf(a, ctrl->amax[kk][r]);
      write_row(r, a);
    }
    fence_proxy_async_smem();                  // codes -> visible to the tensor cores
    __syncthreads();
  }

  // ---------------- weights and MMAs ----------------
  if (warp == 0) {
    bool ok = true;
    for (int u = p.stages; ok && u < nku; ++u) {
      ok = mbar_wait(smem_u32(&ctrl->empty[u % p.stages]), static_cast<uint32_t>(u / p.stages - 1) & 1u, abort_flag,
                     kDevTimeoutEmpty);
      ok = __all_sync(0xffffffffu, ok);
      if (ok && elect_one()) load_stage(u);
    }
    __syncwarp();
  } else if (warp == 1) {
    tc_fence_after_sync();
    const uint32_t idesc = make_idesc_i8(kTileW, static_cast<uint32_t>(p.block_t), kSparse);
    const uint64_t desc_const = make_smem_desc(0, 1024, 128);
    const uint32_t desc_hi = static_cast<uint32_t>(desc_const >> 32), lo_const = static_cast<uint32_t>(desc_const);
    const uint64_t desc_e = make_smem_desc(0, 128, 0);
    const uint32_t e_col = tmem_base + static_cast<uint32_t>(p.block_t);     // sparse: metadata columns behind the accumulator
    // Running low words of the two operands' descriptors (address fields; +2 per 32 bytes).
    const uint32_t a_first = lo_const | ((ring & 0x3FFFFu) >> 4), tok_step = tok_atom >> 4;
    uint32_t a_lo = a_first, b_lo = lo_const | ((smem_base & 0x3FFFFu) >> 4);
    uint32_t phase = 0;
    int s = 0, left = klen;
    bool ok = true;
    for (int u = 0; u < nku; ++u) {
      const uint32_t full = smem_u32(&ctrl->full[s]);
      ok = mbar_test_wait(full, phase);
      if (!__all_sync(0xffffffffu, ok)) {
        if (!ok) ok = mbar_wait<true>(full, phase, abort_flag, kDevTimeoutFull);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
      }
      if (elect_one()) {
        if (kSparse) {
          const uint32_t se = (a_lo & 0x3FFFu) + kTileW * 128 / 16;
          tmem_cp_128x128b_1cta(e_col, desc_e | se);
          tmem_cp_128x128b_1cta(e_col + 4, desc_e | (se + kTileW));
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (64 * k < left) {
              const uint64_t da = static_cast<uint64_t>(desc_hi) << 32 | (a_lo + 2 * k);
              const uint64_t db = static_cast<uint64_t>(desc_hi) << 32 | (k < 2 ? b_lo + 4 * k : b_lo + tok_step + 4 * (k - 2));
              mma_sp_i8_1cta(tmem_base, da, db, e_col + 2 * k, idesc, (u | k) != 0 ? 1u : 0u);
            }
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (32 * k < left) mma_i8_lohi<1>(tmem_base, a_lo + 2 * k, b_lo + 2 * k, desc_hi, idesc, (u | k) != 0 ? 1u : 0u);
        }
        tc_commit_1cta(smem_u32(&ctrl->empty[s]));
      }
      left -= kUnitK;
      b_lo += kTokAtoms * tok_step;
      a_lo += kStage >> 4;
      if (++s == p.stages) { s = 0; phase ^= 1; a_lo = a_first; }
    }
    if (ok && elect_one()) tc_commit_1cta(smem_u32(&ctrl->tmem_full));
    __syncwarp();
  }

  // ---------------- epilogue (all warps) ----------------
  const int quarter = warp & 3, first_slab = warp >> 2;
  const int nslab = (p.block_t + kSlab - 1) / kSlab;
  float wsr[4], bsr[4];                                  // fragment rows lane / 4 + 8 i
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int nr = w0 + quarter * 32 + (lane >> 2) + 8 * i;
    wsr[i] = nr < p.N ? load_scalar(p.w_scale, p.ws_dtype, nr) : 0.0f;
    bsr[i] = (p.bias && nr < p.N) ? load_scalar(p.bias, p.bias_dtype, nr) : 0.0f;
  }
  bool ok = mbar_wait(smem_u32(&ctrl->tmem_full), 0, abort_flag, kDevTimeoutTmemFull);
  ok = __all_sync(0xffffffffu, ok);
  tc_fence_after_sync();
  const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
  if (p.ks > 1) {
    // 32 x 32 unit (slab, quarter) number i belongs to range i % ks
    for (int s = first_slab; ok && s < nslab; s += kWarps / 4) {
      const int unit = 4 * s + quarter, owner = unit % p.ks;
      if (owner == k_rank) continue;
      uint32_t ra[16], rb[16];
      __syncwarp();
      tmem_ld_16x256b_x4(t_row + s * kSlab, ra);
      tmem_ld_16x256b_x4(t_row + (16u << 16) + s * kSlab, rb);
      tmem_ld_wait();
      const uint32_t dst = map_to_cta(red + static_cast<uint32_t>(unit / p.ks * p.ks + k_rank) * kUnitBytes + lane * 16u,
                                      static_cast<uint32_t>(owner));
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        st_cluster_v4(dst + 512u * j, ra[4 * j], ra[4 * j + 1], ra[4 * j + 2], ra[4 * j + 3]);
        st_cluster_v4(dst + 512u * (j + 4), rb[4 * j], rb[4 * j + 1], rb[4 * j + 2], rb[4 * j + 3]);
      }
    }
    __syncwarp();
    cluster_arrive();
    cluster_wait();
  }
  constexpr bool geglu = kEpi == HY3D_EPI_GEGLU;
  constexpr bool gelu = kEpi == HY3D_EPI_GELU;
  const int64_t ldo = geglu ? (p.N >> 1) : p.N;
  // The weight stages are free now (every MMA has completed): the slabs are staged there.  Layouts as in
  // the sparse GEMM: 64-byte rows with 64-byte swizzle, 32-byte rows with 32-byte swizzle after the gate.
  const uint32_t stage_buf = ring + static_cast<uint32_t>(warp) * kSlabBytes;
  float* asw = ctrl->slab_scale[warp];
  bool wide_gates = false;                               // not asked for: a warp has a slab or two
  const int frag_tok = 2 * (lane & 3);
  const uint32_t st_row = static_cast<uint32_t>(lane) & 7u, st_mat = static_cast<uint32_t>(lane) >> 3;
  const uint32_t st_addr =
      geglu ? stage_buf + (8u * (st_mat >> 1) + st_row) * 32u + (((st_mat & 1u) ^ ((st_row >> 2) & 1u)) << 4)
            : stage_buf + st_row * 64u + ((st_mat ^ ((st_row >> 1) & 3u)) << 4);
  for (int s = first_slab; ok && s < nslab; s += kWarps / 4) {
    const int unit = 4 * s + quarter;
    if (p.ks > 1 && unit % p.ks != k_rank) continue;
    uint32_t ra[16], rb[16];
    __syncwarp();
    asw[lane] = s * kSlab + lane < rows ? ctrl->scale[s * kSlab + lane] : 0.0f;
    tmem_ld_16x256b_x4(t_row + s * kSlab, ra);
    tmem_ld_16x256b_x4(t_row + (16u << 16) + s * kSlab, rb);
    tmem_ld_wait();
    if (p.ks > 1) {
      for (int kk = 0; kk < p.ks; ++kk) {
        if (kk == k_rank) continue;
        const uint8_t* part = smem_raw + (red - smem_base) + static_cast<uint32_t>(unit / p.ks * p.ks + kk) * kUnitBytes;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 a = reinterpret_cast<const uint4*>(part)[32 * j + lane];
          const uint4 b = reinterpret_cast<const uint4*>(part)[32 * (j + 4) + lane];
          ra[4 * j] += a.x; ra[4 * j + 1] += a.y; ra[4 * j + 2] += a.z; ra[4 * j + 3] += a.w;
          rb[4 * j] += b.x; rb[4 * j + 1] += b.y; rb[4 * j + 2] += b.z; rb[4 * j + 3] += b.w;
        }
      }
    }
    if (elect_one()) tma_store_wait_read<0>();
    __syncwarp();
    auto scaled = [&](uint32_t a0, uint32_t a1, float2 as2, int i) {
      return __ffma2_rn(make_float2(static_cast<float>(static_cast<int32_t>(a0)), static_cast<float>(static_cast<int32_t>(a1))),
                        __fmul2_rn(as2, make_float2(wsr[i], wsr[i])), make_float2(bsr[i], bsr[i]));
    };
    if (geglu) {
      // pair 2 o + h: tokens 8 o + frag_tok, + 1 of weight row r + 8 h and its gate row, 16 further on
      uint32_t out[8];
      auto pair = [&](int j, float2& v, float2& g) {
        const int i = 2 * j, h = j & 1;
        const float2 as2 = *reinterpret_cast<const float2*>(asw + 8 * (j >> 1) + frag_tok);
        v = scaled(ra[i], ra[i + 1], as2, h);
        g = scaled(rb[i], rb[i + 1], as2, 2 + h);
      };
      gated_pairs<kBf16>(out, pair, wide_gates);
      __syncwarp();
      stmatrix_x4_trans(st_addr, out[0], out[1], out[2], out[3]);
      stmatrix_x4_trans(st_addr + 512u, out[4], out[5], out[6], out[7]);
    } else {
#pragma unroll
      for (int o = 0; o < 4; ++o) {              // eight tokens at a time
        const float2 as2 = *reinterpret_cast<const float2*>(asw + 8 * o + frag_tok);
        float2 y0 = scaled(ra[4 * o], ra[4 * o + 1], as2, 0), y1 = scaled(ra[4 * o + 2], ra[4 * o + 3], as2, 1);
        float2 y2 = scaled(rb[4 * o], rb[4 * o + 1], as2, 2), y3 = scaled(rb[4 * o + 2], rb[4 * o + 3], as2, 3);
        if (gelu) { y0 = gelu_phi2(y0); y1 = gelu_phi2(y1); y2 = gelu_phi2(y2); y3 = gelu_phi2(y3); }
        stmatrix_x4_trans(st_addr + o * 512u, pack2(y0.x, y0.y, kOutDtype), pack2(y1.x, y1.y, kOutDtype),
                          pack2(y2.x, y2.y, kOutDtype), pack2(y3.x, y3.y, kOutDtype));
      }
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (elect_one()) {
      const int out_col = geglu ? ((w0 + quarter * 32) >> 1) : (w0 + quarter * 32);
      const int out_row = t0 + s * kSlab;
      if (out_col < ldo && out_row < p.M) tma_store_2d(&tm_o, stage_buf, out_col * 2, out_row);
      tma_store_commit();
    }
  }
  if (elect_one()) tma_store_wait_all<0>();

  // ---------------- teardown ----------------
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    const uint64_t start = global_timer_ns();
    while (global_timer_ns() - start < 200000ull) { }
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_1cta(tmem_base, static_cast<uint32_t>(p.tmem_cols));
  }
}

struct Plan {
  int block_t = 0, ks = 0, ku_per = 0, num_ku = 0, stages = 0, w_tiles = 0, t_tiles = 0, red_bytes = 0, smem = 0;
};

// Fills in what follows from the shape and (block_t, ns, ks); false where they do not fit.
bool complete(Plan* p, int64_t M, int64_t N, int64_t K, bool sparse) {
  const int unit_k = sparse ? 256 : 128, stage = sparse ? kSparseStage : kDenseStage;
  p->w_tiles = static_cast<int>((N + kTileW - 1) / kTileW);
  p->num_ku = static_cast<int>((K + unit_k - 1) / unit_k);
  p->ku_per = (p->num_ku + p->ks - 1) / p->ks;
  if (static_cast<int64_t>(p->ks - 1) * p->ku_per >= p->num_ku) return false;    // an empty range
  p->t_tiles = static_cast<int>((M + p->block_t - 1) / p->block_t);
  if (p->t_tiles > 1 && (p->block_t & 31)) return false;          // 32-token stores must not reach the next block
  const int units = 4 * ((p->block_t + kSlab - 1) / kSlab);
  p->red_bytes = p->ks > 1 ? (units + p->ks - 1) / p->ks * p->ks * kUnitBytes : 0;
  const int tok = p->ku_per * (unit_k / 128) * p->block_t * 128;
  const int fixed = tok + p->red_bytes + static_cast<int>(sizeof(Ctrl));
  int stages = (kSmemLimit - fixed) / stage;
  if (stages > kMaxStages) stages = kMaxStages;
  const int most = p->ku_per > 2 ? p->ku_per : 2;                  // the store staging needs two
  if (stages > most) stages = most;
  if (stages < 2) return false;
  p->stages = stages;
  p->smem = fixed + stages * stage;
  return true;
}

// Device time of a plan in microseconds, fitted to 402 plans over 34 dense and sparse shapes of one wave
// (7 % rms): set-up, first loads and drain; the block's quantisation (every CTA does all of it); the chain
// of K units; the exchanges of a K split; the epilogue's slabs.
double plan_us(const Plan& p, int64_t M, bool sparse) {
  const int64_t rows = M < p.block_t ? M : p.block_t;
  const int64_t vecs = rows * p.ku_per * (sparse ? 32 : 16);
  const int slabs = (p.block_t + kSlab - 1) / kSlab;
  return 3.6 + 0.24 * static_cast<double>((vecs + kThreads - 1) / kThreads) + 0.27 * p.ku_per +
         (p.ks > 1 ? 1.5 + 0.41 * slabs : 0.0) + 0.23 * slabs;
}

// What a caller sees of a plan beside dense_layer_us / sparse_layer_us: fitted to 117 dense and 110 sparse layers
// of random size.  The sparse MMA's metadata chain makes one CTA's K units dearer where there are many weights.
double plan_layer_us(const Plan& p, int64_t M, int64_t N, int64_t K, bool sparse) {
  const double weights = static_cast<double>(N) * K / 1e7;
  return sparse ? 1.289 * plan_us(p, M, true) - 0.96 + 0.38 * weights - (p.ks > 1 ? 0.46 : 0.0)
                : 1.156 * plan_us(p, M, false) - 0.4 + 0.25 * weights + (p.ks > 1 ? 0.2 : 0.0);
}

}  // namespace

// Whether a layer of this size should run as one launch, and with which plan.  Sizes recur in every step of
// a model, so each thread keeps the answers for the last few.
bool linear_cluster_plan(int64_t M, int64_t N, int64_t K, bool sparse, int* block_t, int* ks) {
  struct Entry { int64_t M, N, K; int sparse, sms, block_t, ks; };
  static thread_local Entry memo[64] = {};
  Entry& e = memo[(static_cast<uint64_t>(M) * 31 + static_cast<uint64_t>(N) * 7 + static_cast<uint64_t>(K >> 4) * 3 + sparse) & 63];
  const int sms = planned_sms();
  if (e.M != M || e.N != N || e.K != K || e.sparse != (sparse ? 1 : 0) || e.sms != sms) {
    e = {M, N, K, sparse ? 1 : 0, sms, 0, 0};
    // A layer takes the one launch where it is expected to be the shorter one: below the host's time for two
    // launches, and for few tokens and many dense weights, which the cluster's K split streams over the whole
    // chip (7 x 3200 -> 9632 15.9 -> 10.7 us, 2 x 7680 -> 7520 19.6 -> 15.0, 7 x 1216 -> 9760 10.6 -> 7.1).
    double best = sparse ? sparse_layer_us(M, N, K) : dense_layer_us(M, N, K);
    // more than 148 blocks of 160 tokens and one weight tile: never one wave
    for (int bt = M <= 16 ? 16 : 32; M > 0 && M <= 148 * 160 && K <= 16384 && bt <= 160; bt = bt == 16 ? 32 : bt + 32) {
      for (int k = 1; k <= kMaxRanks; ++k) {
        Plan p;
        p.block_t = bt; p.ks = k;
        if (!complete(&p, M, N, K, sparse)) continue;
        const int64_t clusters = static_cast<int64_t>(p.t_tiles) * p.w_tiles;
        // a second wave doubles the time (253 x 1792 -> 224 in 16 clusters of 7: 14.3 us, two launches 7.8)
        if (clusters * k > (k > 1 ? sms * 7 / 8 : sms) || (k > 1 && clusters > resident_clusters(k, 1))) continue;
        const double t = plan_layer_us(p, M, N, K, sparse);
        if (t < best) { best = t; e.block_t = bt; e.ks = k; }
      }
      if (bt >= M) break;
    }
  }
  *block_t = e.block_t;
  *ks = e.ks;
  return e.block_t != 0;
}

int linear_cluster(const void* x, int x_dtype, int64_t ldx, const int8_t* w, const uint32_t* meta, int64_t meta_ld,
                   const void* w_scale, int ws_dtype, const void* bias, int bias_dtype, void* out, int64_t M, int64_t N,
                   int64_t K, int epilogue, int block_t, int ks, cudaStream_t stream) {
  if (x_dtype != HY3D_F16 && x_dtype != HY3D_BF16) return HY3D_ERR_ARG;
  if (epilogue < HY3D_EPI_LINEAR || epilogue > HY3D_EPI_GEGLU) return HY3D_ERR_ARG;
  if (ws_dtype < HY3D_F16 || ws_dtype > HY3D_F32) return HY3D_ERR_ARG;
  if (bias && (bias_dtype < HY3D_F16 || bias_dtype > HY3D_F32)) return HY3D_ERR_ARG;
  const bool sparse = meta != nullptr, geglu = epilogue == HY3D_EPI_GEGLU;
  if (M < 0 || N <= 0 || K <= 0 || (K & (sparse ? 63 : 31)) || (N & (geglu ? 31 : 15)) || ldx < K || (ldx & 7)) return HY3D_ERR_SHAPE;
  if (M > (1 << 30) || N > (1 << 30) || K > 16384) return HY3D_ERR_SHAPE;
  if (sparse && meta_ld != 4 * ((K + 127) / 128)) return HY3D_ERR_SHAPE;
  if (M == 0) return HY3D_OK;
  if (!x || !w || !w_scale || !out) return HY3D_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(meta) |
       reinterpret_cast<uintptr_t>(out)) & 15)
    return HY3D_ERR_SHAPE;
  Plan pl;
  pl.block_t = block_t; pl.ks = ks;
  if (block_t < 16 || block_t > kMaxTok || (block_t & 15) || ks < 1 || ks > kMaxRanks) return HY3D_ERR_SHAPE;
  if (!complete(&pl, M, N, K, sparse)) return HY3D_ERR_SHAPE;

  Args p;
  p.x = static_cast<const uint16_t*>(x); p.ldx = ldx;
  p.w_scale = w_scale; p.bias = bias; p.ws_dtype = ws_dtype; p.bias_dtype = bias_dtype;
  p.M = static_cast<int>(M); p.N = static_cast<int>(N); p.K = static_cast<int>(K);
  p.block_t = pl.block_t; p.ks = pl.ks; p.ku_per = pl.ku_per; p.num_ku = pl.num_ku;
  p.stages = pl.stages; p.w_tiles = pl.w_tiles; p.red_bytes = pl.red_bytes;
  const int rows = M < pl.block_t ? static_cast<int>(M) : pl.block_t;
  p.q_lanes = 32;
  while (p.q_lanes > 1 && rows * p.q_lanes > kThreads) p.q_lanes >>= 1;
  p.tmem_cols = 32;
  while (p.tmem_cols < pl.block_t + (sparse ? 8 : 0)) p.tmem_cols <<= 1;

  CUtensorMap tm_w, tm_e, tm_o;
  const uint64_t w_row = static_cast<uint64_t>(sparse ? K / 2 : K);
  int rc = encode_tmap_2d_u8(&tm_w, w, w_row, static_cast<uint64_t>(N), w_row, 128, kTileW, 128);
  if (rc != HY3D_OK) return rc;
  if (sparse) {
    rc = encode_tmap_2d_u8(&tm_e, meta, static_cast<uint64_t>(meta_ld * 4), static_cast<uint64_t>(N),
                           static_cast<uint64_t>(meta_ld * 4), 16, kTileW, 0);
    if (rc != HY3D_OK) return rc;
  } else {
    tm_e = tm_w;      // unused by the kernel
  }
  const uint64_t row_bytes = static_cast<uint64_t>(geglu ? N / 2 : N) * 2;
  rc = encode_tmap_2d_u8(&tm_o, out, row_bytes, static_cast<uint64_t>(M), row_bytes, geglu ? 32 : 64, kSlab, geglu ? 32 : 64);
  if (rc != HY3D_OK) return rc;

  using KernelFn = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const Args);
#define HY3D_CL_ROW(S)                                                                                                     \
  {{linear_cluster_kernel<S, false, HY3D_EPI_LINEAR>, linear_cluster_kernel<S, false, HY3D_EPI_GELU>,                      \
    linear_cluster_kernel<S, false, HY3D_EPI_GEGLU>},                                                                      \
   {linear_cluster_kernel<S, true, HY3D_EPI_LINEAR>, linear_cluster_kernel<S, true, HY3D_EPI_GELU>,                        \
    linear_cluster_kernel<S, true, HY3D_EPI_GEGLU>}}
  static const KernelFn kernels[2][2][3] = {HY3D_CL_ROW(false), HY3D_CL_ROW(true)};
#undef HY3D_CL_ROW
  const KernelFn kernel = kernels[sparse ? 1 : 0][x_dtype == HY3D_BF16 ? 1 : 0][epilogue];
  rc = ensure_max_smem(reinterpret_cast<const void*>(kernel), kSmemLimit);
  if (rc != HY3D_OK) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(pl.ks) * static_cast<unsigned>(pl.w_tiles) * static_cast<unsigned>(pl.t_tiles));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(pl.smem);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0] = pdl_attribute();
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = static_cast<unsigned>(pl.ks);
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pl.ks > 1 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kernel, tm_w, tm_e, tm_o, p) != cudaSuccess) {
    cudaGetLastError();
    return HY3D_ERR_CUDA;
  }
  return HY3D_OK;
}

}  // namespace lincl

using lincl::linear_cluster;
using lincl::linear_cluster_plan;

}  // namespace hy3d
