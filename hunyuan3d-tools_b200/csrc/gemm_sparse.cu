// 2:4 structured-sparse W8A8 GEMM for sm_100a:
//     out(M tokens, N) = epilogue( X(M,K) s8 * Wpruned(N,K)^T -> s32 )
// The pruned weight is the sparse A operand of tcgen05.mma.sp kind::i8 (128 weight rows per
// tile on the 128 tensor-memory lanes); a block of tokens is the dense B operand, so the
// accumulator tile is D[weight row, token] and the epilogue writes it transposed.
//
// Per 256-deep K block a stage of shared memory holds
//     A  128 rows x 128 B      compressed weights, 128-byte swizzle            (TMA)
//     E  2 x (128 rows x 16 B) metadata, 8 nibbles per 32 K, plain rows        (TMA, no swizzle)
//     B  2 x (block_t rows x 128 B) int8 activations, 128-byte swizzle         (TMA)
// The MMA thread copies E into tensor memory with two tcgen05.cp (128 lanes x 128 bits each =
// the metadata of two K=64 instructions) and issues four tcgen05.mma.sp per stage.  tcgen05.cp
// and tcgen05.mma issued by one thread execute in issue order, so one 8-column metadata slot
// in tensor memory is enough.  Roles, accumulator double-buffering and bounded waits are as in
// the dense kernel.
//
// CTA-pair variant (kG == 2, cta_group::2): a tile is 256 weight rows x block_t tokens; each
// CTA stages its own 128 weight rows (A and E) and HALF of the token tile, so the activation
// traffic into shared memory -- most of a stage -- is halved per CTA.  Loads are plain
// cp.async.bulk.tensor ... .cta_group::2 crediting the leader's barrier (no multicast); the
// leader issues tcgen05.cp / tcgen05.mma.sp for the pair and commits to both CTAs' barriers.
#include "common.cuh"
#include <cstdlib>

namespace hy3d {
namespace sparse {
namespace {

constexpr int kTileW = 128;          // weight rows per tile (tensor-memory lanes)
constexpr int kBlockK = 256;         // logical K per stage (four K=64 instructions)
constexpr int kABytes = kTileW * (kBlockK / 2);   // 16384: 128 rows x 128 B of compressed weights
constexpr int kEBytes = kTileW * (kBlockK / 8);   // 4096: two 128 x 16 B metadata tiles
constexpr int kMaxStages = 8;
constexpr int kEpiWarps = 16;                         // four per 32-lane quarter of tensor memory
constexpr int kWarpsPerQuarter = kEpiWarps / 4;
constexpr int kEpiThreads = kEpiWarps * 32;
constexpr int kThreads = 64 + kEpiThreads;
constexpr int kSlabTokens = 32;                       // tokens per TMA store
constexpr int kSlabBytes = kSlabTokens * 64;          // 32 tokens x 32 columns x 2 B
constexpr int kSmemLimit = 227 * 1024;
constexpr int kMaxBlockT = 240;      // 2 * 240 accumulator columns + 8 metadata columns <= 512
// With one accumulator buffer, for launches in which no CTA has a second tile.  A stage of a pair then brings 52 KB for 512
// cycles of MMA instead of 36 KB for 256 at 128 tokens, and the fill of shared memory is what paces deep stages:
// 2915 x 5120 -> 1296 in one round of 72 tiles 14.4 us, in two rounds of 128 tokens 17.1 (with GELU 15.7 and 17.8);
// 256 x 1280 -> 18944 8.4 -> 7.6.
constexpr int kWideBlockT = 256;

struct SparseArgs {
  const float* act_scale;
  const void* w_scale;
  const void* bias;
  void* out;
  int ws_dtype, bias_dtype, out_dtype, epilogue;
  int M, N, K;
  int block_t, stages, tma_store;
  int num_kb, last_ksteps;
  int fast_tiles, total_tiles;      // tile order: weight or token tiles run fastest (see tokens_fastest)
  int share, rest;        // tokens fastest: tiles of a CTA's (pair's) contiguous range, the first `rest` have one more; else 0
};

// A launch whose arguments take 616 bytes with the four tensor maps costs the calling thread 0.2 to 0.3 us more than one of
// 608 (924 x 1024 -> 640, whole layer in a loop 7.9 and 7.6 us; LayerNorm-quantise with 104 bytes of them 4.9, with 96 4.5).
static_assert(sizeof(SparseArgs) <= 96, "");

struct __align__(16) SparseCtrl {
  float as[2][256];     // per-token activation scales of the current tile, per accumulator buffer
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};

__device__ __forceinline__ void epi_bar_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(kEpiThreads) : "memory");
}

__device__ __forceinline__ void store_one(void* out, int out_dtype, int64_t idx, float v) {
  if (out_dtype == HY3D_BF16)
    reinterpret_cast<__nv_bfloat16*>(out)[idx] = __float2bfloat16_rn(v);
  else
    reinterpret_cast<__half*>(out)[idx] = __float2half_rn(v);
}

// kBf16 / kEpi select the output packing and the epilogue at compile time for the 16-bit
// outputs (raw int32 output runs the <false, LINEAR> instance's direct-store path).
template <int kG, bool kBf16, int kEpi>
__global__ void __launch_bounds__(kThreads, 1)
gemm_sparse_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_e,
                   const __grid_constant__ CUtensorMap tm_x, const __grid_constant__ CUtensorMap tm_o,
                   const SparseArgs p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  const uint32_t smem_base = smem_u32(smem_raw);
  if (smem_base & 1023u) {   // the swizzled tiles need a 1024-byte aligned base
    if (threadIdx.x == 0) atomicCAS(&g_device_status, 0, static_cast<int>(kDevBadAlignment));
    return;
  }

  // One 128-byte-wide box of tokens; with a CTA pair each CTA stages half of the token tile.
  const uint32_t b_half = static_cast<uint32_t>(p.block_t / kG) * 128u;
  const uint32_t b_bytes = 2u * b_half;
  const uint32_t stage_bytes = kABytes + kEBytes + b_bytes;
  const uint32_t staging_base = smem_base + static_cast<uint32_t>(p.stages) * stage_bytes;
  SparseCtrl* ctrl = reinterpret_cast<SparseCtrl*>(smem + static_cast<size_t>(p.stages) * stage_bytes +
                                                   kEpiWarps * kSlabBytes);
  volatile int* abort_flag = &ctrl->abort_flag;

  // Warp index through a shuffle: known warp-uniform to the compiler, so the producer and MMA
  // roles run as warp-uniform loops (all lanes wait, the elected one issues) with their descriptors and
  // coordinates in uniform registers.
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = kG == 2 ? cluster_cta_rank() : 0u;
  const bool leader = cta_rank == 0;
  const int walker = static_cast<int>(blockIdx.x) / kG;
  const bool w_fastest = p.share == 0;
  const int first_tile = w_fastest ? walker : walker * p.share + min(walker, p.rest);
  const int end_tile = w_fastest ? p.total_tiles : first_tile + p.share + (walker < p.rest ? 1 : 0);
  const int tile_step = w_fastest ? static_cast<int>(gridDim.x) / kG : 1;
  const int row_off = static_cast<int>(cta_rank) * kTileW;                 // this CTA's weight rows
  const int tok_off = static_cast<int>(cta_rank) * (p.block_t / kG);       // this CTA's share of B
  const uint32_t tmem_cols = 512;
  const uint32_t e_col = static_cast<uint32_t>((p.block_t > kMaxBlockT ? 1 : 2) * p.block_t);     // behind the accumulators

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(smem_u32(&ctrl->full[s]), 1);
      mbar_init(smem_u32(&ctrl->empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&ctrl->tmem_full[b]), 1);
      mbar_init(smem_u32(&ctrl->tmem_empty[b]), kG * kEpiWarps);   // one arrival per epilogue warp
    }
    ctrl->abort_flag = 0;
    fence_barrier_init();
    tma_prefetch_desc(&tm_w);
    tma_prefetch_desc(&tm_e);
    tma_prefetch_desc(&tm_x);
    if (p.tma_store) tma_prefetch_desc(&tm_o);
  }
  if (warp == 1) {
    if (kG == 2) {
      tmem_alloc_2cta(smem_u32(&ctrl->tmem_base), tmem_cols);
      tmem_relinquish_2cta();
    } else {
      tmem_alloc_1cta(smem_u32(&ctrl->tmem_base), tmem_cols);
      tmem_relinquish_1cta();
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (kG == 2) cluster_sync_all();   // the peer's barriers exist before anything signals them
  tc_fence_after_sync();
  const uint32_t tmem_base = ctrl->tmem_base;
  pdl_launch_dependents();
  pdl_wait();

  if (warp == 0) {
    // ---------------- TMA producer (all lanes walk the loop, the elected one issues) ----------------
    {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = first_tile; ok && tile < end_tile; tile += tile_step) {
        const int slow = tile / p.fast_tiles, fast = tile - slow * p.fast_tiles;
        const int w0 = (w_fastest ? fast : slow) * (kTileW * kG) + row_off;
        const int t0 = (w_fastest ? slow : fast) * p.block_t + tok_off;
        for (int kb = 0; kb < p.num_kb; ++kb) {
          ok = mbar_wait(smem_u32(&ctrl->empty[stage]), phase ^ 1, abort_flag, kDevTimeoutEmpty);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          const uint32_t full = smem_u32(&ctrl->full[stage]);
          const uint32_t sa = smem_base + stage * stage_bytes;
          const uint32_t sb = sa + kABytes + kEBytes;
          if (!elect_one()) {
            // only the elected lane issues
          } else if (kG == 1) {
            mbar_arrive_expect_tx(full, stage_bytes);
            tma_load_2d(sa, &tm_w, full, kb * (kBlockK / 2), w0);
            tma_load_2d(sa + kABytes, &tm_e, full, kb * (kBlockK / 8), w0);
            tma_load_2d(sa + kABytes + kEBytes / 2, &tm_e, full, kb * (kBlockK / 8) + 16, w0);
            tma_load_2d(sb, &tm_x, full, kb * kBlockK, t0);
            tma_load_2d(sb + b_half, &tm_x, full, kb * kBlockK + 128, t0);
          } else {
            // Both CTAs credit their bytes to the leader's barrier; only the leader arrives.
            const uint32_t full_leader = map_to_cta(full, 0);
            if (leader) mbar_arrive_expect_tx(full, 2 * stage_bytes);
            tma_load_2d_pair(sa, &tm_w, full_leader, kb * (kBlockK / 2), w0);
            tma_load_2d_pair(sa + kABytes, &tm_e, full_leader, kb * (kBlockK / 8), w0);
            tma_load_2d_pair(sa + kABytes + kEBytes / 2, &tm_e, full_leader, kb * (kBlockK / 8) + 16, w0);
            tma_load_2d_pair(sb, &tm_x, full_leader, kb * kBlockK, t0);
            tma_load_2d_pair(sb + b_half, &tm_x, full_leader, kb * kBlockK + 128, t0);
          }
          if (++stage == p.stages) { stage = 0; phase ^= 1; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ---------------- MMA issuer (one thread) ----------------
    if (leader) {
      // One thread issues, named by elect.sync: the compiler then knows that there is one, and descriptors stay in
      // uniform registers (behind `lane == 0` every issue converted them for whichever lanes were active).
      // Descriptors advance as low words, see the dense kernel.
      const uint32_t idesc = make_idesc_i8(kTileW * kG, static_cast<uint32_t>(p.block_t), true);
      const uint64_t desc_const = make_smem_desc(0, 1024, 128);
      const uint32_t desc_hi = static_cast<uint32_t>(desc_const >> 32);
      const uint64_t desc_e = make_smem_desc(0, 128, 0);
      const uint32_t a_lo0 = static_cast<uint32_t>(desc_const) | ((smem_base & 0x3FFFFu) >> 4);
      const uint32_t stage_step = stage_bytes >> 4, e_off = kABytes >> 4, b_off = (kABytes + kEBytes) >> 4, b_box = b_half >> 4;
      const uint32_t e_tmem = tmem_base + e_col;
      int stage = 0;
      uint32_t phase = 0, a_lo = a_lo0;
      bool ok = true;
      int it = 0;
      for (int tile = first_tile; ok && tile < end_tile; tile += tile_step, ++it) {
        const int buf = it & 1;
        const uint32_t acc_phase = (it >> 1) & 1;
        ok = mbar_wait(smem_u32(&ctrl->tmem_empty[buf]), acc_phase ^ 1, abort_flag,
                       kDevTimeoutTmemEmpty);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(buf * p.block_t);
        uint32_t acc = 0;   // the first MMA of a tile overwrites the accumulator
        for (int kb = 0; kb < p.num_kb; ++kb) {
          const uint32_t bar = smem_u32(&ctrl->full[stage]);
          ok = mbar_test_wait(bar, phase);
          if (!__all_sync(0xffffffffu, ok)) {
            if (!ok) ok = mbar_wait<true>(bar, phase, abort_flag, kDevTimeoutFull);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
          }
          const int nk = kb == p.num_kb - 1 ? p.last_ksteps : 4;
          if (elect_one()) {
            // Metadata of the stage: two 128-lane x 128-bit copies = 8 columns = four K=64 steps.
            const uint64_t de0 = desc_e | ((a_lo + e_off) & 0x3FFFu), de1 = desc_e | ((a_lo + e_off + (kEBytes >> 5)) & 0x3FFFu);
            if (kG == 1) {
              tmem_cp_128x128b_1cta(e_tmem, de0);
              tmem_cp_128x128b_1cta(e_tmem + 4, de1);
            } else {
              tmem_cp_128x128b_2cta(e_tmem, de0);
              tmem_cp_128x128b_2cta(e_tmem + 4, de1);
            }
            // Per K=64 instruction: 32 compressed bytes of A (+2 address units), 64 bytes of B
            // (+4; the second 128-byte box after two steps) and two metadata columns.
            const uint32_t b_lo = a_lo + b_off;
            mma_sp_i8_lohi<kG>(d_tmem, a_lo, b_lo, desc_hi, e_tmem, idesc, acc);
            if (nk > 1) mma_sp_i8_lohi<kG>(d_tmem, a_lo + 2, b_lo + 4, desc_hi, e_tmem + 2, idesc, 1u);
            if (nk > 2) mma_sp_i8_lohi<kG>(d_tmem, a_lo + 4, b_lo + b_box, desc_hi, e_tmem + 4, idesc, 1u);
            if (nk > 3) mma_sp_i8_lohi<kG>(d_tmem, a_lo + 6, b_lo + b_box + 4, desc_hi, e_tmem + 6, idesc, 1u);
            if (kG == 1) tc_commit_1cta(smem_u32(&ctrl->empty[stage]));
            else tc_commit_2cta(smem_u32(&ctrl->empty[stage]), 3);
          }
          acc = 1u;
          a_lo += stage_step;
          if (++stage == p.stages) { stage = 0; phase ^= 1; a_lo = a_lo0; }
        }
        if (ok && elect_one()) {
          if (kG == 1) tc_commit_1cta(smem_u32(&ctrl->tmem_full[buf]));
          else tc_commit_2cta(smem_u32(&ctrl->tmem_full[buf]), 3);
        }
        __syncwarp();
      }
    }
    __syncwarp();
  } else {
    // ---------------- epilogue ----------------
    const int quarter = warp & 3;                   // tensor-memory lane quarter
    const int half = (warp - 2) >> 2;               // which of the warps sharing it
    const int row_in_tile = quarter * 32 + lane;    // weight row within the tile
    const int et = threadIdx.x - 64;
    constexpr bool geglu = kEpi == HY3D_EPI_GEGLU;
    constexpr bool gelu = kEpi == HY3D_EPI_GELU;
    constexpr int kOutDtype = kBf16 ? HY3D_BF16 : HY3D_F16;
    const int64_t ldo = geglu ? (p.N >> 1) : p.N;
    const uint32_t stage_buf = staging_base + static_cast<uint32_t>(warp - 2) * kSlabBytes;
    bool ok = true, wide_gates = false;
    int it = 0;
    float wsr[4] = {0.0f, 0.0f, 0.0f, 0.0f}, bsr[4] = {0.0f, 0.0f, 0.0f, 0.0f};   // of the fragment rows of w0
    int cur_w0 = -1;
    for (int tile = first_tile; tile < end_tile; tile += tile_step, ++it) {
      const int buf = it & 1;
      const uint32_t acc_phase = (it >> 1) & 1;
      const int slow = tile / p.fast_tiles, fast = tile - slow * p.fast_tiles;
      const int w0 = (w_fastest ? fast : slow) * (kTileW * kG) + row_off;
      const int t0 = (w_fastest ? slow : fast) * p.block_t;
      const int n = w0 + row_in_tile;
      const bool n_ok = n < p.N;
      // Which slabs a warp takes moves on from tile to tile: with a number of slabs that four does not divide (seven
      // of 224 tokens) the same warps would always have one more.
      const int first_slab = (half + it) & (kWarpsPerQuarter - 1);
      bool arrived = false;
      // The accumulator buffer goes back to the leader's MMA warp (own CTA or the peer) once this warp's loads have landed.
      auto release_acc = [&]() {
        tc_fence_before_sync();
        __syncwarp();
        if (elect_one()) {
          if (kG == 1 || leader) mbar_arrive(smem_u32(&ctrl->tmem_empty[buf]));
          else mbar_arrive_cluster(smem_u32(&ctrl->tmem_empty[buf]), 0);
        }
        arrived = true;
      };
      float ws = 0.0f, bs = 0.0f;                            // direct stores: weight row n
      float sc_next = 0.0f;
      if (p.out_dtype != HY3D_S32) {
        if (p.tma_store) {
          // Each warp stages the 32 token scales of its own slab (fetched one slab ahead), so
          // the tile needs no CTA-wide barrier.
          const int t = t0 + first_slab * kSlabTokens + lane;
          if (first_slab * kSlabTokens < p.block_t && t < p.M) sc_next = p.act_scale[t];
          if (w0 != cur_w0) {
            cur_w0 = w0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int nr = w0 + quarter * 32 + (lane >> 2) + 8 * i;
              wsr[i] = bsr[i] = 0.0f;
              if (nr < p.N) {
                wsr[i] = load_scalar(p.w_scale, p.ws_dtype, nr);
                bsr[i] = p.bias ? load_scalar(p.bias, p.bias_dtype, nr) : 0.0f;
              }
            }
          }
        } else {
          for (int c = et; c < p.block_t; c += kEpiThreads)
            ctrl->as[buf][c] = (t0 + c) < p.M ? p.act_scale[t0 + c] : 0.0f;
        }
        if (!p.tma_store && n_ok) {
          ws = load_scalar(p.w_scale, p.ws_dtype, n);
          bs = p.bias ? load_scalar(p.bias, p.bias_dtype, n) : 0.0f;
        }
      }
      if (!p.tma_store) epi_bar_sync();
      if (ok) ok = mbar_wait(smem_u32(&ctrl->tmem_full[buf]), acc_phase, abort_flag,
                             kDevTimeoutTmemFull);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) continue;
      tc_fence_after_sync();
      const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                             static_cast<uint32_t>(buf * p.block_t);
      const float* asb = ctrl->as[buf];
      if (p.tma_store) {
        float* asw = &ctrl->as[0][0] + (warp - 2) * kSlabTokens;   // this warp's 32 scales
        // Slabs of 32 tokens x the warp's 32 weight rows, read from tensor memory in accumulator-
        // fragment order: a thread then holds neighbouring tokens of four weight rows (r, r + 8 from
        // lanes 0-15; r + 16, r + 24 from lanes 16-31, r = lane / 4), which is what a transposing
        // stmatrix takes -- four of those write the slab, where one thread per output column needed
        // 32 two-byte stores.  With GEGLU, weight rows come in blocks of 16 value rows and their 16
        // gate rows, so value and gate of an output sit in the same register of the two loads: no
        // exchange between lanes, and every lane works on a gate.
        const int nslab = p.block_t / kSlabTokens;
        const int frag_tok = 2 * (lane & 3);
        // Output rows in the staging buffer: 64 bytes with 64-byte swizzle (16-byte chunk c of token j
        // at c ^ ((j >> 1) & 3)), or 32 bytes with 32-byte swizzle after the gate (c ^ ((j >> 2) & 1));
        // either way the eight rows of a matrix fall into different banks.
        const uint32_t st_row = static_cast<uint32_t>(lane) & 7u, st_mat = static_cast<uint32_t>(lane) >> 3;
        const uint32_t st_addr =
            geglu ? stage_buf + (8u * (st_mat >> 1) + st_row) * 32u + (((st_mat & 1u) ^ ((st_row >> 2) & 1u)) << 4)
                  : stage_buf + st_row * 64u + ((st_mat ^ ((st_row >> 1) & 3u)) << 4);
        for (int s = first_slab; s < nslab; s += kWarpsPerQuarter) {
          const int c0 = s * kSlabTokens;
          uint32_t ra[16], rb[16];
          const float sc = sc_next;
          {
            const int sn = s + kWarpsPerQuarter;
            const int t = t0 + sn * kSlabTokens + lane;
            sc_next = (sn < nslab && t < p.M) ? p.act_scale[t] : 0.0f;
          }
          __syncwarp();
          asw[lane] = sc;
          tmem_ld_16x256b_x4(t_row + c0, ra);
          tmem_ld_16x256b_x4(t_row + (16u << 16) + c0, rb);
          tmem_ld_wait();
          if (s + kWarpsPerQuarter >= nslab) release_acc();
          if (elect_one()) tma_store_wait_read<0>();
          __syncwarp();
          // `as * ws` and the fused multiply-add of two neighbouring tokens of one weight row
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
            if (kBf16 && wide_gates) gated_pairs_wide(out, pair, wide_gates);
            else gated_pairs<kBf16>(out, pair, wide_gates);
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
            const int out_row = t0 + c0;
            if (out_col < ldo && out_row < p.M) tma_store_2d(&tm_o, stage_buf, out_col * 2, out_row);
            tma_store_commit();
          }
        }
      } else {
        // GEGLU: weight rows come in blocks of 32 = 16 value rows then their 16 gate rows, so
        // lanes 0-15 hold values and lanes 16-31 the matching gates.
        const int64_t out_col = geglu ? ((w0 + quarter * 32) >> 1) + (lane & 15) : n;
        for (int c = 16 * half; c < p.block_t; c += 16 * kWarpsPerQuarter) {
          uint32_t r[16];
          __syncwarp();
          tmem_ld_x16(t_row + c, r);
          tmem_ld_wait();
          if (p.out_dtype == HY3D_S32) {
            if (n_ok) {
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const int t = t0 + c + j;
                if (t < p.M)
                  reinterpret_cast<int32_t*>(p.out)[static_cast<int64_t>(t) * ldo + n] =
                      static_cast<int32_t>(r[j]);
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const int t = t0 + c + j;
              float y = fmaf(static_cast<float>(static_cast<int32_t>(r[j])), asb[c + j] * ws, bs);
              if (gelu) y = gelu_phi(y);
              if (geglu) {
                const float g = __shfl_down_sync(0xffffffffu, y, 16);
                y = gated1<kBf16>(y, g);
                if (lane < 16 && n_ok && t < p.M)
                  store_one(p.out, p.out_dtype, static_cast<int64_t>(t) * ldo + out_col, y);
              } else if (n_ok && t < p.M) {
                store_one(p.out, p.out_dtype, static_cast<int64_t>(t) * ldo + out_col, y);
              }
            }
          }
        }
      }
      if (!arrived) release_acc();
    }
    __syncwarp();
    if (p.tma_store && elect_one()) tma_store_wait_all<0>();
  }

  // ---------------- teardown ----------------
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) { }
    __syncthreads();
  }
  // Neither CTA of a pair may retire while the other can still touch its shared memory,
  // barriers or tensor memory.
  if (kG == 2) cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    if (kG == 2) tmem_dealloc_2cta(tmem_base, tmem_cols);
    else tmem_dealloc_1cta(tmem_base, tmem_cols);
  }
}

// Tile shape.  CTA pairs (256 weight rows sharing one token tile) halve each CTA's activation traffic into
// shared memory, which is what paces deep-K stages, and cost more per tile hand-off; a wide token tile
// amortises the weights, a narrow one spreads few tokens over the chip.  Both come from one cost model, in
// microseconds, fitted to 120 shapes of random size with each epilogue x all tiles (7 % rms); the tile it picks is
// 0.6 % from the best on average (the model before, fitted when a pair's hand-over cost 2000 cycles: 1.3 %):
//   2915 x 5120 -> 1296 with GELU: single CTAs of 128 tokens 21.1 us, pairs of 128 17.8, one round of 256 15.7
// (the same constants hold for those: over 54 shapes that could take them none got slower by more than 2 %).
struct SparseTile {
  int block_t = 0, group = 1;
  double us = 1e30;
};
SparseTile search_tile(int64_t M, int64_t N, int64_t K, int epilogue, int block_t, int sms, int cta_group = 0) {
  SparseTile best;
  const int64_t kblocks = (K + kBlockK - 1) / kBlockK;
  for (int g = 1; g <= 2; ++g) {
    if (cta_group != 0 && g != cta_group) continue;
    for (int bt = 32; bt <= kWideBlockT; bt += 32) {
      if (block_t != 0 && bt != 32) break;             // the caller's width, one pass per group
      const int t = block_t != 0 ? block_t : bt;
      if (t < 16 || t > kWideBlockT || (t & 15) || (g == 2 && (t & 31))) continue;
      if (block_t == 0 && bt > 32 && bt >= M + 32) break;
      if (block_t == 0 && bt == 32 && M > 1024) continue;      // one store per 32 tokens and 32 columns
      const double tiles = static_cast<double>((N + kTileW * g - 1) / (kTileW * g)) * static_cast<double>((M + t - 1) / t);
      const double rounds = static_cast<double>((static_cast<int64_t>(tiles) + sms / g - 1) / (sms / g));
      if (t > kMaxBlockT && (rounds > 1.0 || block_t != 0)) continue;
      const double w = t / 100.0;
      double stage = g == 1 ? 0.179 + 0.159 * w : 0.223 + 0.058 * w;
      if (g == 1 && stage < 0.256) stage = 0.256;
      const double gate = epilogue == HY3D_EPI_GEGLU ? 1.79 : epilogue == HY3D_EPI_GELU ? 2.23 : 1.0;
      const double operand_mb = tiles * g * static_cast<double>(kblocks) * (kABytes + kEBytes + 256.0 * t / g) / 1e7;
      const double us = 2.98 + rounds * (static_cast<double>(kblocks) * stage + (g == 1 ? 0.253 : 0.403) * w * gate + (gate > 1.0 ? 0.1 : 0.0)) + 0.071 * operand_mb +
                        (g == 2 ? 0.56 : 0.0) + 0.1 * static_cast<double>(M) * static_cast<double>(N) * (epilogue == HY3D_EPI_GEGLU ? 1.0 : 2.0) / 1e6;
      if (us < best.us) { best.us = us; best.block_t = t; best.group = g; }
    }
  }
  return best;
}

// Tile order of launches of several rounds.  Weights fastest: the CTAs share a token block, which comes from HBM once, but
// each of them goes to other weight rows with every tile, loads their scales and bias anew, and neighbours write their
// pieces of the output's rows side by side.  Tokens fastest, a contiguous range for each CTA: the weight rows change once or
// twice a launch, and the tokens are read once per column of weight tiles, from L2 as long as they stay there.  Over 75
// shapes of several rounds, time with weights fastest over time with tokens fastest:
//   GEGLU, codes below 10 MB 0.99 to 1.19, 1.074 on average (3072 x 1280 -> 10240 37.0 -> 34.3 us, 12288 x 640 -> 5120 62.7 -> 56.2);
//     10 to 25 MB 0.97 to 1.12, below 1 where N is under 1024
//   GELU, codes below 10 MB 0.99 to 1.15, 1.045 on average; more 0.87 to 1.07
//   plain, codes below 10 MB, M below 10,000 and K below 1600 0.975 to 1.12, 1.049 on average; the others 0.82 to 1.10, since
//     the output's stream displaces the tokens (49152 x 640 -> 640 27.6 us and 31.9)
bool tokens_fastest(int64_t M, int64_t N, int64_t K, int epilogue, bool rounds) {
  const int64_t codes = M * K;
  if (!rounds) return false;
  if (epilogue == HY3D_EPI_GEGLU && N >= 1024) return codes < 25000000;
  if (epilogue != HY3D_EPI_LINEAR) return codes < 10000000;
  return codes < 10000000 && M < 10000 && K < 1600;
}

}  // namespace

// The same for a sparse layer, whose GEMM waits more for the change of split, most of all where it is a single round of
// the grid: 1138 x 640 -> 3600 8.3 us, 9.3 with L1; 584 x 2752 -> 2064 10.2 and 11.2 (inputs in L2), 4375 x 1088 -> 528 12.2
// and 10.7 (from HBM).  More rounds gain from a million elements on (2 to 4 million 0.97 of the time), one from three.
double sparse_l1_elements(int64_t M, int64_t N, int64_t K, int epilogue, int block_t) {
  constexpr double kRounds = 1e6, kSingleRound = 3e6;
  const double elements = static_cast<double>(M) * static_cast<double>(K);
  if (M <= 0 || N <= 0 || K <= 0 || elements < kRounds || elements >= kSingleRound) return kRounds;
  const int sms = planned_sms();
  const SparseTile t = search_tile(M, N, K, epilogue, block_t, sms);
  const int64_t tiles = t.block_t > 0 ? (N + kTileW * t.group - 1) / (kTileW * t.group) * ((M + t.block_t - 1) / t.block_t) : 0;
  return tiles * t.group <= sms ? kSingleRound : kRounds;
}

// Expected time of a layer that quantises and multiplies in separate launches, in microseconds: the greater of
// the device's and the calling thread's (7.5).  The coefficients were fitted over an earlier tile model; against calls of
// today's library they are 10 % rms off where a layer waits for the device.  (That the search may answer with one round of 256
// tokens changes no choice between one launch and two: 400,000 random sizes, M to 24,000, N to 48,000, K to 16,384.)
double sparse_layer_us(int64_t M, int64_t N, int64_t K) {
  const double us = 1.271 * search_tile(M, N, K, HY3D_EPI_LINEAR, 0, planned_sms()).us + 0.424 * static_cast<double>(M) * K / 1e6 - 0.08;
  return us > 7.5 ? us : 7.5;
}

namespace {

// A launch's tiles and walk.
struct SparsePlan {
  int block_t = 0, group = 1;
  int w_tiles = 0, t_tiles = 0, total_tiles = 0;
  int clusters = 0;           // CTAs, or pairs
  bool in_ranges = false;     // tokens fastest
};
int plan_launch(int64_t M, int64_t N, int64_t K, int epilogue, int cta_group, int block_t, int sms, SparsePlan* p) {
#ifdef HY3D_TRACE
  if (const char* e = getenv("HY3D_SPARSE_CTA_GROUP")) cta_group = atoi(e) == 2 ? 2 : 1;
#endif
  const SparseTile tile = search_tile(M, N, K, epilogue, block_t, sms, cta_group);
  p->block_t = tile.block_t;
  p->group = tile.group;
  if (p->block_t < 16 || p->block_t > kWideBlockT || (p->block_t & 15)) return HY3D_ERR_SHAPE;
  p->w_tiles = static_cast<int>((N + kTileW * p->group - 1) / (kTileW * p->group));
  p->t_tiles = static_cast<int>((M + p->block_t - 1) / p->block_t);
  p->total_tiles = p->w_tiles * p->t_tiles;
  const int most = sms / p->group;
  p->clusters = p->total_tiles < most ? p->total_tiles : most;
  // The second accumulator buffer of so wide a tile would lie on the metadata columns and beyond the allocation.
  if (p->block_t > kMaxBlockT && p->total_tiles > p->clusters) return HY3D_ERR_SHAPE;
  p->in_ranges = tokens_fastest(M, N, K, epilogue, p->total_tiles > p->clusters);
  return HY3D_OK;
}

}  // namespace

// The plan of a launch in whole numbers (hy3d_gemm_plan).
int sparse_gemm_plan(int64_t M, int64_t N, int64_t K, int epilogue, int cta_group, int block_t, int sms, int* out) {
  if (N <= 0 || (N & 15) || K <= 0 || (K & 63)) return HY3D_ERR_SHAPE;
  SparsePlan plan;
  const int rc = plan_launch(M, N, K, epilogue, cta_group, block_t, sms, &plan);
  if (rc != HY3D_OK) return rc;
  out[0] = plan.block_t;
  out[1] = plan.group;
  out[2] = plan.clusters;
  out[3] = (plan.total_tiles + plan.clusters - 1) / plan.clusters;
  out[4] = plan.in_ranges ? 1 : 0;
  return HY3D_OK;
}

int gemm_sparse24(const int8_t* X, const float* act_scale, const int8_t* w_comp,
                  const uint32_t* w_meta, int64_t meta_ld, const void* w_scale, int ws_dtype,
                  const void* bias, int bias_dtype, void* out, int out_dtype, int64_t M, int64_t N,
                  int64_t K, int epilogue, int block_t, cudaStream_t stream) {
  if (out_dtype != HY3D_F16 && out_dtype != HY3D_BF16 && out_dtype != HY3D_S32) return HY3D_ERR_ARG;
  if (epilogue < HY3D_EPI_LINEAR || epilogue > HY3D_EPI_GEGLU) return HY3D_ERR_ARG;
  if (out_dtype == HY3D_S32 && epilogue != HY3D_EPI_LINEAR) return HY3D_ERR_ARG;
  if (ws_dtype < HY3D_F16 || ws_dtype > HY3D_F32) return HY3D_ERR_ARG;
  if (bias && (bias_dtype < HY3D_F16 || bias_dtype > HY3D_F32)) return HY3D_ERR_ARG;
  if (M < 0 || N <= 0 || K <= 0 || (K & 63) || (N & 15)) return HY3D_ERR_SHAPE;
  if (M > (1 << 30) || N > (1 << 30) || K > (1 << 30)) return HY3D_ERR_SHAPE;
  if (epilogue == HY3D_EPI_GEGLU && (N & 31)) return HY3D_ERR_SHAPE;
  const int64_t kblocks = (K + kBlockK - 1) / kBlockK;
  if (meta_ld != 4 * ((K + 127) / 128)) return HY3D_ERR_SHAPE;   // rows padded to 128-deep K blocks
  if (M == 0) return HY3D_OK;
  if (!X || !w_comp || !w_meta || !out) return HY3D_ERR_ARG;
  if (out_dtype != HY3D_S32 && (!act_scale || !w_scale)) return HY3D_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(w_comp) |
       reinterpret_cast<uintptr_t>(w_meta) | reinterpret_cast<uintptr_t>(out)) & 15)
    return HY3D_ERR_SHAPE;

  const int sms = device_sm_count();
  if (sms <= 0) return HY3D_ERR_CUDA;
  SparsePlan plan;
  int rc = plan_launch(M, N, K, epilogue, 0, block_t, sms, &plan);
  if (rc != HY3D_OK) return rc;
  block_t = plan.block_t;
  const int group = plan.group, clusters = plan.clusters;

  SparseArgs p;
  p.act_scale = act_scale; p.w_scale = w_scale; p.bias = bias; p.out = out;
  p.ws_dtype = ws_dtype; p.bias_dtype = bias_dtype; p.out_dtype = out_dtype; p.epilogue = epilogue;
  p.M = static_cast<int>(M); p.N = static_cast<int>(N); p.K = static_cast<int>(K);
  p.block_t = block_t;
  p.total_tiles = plan.total_tiles;
  p.num_kb = static_cast<int>(kblocks);
  const int k_last = static_cast<int>(K - (kblocks - 1) * kBlockK);
  p.last_ksteps = (k_last + 63) / 64;
  const int stage_bytes = kABytes + kEBytes + (block_t / group) * kBlockK;
  p.tma_store = (out_dtype != HY3D_S32 && block_t % kSlabTokens == 0) ? 1 : 0;
  const int fixed = static_cast<int>(sizeof(SparseCtrl)) + kEpiWarps * kSlabBytes;
  int stages = (kSmemLimit - fixed) / stage_bytes;
  if (stages > kMaxStages) stages = kMaxStages;
  if (stages < 2) return HY3D_ERR_SHAPE;
  p.stages = stages;
  // One CTA per SM: the kernel allocates all 512 tensor-memory columns, so a second
  // resident CTA would wait for them.  Keep the footprint above half an SM's shared memory.
  int smem_bytes = stages * stage_bytes + fixed;
  if (smem_bytes < 120 * 1024) smem_bytes = 120 * 1024;

  CUtensorMap tm_w, tm_e, tm_x, tm_o;
  rc = encode_tmap_2d_u8(&tm_w, w_comp, static_cast<uint64_t>(K / 2), static_cast<uint64_t>(N),
                             static_cast<uint64_t>(K / 2), 128, kTileW, 128);
  if (rc != HY3D_OK) return rc;
  rc = encode_tmap_2d_u8(&tm_e, w_meta, static_cast<uint64_t>(meta_ld * 4), static_cast<uint64_t>(N),
                         static_cast<uint64_t>(meta_ld * 4), 16, kTileW, 0);
  if (rc != HY3D_OK) return rc;
  rc = encode_tmap_2d_u8(&tm_x, X, static_cast<uint64_t>(K), static_cast<uint64_t>(M),
                         static_cast<uint64_t>(K), 128, static_cast<uint32_t>(block_t / group), 128);
  if (rc != HY3D_OK) return rc;

  if (p.tma_store) {
    // A warp's slab is 32 tokens x 32 weight rows = 64 output bytes per token, or 16 outputs =
    // 32 bytes per token after the GEGLU gate.
    const bool geglu = epilogue == HY3D_EPI_GEGLU;
    const uint64_t row_bytes = static_cast<uint64_t>(geglu ? N / 2 : N) * 2;
    rc = encode_tmap_2d_u8(&tm_o, out, row_bytes, static_cast<uint64_t>(M), row_bytes, geglu ? 32 : 64,
                           kSlabTokens, geglu ? 32 : 64);
    if (rc != HY3D_OK) return rc;
  } else {
    tm_o = tm_x;   // unused by the kernel
  }

  using KernelFn = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap,
                            const CUtensorMap, const SparseArgs);
#define HY3D_SPARSE_ROW(G)                                                                                     \
  {{gemm_sparse_kernel<G, false, HY3D_EPI_LINEAR>, gemm_sparse_kernel<G, false, HY3D_EPI_GELU>,              \
    gemm_sparse_kernel<G, false, HY3D_EPI_GEGLU>},                                                            \
   {gemm_sparse_kernel<G, true, HY3D_EPI_LINEAR>, gemm_sparse_kernel<G, true, HY3D_EPI_GELU>,                \
    gemm_sparse_kernel<G, true, HY3D_EPI_GEGLU>}}
  static const KernelFn kernels[2][2][3] = {HY3D_SPARSE_ROW(1), HY3D_SPARSE_ROW(2)};
#undef HY3D_SPARSE_ROW
  const KernelFn kernel = kernels[group - 1][out_dtype == HY3D_BF16 ? 1 : 0][epilogue];
  rc = ensure_max_smem(reinterpret_cast<const void*>(kernel), kSmemLimit);
  if (rc != HY3D_OK) return rc;
  p.fast_tiles = plan.in_ranges ? plan.t_tiles : plan.w_tiles;
  p.share = plan.in_ranges ? p.total_tiles / clusters : 0;
  p.rest = plan.in_ranges ? p.total_tiles - p.share * clusters : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(group * clusters));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem_bytes);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(group);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1] = pdl_attribute();
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  if (cudaLaunchKernelEx(&cfg, kernel, tm_w, tm_e, tm_x, tm_o, p) != cudaSuccess) {
    cudaGetLastError();
    return HY3D_ERR_CUDA;
  }
  return cudaGetLastError() == cudaSuccess ? HY3D_OK : HY3D_ERR_CUDA;
}

}  // namespace sparse

using sparse::gemm_sparse24;
using sparse::sparse_gemm_plan;
using sparse::sparse_l1_elements;
using sparse::sparse_layer_us;

}  // namespace hy3d
