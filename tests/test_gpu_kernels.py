"""GPU parity tests of the CUDA kernels, called through the C ABI (ctypes binding), against
the CPU oracle.  Integer results must be bit-exact; floating-point outputs are compared with
the tolerance written in each test."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import oracle as O
from conftest import as_half

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _runs_as_one_launch(tc, M, N, K, sparse=0):
    """Whether a layer of this size takes the one-launch kernel (outside a graph capture)."""
    block_t, ks = ctypes.c_int(0), ctypes.c_int(0)
    return tc._lib.hy3d_linear_cluster_plan(M, N, K, sparse, ctypes.byref(block_t), ctypes.byref(ks)) == 1


# ------------------------------------------------------------------ activation quantiser
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K", [(257, 320), (1000, 640), (333, 1280), (64, 2560), (77, 5120),
                                 (924, 1024), (9, 64), (5, 8), (3, 16384), (1, 320), (4096, 320)])
def test_quantize_rows_bit_exact(ik, dtype, M, K):
    x, _, _ = O.make_case(M, K, 16, seed=M * 7 + K, dtype=dtype)
    if M > 8:
        x[3] = 0                                   # all-zero token
        x[4] = x[4] * 1e-4                         # tiny row: scale far below 1
    q, s = ik.fused_quantize_activation(x.to(DEV))
    qo, so = O.quantize_activation(x)
    assert torch.equal(s.cpu(), so)
    assert torch.equal(q.cpu(), qo)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_quantizer_rounding_is_exact_for_every_16_bit_input(ik, dtype):
    """The kernel refines x * rcp(scale) instead of dividing.  Its inputs are 16-bit, so the
    claim "codes equal rint(x / scale)" is checked by enumeration on the device: every amax
    pattern x every x pattern with |x| <= amax, against IEEE division."""
    pairs, bad = ik.quantizer_enum_check(dtype)
    assert pairs > 1_000_000_000
    assert bad == 0


def test_quantize_rounding_boundaries(ik):
    """Values that sit exactly on, or one ulp beside, a x.5 quotient."""
    K = 256
    x = torch.zeros(64, K, dtype=torch.float16)
    x[:, 0] = 127.0                                # scale exactly 1
    vals = torch.arange(-126, 126, dtype=torch.float32) + 0.5       # 252 exact ties
    x[0, 1:253] = vals.half()
    x[1, 1:253] = (vals + 0.0625).half()                            # just above the tie
    x[3, 1:253] = (vals - 0.0625).half()                            # just below
    x[2, 0] = 63.5                                 # scale 0.5: every multiple of .25 is a tie
    x[2, 1:] = (torch.arange(K - 1) * 0.25 - 30).half()
    q, s = ik.fused_quantize_activation(x.to(DEV))
    qo, so = O.quantize_activation(x)
    assert torch.equal(q.cpu(), qo) and torch.equal(s.cpu(), so)


def test_quantize_matches_reference_golden(ik, golden):
    for tag in "abc":
        x = as_half(golden[f"{tag}_x"])
        q, _ = ik.fused_quantize_activation(x.to(DEV))
        assert torch.equal(q.cpu(), torch.from_numpy(golden[f"{tag}_x_int8"]))


def test_quantize_rejects_bad_arguments(ik):
    with pytest.raises(RuntimeError):
        ik.fused_quantize_activation(torch.zeros(4, 12, dtype=torch.float16, device=DEV))   # K % 8
    with pytest.raises(RuntimeError):
        ik.fused_quantize_activation(torch.zeros(4, 16, dtype=torch.float32, device=DEV))
    q, s = ik.fused_quantize_activation(torch.zeros(0, 64, dtype=torch.float16, device=DEV))
    assert q.shape == (0, 64) and s.shape == (0,)


# ------------------------------------------------------------------ prune / compress / pack
@pytest.mark.parametrize("N,K", [(4, 8), (64, 256), (320, 1280), (1280, 320), (128, 64), (16, 36),
                                 (640, 2560)])
def test_prune_compress_bit_exact(sp, N, K):
    g = torch.Generator().manual_seed(N + K)
    w = torch.randint(-128, 128, (N, K), dtype=torch.int8, generator=g)
    w[:, : K // 2] = torch.randint(-3, 4, (N, K // 2), dtype=torch.int8, generator=g)   # ties
    comp, raw = sp.sparse_prune_compress(w.to(DEV))
    co, no = O.prune_compress(w)
    assert torch.equal(comp.cpu(), co)
    assert raw.shape == (N * K // 4,) and raw.dtype == torch.uint8
    assert torch.equal(raw.cpu().view(N, -1), no)
    if K % 32 == 0:
        comp2, meta = sp.sparse_prune_and_pack(w.to(DEV))
        assert meta.dtype == torch.int32 and meta.shape == (N, 4 * ((K + 127) // 128))
        assert torch.equal(comp2.cpu(), co)
        assert torch.equal(meta.cpu(), O.pack_metadata(no, meta.shape[1]))


def test_prune_known_answer_from_reference_tests(sp, golden):
    comp, raw = sp.sparse_prune_compress(torch.from_numpy(golden["kat_prune_w"]).to(DEV))
    assert torch.equal(comp.cpu(), torch.from_numpy(golden["kat_prune_comp"]))
    assert raw.cpu().tolist() == golden["kat_prune_nibbles"].tolist()


# ------------------------------------------------------------------ dense GEMM
def _rand_i8(shape, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randint(-128, 128, shape, dtype=torch.int8, generator=g)


@pytest.mark.parametrize("M,K,N,bn", [
    (128, 32, 16, 0), (128, 64, 64, 0), (128, 128, 128, 0), (128, 256, 256, 0), (128, 320, 160, 0),
    (100, 320, 320, 0), (256, 640, 640, 0), (4096, 320, 1280, 0), (4096, 320, 1280, 128),
    (777, 1024, 320, 0), (3072, 5120, 1280, 0), (1, 64, 16, 0), (3, 1280, 1280, 0), (31, 192, 48, 0),
    (257, 1536, 1536, 0), (924, 1024, 640, 0), (2000, 320, 2560, 208), (500, 64, 272, 0),
    (130, 16, 16, 0), (640, 2560, 640, 80),
])
def test_dense_accumulators_bit_exact(tc, M, K, N, bn):
    A, B = _rand_i8((M, K), M + K), _rand_i8((N, K), N + K + 1)
    acc = tc.int8_gemm_tc(A.to(DEV), B.to(DEV), None, None, None, out_dtype=torch.int32, block_n=bn)
    assert torch.equal(acc.cpu(), O.int32_matmul(A, B))


def _dense_by_slices(tc, A, B, a_s, w_s, bias):
    """The layer's output from single-CTA launches of 2048 rows: fewer than two tiles per CTA, so both operands stream."""
    return torch.cat([tc.int8_gemm_tc(A[i:i + 2048], B, a_s[i:i + 2048], w_s, bias, out_dtype=torch.bfloat16, cta_group=1)
                      for i in range(0, A.shape[0], 2048)])


@pytest.mark.parametrize("M,K,N,bn", [
    (40000, 192, 256, 0),     # one tile column, 313 row tiles (last one ragged), two K blocks
    (38000, 320, 640, 0),     # three columns of 224; ragged last K block
    (37900, 640, 160, 160),   # five K blocks resident
    (40000, 320, 2560, 256),  # ten columns
    (39000, 1024, 128, 128),  # eight K blocks: the fewest A stages (four) fit beside them
    (39000, 1040, 128, 128),  # nine do not leave four: both operands stream
])
def test_dense_resident_b_tile_bit_exact(tc, M, K, N, bn):
    """Launches that keep one tile column per CTA with at least two tiles each load their B tile
    once and stream only A (single-CTA tiles; two to eight K
    blocks, ragged last row tile, ragged last K block, one and several tile columns)."""
    A, B = _rand_i8((M, K), M + K + 5), _rand_i8((N, K), N + K + 6)
    acc = tc.int8_gemm_tc(A.to(DEV), B.to(DEV), None, None, None, out_dtype=torch.int32,
                          cta_group=1, block_n=bn)
    assert torch.equal(acc.cpu(), O.int32_matmul(A, B))
    g = torch.Generator().manual_seed(M)
    a_s = torch.rand(M, generator=g) * 0.05 + 1e-3
    w_s = (torch.rand(N, generator=g) * 1e-3 + 1e-5).bfloat16()
    bias = (torch.randn(N, generator=g) * 0.1).bfloat16()
    y = tc.int8_gemm_tc(A.to(DEV), B.to(DEV), a_s.to(DEV), w_s.to(DEV), bias.to(DEV),
                        out_dtype=torch.bfloat16, cta_group=1, block_n=bn)
    ref = O.epilogue(O.int32_matmul(A, B), a_s, w_s, bias, torch.bfloat16, "linear")
    assert O.rel_l2(y, ref) < 2e-3          # same accumulators and formula; fma contraction only
    # and the resident-B launch equals streaming ones, and pairs, bit for bit
    operands = (A.to(DEV), B.to(DEV), a_s.to(DEV), w_s.to(DEV), bias.to(DEV))
    assert torch.equal(y, _dense_by_slices(tc, *operands))
    assert torch.equal(y, tc.int8_gemm_tc(*operands, out_dtype=torch.bfloat16, cta_group=2, block_n=bn))
    assert tc.device_status() == 0


@pytest.mark.parametrize("M,K,N,bn", [
    (40000, 320, 320, 160),   # two columns of pairs, K ends in half a block
    (38001, 640, 1280, 256),  # five columns, five K blocks, seven A stages; ragged last row tile
    (39000, 976, 192, 192),   # one column, eight K blocks of which the last has three steps, six A stages
    (39000, 1008, 256, 256),  # the most that pairs with one block a stage keep: four A stages beside eight blocks
    (38100, 336, 176, 0),     # the library's own width; last K block of three steps, columns clipped
])
def test_dense_resident_b_tile_of_pairs_bit_exact(tc, M, K, N, bn):
    """CTA pairs that keep their tile column hold half of the B tile each (K < 1024): integer sums of the oracle, and
    the same bits as single CTAs that stream both operands and as the library's own choice."""
    A, B = _rand_i8((M, K), M + K + 7), _rand_i8((N, K), N + K + 8)
    acc = tc.int8_gemm_tc(A.to(DEV), B.to(DEV), None, None, None, out_dtype=torch.int32, cta_group=2, block_n=bn)
    assert torch.equal(acc.cpu(), O.int32_matmul(A, B))
    g = torch.Generator().manual_seed(M)
    a_s, w_s = torch.rand(M, generator=g) * 0.05 + 1e-3, (torch.rand(N, generator=g) * 1e-3 + 1e-5).bfloat16()
    operands = (A.to(DEV), B.to(DEV), a_s.to(DEV), w_s.to(DEV), None)
    y = tc.int8_gemm_tc(*operands, out_dtype=torch.bfloat16, cta_group=2, block_n=bn)
    assert torch.equal(y, _dense_by_slices(tc, *operands)) and torch.equal(y, tc.int8_gemm_tc(*operands, out_dtype=torch.bfloat16))
    assert tc.device_status() == 0


@pytest.mark.parametrize("M,K,N,bn", [
    (2600, 2064, 512, 0),     # K = 8 deep stages + a 16-element tail; ragged last row tile
    (300, 1024, 256, 256),    # exactly four deep stages, second CTA's rows half empty
    (1000, 1104, 320, 160),   # tail of 80: three K steps of the first block
    (513, 5120, 1280, 224),   # ragged tile columns (1280 = 5 x 224 + 160)
    (256, 320, 640, 128),     # short K with pairs: single 128-byte blocks per stage
])
def test_dense_cta_pairs_bit_exact(tc, M, K, N, bn):
    """The CTA-pair variant (cta_group = 2: 256-row tiles; deep two-block stages from K = 1024)."""
    A, B = _rand_i8((M, K), M + K + 2), _rand_i8((N, K), N + K + 3)
    acc = tc.int8_gemm_tc(A.to(DEV), B.to(DEV), None, None, None, out_dtype=torch.int32,
                          cta_group=2, block_n=bn)
    assert torch.equal(acc.cpu(), O.int32_matmul(A, B))
    assert tc.device_status() == 0


def test_dense_extreme_values_no_overflow(tc):
    """|acc| reaches 128*128*K: the int32 accumulators must not saturate or wrap."""
    M, K, N = 128, 5120, 64
    A = torch.full((M, K), -128, dtype=torch.int8)
    B = torch.full((N, K), -128, dtype=torch.int8)
    B[1::2] = 127
    acc = tc.int8_gemm_tc(A.to(DEV), B.to(DEV), None, None, None, out_dtype=torch.int32)
    assert torch.equal(acc.cpu(), A.int() @ B.int().t())
    assert int(acc.max()) == 128 * 128 * K


def test_dense_single_tile_known_answer(tc):
    a = torch.ones(128, 32, dtype=torch.int8)
    b = torch.ones(16, 32, dtype=torch.int8)
    d = tc.test_mma(a.to(DEV), b.to(DEV))
    assert d.shape == (128, 16) and bool((d == 32).all())
    a2, b2 = _rand_i8((128, 128), 1), _rand_i8((256, 128), 2)
    assert torch.equal(tc.test_mma(a2.to(DEV), b2.to(DEV)).cpu(), a2.int() @ b2.int().t())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("mode,code", [("linear", 0), ("gelu", 1), ("geglu", 2)])
@pytest.mark.parametrize("M,K,N", [(300, 320, 1280), (1000, 640, 320), (64, 1280, 2560)])
def test_dense_epilogue_matches_oracle(tc, dtype, mode, code, M, K, N):
    A, B = _rand_i8((M, K), 11), _rand_i8((N, K), 12)
    g = torch.Generator().manual_seed(13)
    a_s = torch.rand(M, generator=g) * 0.05 + 1e-3
    w_s = (torch.rand(N, generator=g) * 1e-3 + 1e-5).to(dtype)
    bias = (torch.randn(N, generator=g) * 0.1).to(dtype)
    y = tc.int8_gemm_tc(A.to(DEV), B.to(DEV), a_s.to(DEV), w_s.to(DEV), bias.to(DEV),
                        out_dtype=dtype, epilogue=code)
    ref = O.epilogue(O.int32_matmul(A, B), a_s, w_s, bias, dtype, mode)
    assert y.shape == ref.shape and y.dtype == dtype
    # same int32 accumulators, same formula: only the final rounding (and fma contraction /
    # erf implementation, ~1e-6) can differ -> far inside the 1e-2 gate
    assert O.rel_l2(y, ref) < 2e-3
    y0 = tc.int8_gemm_tc(A.to(DEV), B.to(DEV), a_s.to(DEV), w_s.to(DEV), torch.empty(0, dtype=dtype, device=DEV),
                         out_dtype=dtype, epilogue=code)
    assert O.rel_l2(y0, O.epilogue(O.int32_matmul(A, B), a_s, w_s, None, dtype, mode)) < 2e-3


def test_dense_linear_config0(tc):
    """Config 0 of the benchmark: X bf16 [4096,320], W bf16 [1280,320], bias bf16 [1280]."""
    g = torch.Generator().manual_seed(0)
    x = torch.randn(4096, 320, generator=g).bfloat16()
    w = (torch.randn(1280, 320, generator=g) * 0.02).bfloat16()
    b = (torch.randn(1280, generator=g) * 0.01).bfloat16()
    wq, ws = O.quantize_weight(w)
    y = tc.int8_linear_tc(x.to(DEV), wq.to(DEV), ws.bfloat16().to(DEV), b.to(DEV))
    ref = O.linear_w8a8(x, wq, ws.bfloat16(), b)
    assert y.shape == (4096, 1280) and y.dtype == torch.bfloat16
    assert O.rel_l2(y, ref) < 1e-2                      # the stated output gate
    assert O.rel_l2(y, ref) < 1e-4                      # what identical accumulators give
    assert O.rel_l2(y, x.float() @ w.float().t() + b.float()) < 2e-2   # vs unquantised math


def test_dense_rejects_bad_arguments(tc):
    A = torch.zeros(128, 40, dtype=torch.int8, device=DEV)     # K % 16 != 0
    B = torch.zeros(16, 40, dtype=torch.int8, device=DEV)
    with pytest.raises(RuntimeError, match="size|alignment"):
        tc.int8_gemm_tc(A, B, None, None, None, out_dtype=torch.int32)
    A = torch.zeros(128, 64, dtype=torch.int8, device=DEV)
    B = torch.zeros(24, 64, dtype=torch.int8, device=DEV)      # N % 16 != 0
    with pytest.raises(RuntimeError):
        tc.int8_gemm_tc(A, B, None, None, None, out_dtype=torch.int32)
    B = torch.zeros(16, 64, dtype=torch.int8, device=DEV)
    with pytest.raises(RuntimeError):                          # scales missing for a float output
        tc.int8_gemm_tc(A, B, None, None, None, out_dtype=torch.float16)
    with pytest.raises(RuntimeError, match="K mismatch"):
        tc.int8_gemm_tc(A, torch.zeros(16, 128, dtype=torch.int8, device=DEV), None, None, None,
                        out_dtype=torch.int32)


def test_dequant_bias_kernel(ik):
    g = torch.Generator().manual_seed(3)
    acc = torch.randint(-200000, 200000, (257, 320), dtype=torch.int32, generator=g)
    a_s = torch.rand(257, generator=g) * 0.01
    w_s = (torch.rand(320, generator=g) * 1e-3).half()
    b = torch.randn(320, generator=g).half()
    y = ik.fused_dequantize_bias(acc.to(DEV), a_s.to(DEV), w_s.to(DEV), b.to(DEV))
    assert O.rel_l2(y, O.epilogue(acc, a_s, w_s, b, torch.float16)) < 1e-3


# ------------------------------------------------------------------ sparse GEMM
def test_sparse_metadata_layout_probe(sp):
    """X = identity makes the GEMM return the expanded weight itself: every (row, group)
    nibble and every compressed value must land where the 2:4 format says."""
    valid = [0x4, 0x8, 0xC, 0x9, 0xD, 0xE]
    for K in (64, 128, 320):
        N, G = 128, K // 4
        comp = ((torch.arange(K // 2) % 100 + 1)[None, :] + (torch.arange(N) % 20)[:, None]).to(torch.int8)
        nib = torch.tensor([[valid[(r * 7 + g * 5) % 6] for g in range(G)] for r in range(N)],
                           dtype=torch.uint8)
        meta = O.pack_metadata(nib, 4 * ((K + 127) // 128))
        out = sp.sparse_int8_gemm(torch.eye(K, dtype=torch.int8).to(DEV), None, comp.to(DEV),
                                  meta.to(DEV), None, None, out_dtype=torch.int32)
        assert torch.equal(out.cpu(), O.expand_24(comp, nib).int().t().contiguous())


def test_sparse_tile_known_answer_from_reference_tests(sp, golden):
    """The seed-42 random 2:4 tile of the reference's mma.sp test, padded to one tcgen05 tile
    (128 rows, K = 64)."""
    a_comp = torch.zeros(128, 32, dtype=torch.int8)
    a_comp[:16, :16] = torch.from_numpy(golden["kat_mma_a_comp"])
    nib = torch.full((128, 16), 0x4, dtype=torch.uint8)
    nib[:16, :8] = torch.from_numpy(golden["kat_mma_nibbles"])
    b = torch.zeros(16, 64, dtype=torch.int8)
    b[:8, :32] = torch.from_numpy(golden["kat_mma_b"])
    d = sp.test_mma_sp(a_comp.to(DEV), b.to(DEV), O.pack_metadata(nib, 4).to(DEV))
    assert d.shape == (128, 16)
    assert torch.equal(d.cpu()[:16, :8], torch.from_numpy(golden["kat_mma_c"]))
    assert int(d.cpu()[16:].abs().max()) == 0
    ones = sp.test_mma_sp(torch.ones(128, 32, dtype=torch.int8, device=DEV),
                          torch.ones(16, 64, dtype=torch.int8, device=DEV),
                          torch.full((128, 4), 0x44444444, dtype=torch.int32, device=DEV))
    assert bool((ones == 32).all())                  # 32 surviving products per output


@pytest.mark.parametrize("M,K,N,bt", [
    (192, 128, 128, 0), (1000, 640, 640, 0), (3072, 1280, 1280, 0), (924, 1024, 320, 0),
    (4096, 320, 320, 0), (12288, 2560, 640, 240), (3, 1280, 1280, 0), (64, 640, 5120, 0),
    (257, 1536, 4608, 0), (500, 64, 16, 0), (2772, 1024, 320, 128), (1, 64, 16, 0),
    (700, 5120, 1280, 224),
    (2304, 1024, 512, 0), (2100, 2560, 640, 0),
    # CTA pairs (256 weight rows per tile), full and ragged tiles, deep K and short
    (2500, 2560, 1312, 0), (3000, 1280, 1296, 192), (2048, 5120, 1280, 64), (8119, 576, 1696, 0), (13021, 896, 672, 0),
])
def test_sparse_accumulators_bit_exact(sp, M, K, N, bt):
    X, W = _rand_i8((M, K), M + K), _rand_i8((N, K), N + K + 5)
    comp, meta = sp.sparse_prune_and_pack(W.to(DEV))
    acc = sp.sparse_int8_gemm(X.to(DEV), None, comp, meta, None, None, out_dtype=torch.int32,
                              force_tile=bt)
    co, no = O.prune_compress(W)
    assert torch.equal(acc.cpu(), O.int32_matmul(X, O.expand_24(co, no)))


# GEGLU in contiguous ranges down the tile columns: B loaded again inside a range, ragged rows, columns and last K stages,
# single CTAs and pairs, the library's own tile and given ones, both types, against the direct-store form (32-column tiles
# walk strided).  The plan tells that these sizes do walk in ranges on 148 SMs; the last two walk strided.
@pytest.mark.parametrize("M,K,N,group,bn,ranges", [
    (24576, 320, 2560, 0, 0, 1), (12288, 640, 5120, 0, 0, 1), (4219, 1008, 5664, 0, 0, 1), (5000, 512, 4096, 1, 192, 1), (4750, 272, 1888, 1, 128, 1),
    (5003, 272, 1888, 1, 64, 1), (3000, 128, 5120, 1, 64, 1), (9001, 400, 1312, 2, 64, 1), (3073, 640, 3968, 2, 256, 1), (3073, 624, 3968, 2, 256, 1),
    (5003, 272, 1888, 1, 128, 0), (49152, 64, 192, 1, 64, 0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_dense_geglu_ranges(tc, M, K, N, group, bn, ranges, dtype):
    sms, plan = torch.cuda.get_device_properties(0).multi_processor_count, (ctypes.c_int * 5)()
    assert tc._lib.hy3d_gemm_plan(M, N, K, 2, 0, group, bn, 0, plan) == 0
    assert plan[4] == ranges or sms != 148
    A, B = _rand_i8((M, K), M + K).to(DEV), _rand_i8((N, K), N + K + 5).to(DEV)
    g = torch.Generator().manual_seed(33)
    a_s, w_s = (torch.rand(M, generator=g) * 0.05 + 1e-3).to(DEV), (torch.rand(N, generator=g) * 1e-4 + 1e-5).to(dtype).to(DEV)
    bias = (torch.randn(N, generator=g) * 0.1).to(dtype).to(DEV)
    for _ in range(3):
        y = tc.int8_gemm_tc(A, B, a_s, w_s, bias, out_dtype=dtype, epilogue=2, cta_group=group, block_n=bn)
        assert torch.equal(y, tc.int8_gemm_tc(A, B, a_s, w_s, bias, out_dtype=dtype, epilogue=2, cta_group=1, block_n=32))


# Tokens fastest in contiguous ranges: a range that ends inside a column of weight tiles, at its end and beyond it, ragged last
# tiles both ways, more columns than CTAs, pairs and single CTAs; widths that the cost model does not choose.
@pytest.mark.parametrize("M,K,N,bt", [(3072, 1280, 10240, 0), (1500, 640, 10240, 0), (4444, 640, 3040, 0), (2000, 1024, 4096, 160),
                                      (333, 320, 20000, 0), (9000, 384, 1056, 64), (1100, 128, 9600, 32)])
def test_sparse_token_ranges(sp, M, K, N, bt):
    X, W = _rand_i8((M, K), M + K).to(DEV), _rand_i8((N, K), N + K + 5).to(DEV)
    comp, meta = sp.sparse_prune_and_pack(W)
    acc = sp.sparse_int8_gemm(X, None, comp, meta, None, None, out_dtype=torch.int32, force_tile=bt)
    rows = torch.cat([torch.arange(2), torch.arange(M - 20, M), torch.randperm(M, generator=torch.Generator().manual_seed(M))[:40]])
    assert torch.equal(acc[rows.to(DEV)].cpu(), O.int32_matmul(X[rows.to(DEV)].cpu(), O.expand_24(*O.prune_compress(W.cpu()))))
    g = torch.Generator().manual_seed(33)
    a_s, w_s = (torch.rand(M, generator=g) * 0.05 + 1e-3).to(DEV), (torch.rand(N, generator=g) * 1e-4 + 1e-5).bfloat16().to(DEV)
    bias = (torch.randn(N, generator=g) * 0.1).bfloat16().to(DEV)
    base = torch.addcmul(bias.double(), acc.double(), (a_s[:, None] * w_s.float()[None]).double()).float()   # one rounding, as fma
    for epi in (0, 1, 2):
        y = sp.sparse_int8_gemm(X, a_s, comp, meta, w_s, bias, out_dtype=torch.bfloat16, epilogue=epi, force_tile=bt)
        if epi == 0:
            ref = base
        elif epi == 1:
            ref = torch.nn.functional.gelu(base)
        else:
            v, gate = base.view(M, N // 32, 2, 16).unbind(2)
            ref = (v * torch.nn.functional.gelu(gate)).reshape(M, N // 2)
        assert O.rel_l2(y, ref) < 2.5e-3      # one rounding to bf16: 2^-9 / sqrt(3) on average, 1.2e-3


# 256-token tiles with one accumulator buffer: launches of one round, pairs (2817 tokens and more) and single CTAs, whole and
# ragged tiles, deep K and K of a block and less.
@pytest.mark.parametrize("M,K,N", [(2817, 2560, 1312), (3072, 640, 1536), (2915, 5120, 1296), (250, 576, 18944), (497, 704, 9216), (256, 64, 18944)])
def test_sparse_one_round_of_wide_tiles(sp, M, K, N):
    X, W = _rand_i8((M, K), M + K).to(DEV), _rand_i8((N, K), N + K + 5).to(DEV)
    comp, meta = sp.sparse_prune_and_pack(W)
    wp = O.expand_24(*O.prune_compress(W.cpu()))
    acc = sp.sparse_int8_gemm(X, None, comp, meta, None, None, out_dtype=torch.int32)
    rows = torch.cat([torch.arange(3), torch.arange(M - 40, M), torch.randperm(M, generator=torch.Generator().manual_seed(M))[:60]])
    assert torch.equal(acc[rows.to(DEV)].cpu(), O.int32_matmul(X[rows.to(DEV)].cpu(), wp))
    g = torch.Generator().manual_seed(33)
    a_s, w_s = (torch.rand(M, generator=g) * 0.05 + 1e-3).to(DEV), (torch.rand(N, generator=g) * 1e-3 + 1e-5).bfloat16().to(DEV)
    bias = (torch.randn(N, generator=g) * 0.1).bfloat16().to(DEV)
    for epi in (0, 1, 2) if N % 32 == 0 else (0, 1):      # the epilogue is the narrow tiles': the same bits
        y = sp.sparse_int8_gemm(X, a_s, comp, meta, w_s, bias, out_dtype=torch.bfloat16, epilogue=epi)
        assert torch.equal(y, sp.sparse_int8_gemm(X, a_s, comp, meta, w_s, bias, out_dtype=torch.bfloat16, epilogue=epi, force_tile=128))
    with pytest.raises(RuntimeError):      # 256 is the rule's to choose
        sp.sparse_int8_gemm(X, None, comp, meta, None, None, out_dtype=torch.int32, force_tile=256)


@pytest.mark.parametrize("mode,code", [("linear", 0), ("gelu", 1), ("geglu", 2)])
def test_sparse_pair_variant_epilogues(sp, mode, code):
    """Scaled outputs of the CTA-pair variant: the cost model has pairs of 224 tokens 6 to 12 % ahead of single CTAs here."""
    M, K, N = 2500, 2560, 1312
    A, B = _rand_i8((M, K), 31), _rand_i8((N, K), 32)
    g = torch.Generator().manual_seed(33)
    a_s = torch.rand(M, generator=g) * 0.05 + 1e-3
    w_s = (torch.rand(N, generator=g) * 1e-3 + 1e-5).bfloat16()
    bias = (torch.randn(N, generator=g) * 0.1).bfloat16()
    comp, meta = sp.sparse_prune_and_pack(B.to(DEV))
    y = sp.sparse_int8_gemm(A.to(DEV), a_s.to(DEV), comp, meta, w_s.to(DEV), bias.to(DEV),
                            out_dtype=torch.bfloat16, epilogue=code)
    co, no = O.prune_compress(B)
    ref = O.epilogue(O.int32_matmul(A, O.expand_24(co, no)), a_s, w_s, bias, torch.bfloat16, mode)
    assert y.shape == ref.shape
    assert O.rel_l2(y, ref) < 2e-3


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("mode,code", [("linear", 0), ("gelu", 1), ("geglu", 2)])
def test_sparse_epilogue_matches_oracle(sp, dtype, mode, code):
    M, K, N = 500, 640, 1280
    X, W = _rand_i8((M, K), 21), _rand_i8((N, K), 22)
    g = torch.Generator().manual_seed(23)
    a_s = torch.rand(M, generator=g) * 0.05 + 1e-3
    w_s = (torch.rand(N, generator=g) * 1e-3 + 1e-5).to(dtype)
    bias = (torch.randn(N, generator=g) * 0.1).to(dtype)
    comp, meta = sp.sparse_prune_and_pack(W.to(DEV))
    y = sp.sparse_int8_gemm(X.to(DEV), a_s.to(DEV), comp, meta, w_s.to(DEV), bias.to(DEV),
                            out_dtype=dtype, epilogue=code)
    co, no = O.prune_compress(W)
    ref = O.epilogue(O.int32_matmul(X, O.expand_24(co, no)), a_s, w_s, bias, dtype, mode)
    assert y.shape == ref.shape
    assert O.rel_l2(y, ref) < 2e-3


def test_sparse_rejects_bad_arguments(sp):
    X = torch.zeros(64, 96, dtype=torch.int8, device=DEV)          # K % 64 != 0
    comp = torch.zeros(16, 48, dtype=torch.int8, device=DEV)
    meta = torch.zeros(16, 4, dtype=torch.int32, device=DEV)
    with pytest.raises(RuntimeError):
        sp.sparse_int8_gemm(X, None, comp, meta, None, None, out_dtype=torch.int32)
    X = torch.zeros(64, 128, dtype=torch.int8, device=DEV)
    comp = torch.zeros(16, 64, dtype=torch.int8, device=DEV)
    with pytest.raises(RuntimeError):                               # wrong metadata pitch
        sp.sparse_int8_gemm(X, None, comp, torch.zeros(16, 8, dtype=torch.int32, device=DEV), None,
                            None, out_dtype=torch.int32)


def test_results_are_deterministic(tc, sp):
    A, B = _rand_i8((2048, 640), 31).to(DEV), _rand_i8((640, 640), 32).to(DEV)
    a_s = torch.rand(2048, device=DEV)
    w_s = torch.rand(640, device=DEV).half()
    first = tc.int8_gemm_tc(A, B, a_s, w_s, None)
    comp, meta = sp.sparse_prune_and_pack(B)
    first_sp = sp.sparse_int8_gemm(A, a_s, comp, meta, w_s, None)
    for _ in range(5):
        assert torch.equal(first, tc.int8_gemm_tc(A, B, a_s, w_s, None))
        assert torch.equal(first_sp, sp.sparse_int8_gemm(A, a_s, comp, meta, w_s, None))


def test_output_canaries_untouched(tc, sp):
    """Ragged sizes: nothing may be written outside the (M,N) result."""
    M, K, N = 130, 320, 48
    A, B = _rand_i8((M, K), 41).to(DEV), _rand_i8((N, K), 42).to(DEV)
    lib = tc._lib
    buf = torch.full((M + 2, N), 0x5A5A5A5A, dtype=torch.int32, device=DEV)
    st = lib.hy3d_gemm_w8a8_dense(A.data_ptr(), B.data_ptr(), None, None, 2, None, 0,
                                  buf[1:].data_ptr(), 3, M, N, K, 0, 0, 0,
                                  torch.cuda.current_stream().cuda_stream)
    assert st == 0
    torch.cuda.synchronize()
    assert bool((buf[0] == 0x5A5A5A5A).all()) and bool((buf[M + 1] == 0x5A5A5A5A).all())
    assert torch.equal(buf[1:M + 1].cpu(), O.int32_matmul(A.cpu(), B.cpu()))


def test_bounded_wait_gives_up_and_reports(tc):
    """A device-side wait that can never be satisfied (one thread on a barrier nobody signals,
    wait limit shortened to 2 ms) ends by itself: the kernel returns, the error word holds the
    wait's code, the stream check raises with the timeout status, and the next ordinary GEMM on
    the same context is exact."""
    lib = tc._lib
    stream = torch.cuda.current_stream().cuda_stream
    assert lib.hy3d_set_wait_limit_ns(2_000_000) == 0
    try:
        assert lib.hy3d_wait_selftest(stream) == 0
        assert lib.hy3d_stream_status(stream) == 5            # HY3D_ERR_TIMEOUT
        with pytest.raises(RuntimeError, match="timed out"):
            tc.check_stream()
        assert tc.device_status() == 0                        # cleared by the raise
    finally:
        assert lib.hy3d_set_wait_limit_ns(0) == 0             # back to the default
    assert lib.hy3d_stream_status(stream) == 0
    A = torch.randint(-128, 128, (300, 256), dtype=torch.int8)
    B = torch.randint(-128, 128, (192, 256), dtype=torch.int8)
    acc = tc.int8_gemm_tc(A.to(DEV), B.to(DEV), None, None, None, out_dtype=torch.int32)
    assert torch.equal(acc.cpu(), O.int32_matmul(A, B))
    tc.check_stream()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K", [(4096, 320), (1000, 640), (333, 1280), (77, 1024), (5, 64), (129, 2048), (2500, 96)])
def test_layernorm_quantize_equals_quantising_its_own_output(ik, dtype, M, K):
    """The fused LayerNorm + quantise kernel: (1) its codes and scales are exactly those of the
    stand-alone quantiser (and of the CPU oracle) applied to the normalised activations it
    reports; (2) those activations are the fp32 LayerNorm rounded to the activation type, to
    within a last-place difference of the torch op."""
    g = torch.Generator().manual_seed(M + K)
    x = (torch.randn(M, K, generator=g) * 3 + 0.5).to(dtype)
    gamma = (1 + 0.1 * torch.randn(K, generator=g)).to(dtype)
    beta = (0.1 * torch.randn(K, generator=g)).to(dtype)
    q, s, y = ik.layernorm_quantize(x.to(DEV), gamma.to(DEV), beta.to(DEV), 1e-5, return_normalised=True)
    q2, s2 = ik.fused_quantize_activation(y)
    assert torch.equal(q, q2) and torch.equal(s, s2)
    qo, so = O.quantize_activation(y.cpu())
    assert torch.equal(q.cpu(), qo) and torch.equal(s.cpu(), so)
    ref = torch.nn.functional.layer_norm(x.float(), (K,), gamma.float(), beta.float(), 1e-5)
    assert O.rel_l2(y, ref) < (3e-3 if dtype == torch.bfloat16 else 4e-4)       # one output rounding
    assert float((y.float().cpu() - ref).abs().max()) <= (0.04 if dtype == torch.bfloat16 else 0.005) * float(ref.abs().max())
    # without the normalised output the codes are the same
    q3, s3 = ik.layernorm_quantize(x.to(DEV), gamma.to(DEV), beta.to(DEV), 1e-5)
    assert torch.equal(q3, q) and torch.equal(s3, s)


@pytest.mark.parametrize("batches,rows", [(1, 1), (1, 0), (2, 0), (2, 7)])     # row batches of every block, and rows beyond them
def test_layernorm_quantize_uneven_trips(ik, batches, rows):
    K = 1280                                                                  # eight rows a batch, three blocks an SM
    M = 3 * torch.cuda.get_device_properties(0).multi_processor_count * 8 * batches + rows
    g = torch.Generator(device=DEV).manual_seed(M)
    x = (torch.randn(M, K, generator=g, device=DEV) * 3 + 0.5).bfloat16()
    gamma, beta = 1 + 0.1 * torch.randn(K, generator=g, device=DEV), 0.1 * torch.randn(K, generator=g, device=DEV)
    q, s = ik.layernorm_quantize(x, gamma, beta, 1e-5)
    for lo in range(0, M, 1000):                                              # a block of these makes one trip
        qo, so = ik.layernorm_quantize(x[lo:lo + 1000], gamma, beta, 1e-5)
        assert torch.equal(q[lo:lo + 1000], qo) and torch.equal(s.reshape(-1)[lo:lo + 1000], so.reshape(-1))


def test_layernorm_quantize_without_affine_and_argument_checks(ik):
    x = torch.randn(64, 256).bfloat16().to(DEV)
    q, s, y = ik.layernorm_quantize(x, None, None, 1e-6, return_normalised=True)
    ref = torch.nn.functional.layer_norm(x.float().cpu(), (256,), None, None, 1e-6)
    assert O.rel_l2(y, ref) < 3e-3
    with pytest.raises(RuntimeError):
        ik.layernorm_quantize(torch.randn(8, 4096).bfloat16().to(DEV), None, None, 1e-5)   # K > 2048


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("silu", [False, True])
@pytest.mark.parametrize("shape", [(2, 320, 32, 32), (3, 640, 16, 16), (2, 960, 16, 16), (1, 1280, 8, 8),
                                   (2, 2560, 8, 8), (1, 64, 5, 7), (12, 320, 64, 64),
                                   (300, 64, 4, 4), (700, 64, 3, 5)])   # more samples than one wave of blocks
def test_groupnorm_nhwc_matches_torch_fp32(ik, dtype, silu, shape):
    """The channels-last GroupNorm (+ SiLU) kernel against torch's ops on the same values:
    fp32 group_norm, rounded to the activation type, then (optionally) fp32 SiLU of the rounded
    value, rounded again -- the two-op sequence the kernel replaces.  Floating point: the
    statistics are summed in another order, so outputs may differ in the last place of the
    16-bit type (tolerance: 3e-3 / 4e-4 relative L2 for bf16 / fp16, and no element off by more
    than two units in the last place of the largest output)."""
    B, C, H, W = shape
    g = torch.Generator().manual_seed(C + H)
    x = (torch.randn(B, C, H, W, generator=g) * 2 + 0.7).to(dtype).to(DEV).contiguous(memory_format=torch.channels_last)
    gamma = (1 + 0.2 * torch.randn(C, generator=g)).to(dtype).to(DEV)
    beta = (0.2 * torch.randn(C, generator=g)).to(dtype).to(DEV)
    y = ik.groupnorm_nhwc(x, 32, gamma, beta, 1e-5, silu=silu)
    assert y.shape == x.shape and y.is_contiguous(memory_format=torch.channels_last)
    ref = torch.nn.functional.group_norm(x.float(), 32, gamma.float(), beta.float(), 1e-5).to(dtype)
    if silu:
        ref = torch.nn.functional.silu(ref.float()).to(dtype)
    assert not torch.isnan(y).any()
    assert O.rel_l2(y, ref) < (3e-3 if dtype == torch.bfloat16 else 4e-4)
    ulp = (2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10) * float(ref.float().abs().max())
    assert float((y.float() - ref.float()).abs().max()) <= 2 * ulp
    # in place
    x2 = x.clone(memory_format=torch.channels_last)
    ik.groupnorm_nhwc(x2, 32, gamma, beta, 1e-5, silu=silu, out=x2)
    assert torch.equal(x2, y)
    # with a per-(sample, channel) term added first, rounded as a separate add would store it
    add = (torch.randn(B, C, generator=g) * 0.5).to(dtype).to(DEV)
    ya = ik.groupnorm_nhwc(x, 32, gamma, beta, 1e-5, silu=silu, add=add)
    xa = (x + add[:, :, None, None])
    refa = torch.nn.functional.group_norm(xa.float(), 32, gamma.float(), beta.float(), 1e-5).to(dtype)
    if silu:
        refa = torch.nn.functional.silu(refa.float()).to(dtype)
    assert O.rel_l2(ya, refa) < (3e-3 if dtype == torch.bfloat16 else 4e-4)
    ulpa = (2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10) * float(refa.float().abs().max())
    assert float((ya.float() - refa.float()).abs().max()) <= 2 * ulpa


@pytest.mark.parametrize("shape", [(8, 96, 89, 86), (8, 640, 40, 40), (9, 832, 21, 42)])     # fewer ranks, so that one wave does
def test_groupnorm_nhwc_fewer_ranks(ik, shape):
    B, C, H, W = shape
    g = torch.Generator(device=DEV).manual_seed(C)
    x = (torch.randn(B, C, H, W, generator=g, device=DEV) * 2 + 0.7).bfloat16().contiguous(memory_format=torch.channels_last)
    gamma, beta = 1 + 0.2 * torch.randn(C, generator=g, device=DEV), 0.2 * torch.randn(C, generator=g, device=DEV)
    add = (torch.randn(B, C, generator=g, device=DEV) * 0.5).bfloat16()
    for term in (None, add):
        xs = x if term is None else x + term[:, :, None, None]
        ref = torch.nn.functional.group_norm(xs.float(), 32, gamma, beta, 1e-5).bfloat16()
        y = ik.groupnorm_nhwc(x, 32, gamma, beta, 1e-5, silu=True, add=term)
        assert O.rel_l2(y, torch.nn.functional.silu(ref.float()).bfloat16()) < 3e-3


@pytest.mark.parametrize("shape,add,fewer", [((8, 96, 89, 86), 0, 1), ((8, 640, 40, 40), 0, 1), ((8, 320, 86, 10), 1, 1),       # wide; narrow and small
                                             ((9, 1920, 65, 34), 1, 0), ((9, 960, 44, 81), 1, 0), ((7, 1280, 56, 86), 1, 0),   # narrow and large
                                             ((9, 1920, 40, 17), 1, 0)])                                                        # a twentieth left over
def test_groupnorm_nhwc_second_wave(ik, shape, add, fewer):
    """Fewer ranks keep clusters from a second wave, except where narrow CTAs have enough to read to hide it."""
    B, C, H, W = shape
    ranks = ik._lib.hy3d_groupnorm_ranks(B, H * W, C, 32, add)
    assert 0 < ranks < 8 if fewer else ranks == 8
    g = torch.Generator(device=DEV).manual_seed(C)
    x = (torch.randn(B, C, H, W, generator=g, device=DEV) * 2 + 0.7).bfloat16().contiguous(memory_format=torch.channels_last)
    gamma, beta = 1 + 0.2 * torch.randn(C, generator=g, device=DEV), 0.2 * torch.randn(C, generator=g, device=DEV)
    term = (torch.randn(B, C, generator=g, device=DEV) * 0.5).bfloat16() if add else None
    xs = x + term[:, :, None, None] if add else x
    ref = torch.nn.functional.group_norm(xs.float(), 32, gamma, beta, 1e-5).bfloat16()
    y = ik.groupnorm_nhwc(x, 32, gamma, beta, 1e-5, silu=True, add=term)
    assert O.rel_l2(y, torch.nn.functional.silu(ref.float()).bfloat16()) < 3e-3


def test_groupnorm_nhwc_argument_checks(ik):
    x = torch.randn(2, 64, 4, 4, device=DEV).bfloat16()
    with pytest.raises(RuntimeError):
        ik.groupnorm_nhwc(x, 32, None, None, 1e-5)                       # NCHW memory
    xl = x.contiguous(memory_format=torch.channels_last)
    y = ik.groupnorm_nhwc(xl, 32, None, None, 1e-5)                      # no affine
    ref = torch.nn.functional.group_norm(xl.float(), 32, None, None, 1e-5)
    assert O.rel_l2(y, ref) < 3e-3
    with pytest.raises(RuntimeError):
        ik.groupnorm_nhwc(torch.randn(1, 60, 4, 4, device=DEV).bfloat16().contiguous(memory_format=torch.channels_last),
                          32, None, None, 1e-5)                          # C % 8, C % groups


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,N,splits,epi", [
    (109, 8064, 752, None, 0),      # the library's own plan
    (257, 6144, 1536, 5, 1),        # GELU, five ranges (48 K blocks: 10 + 10 + 10 + 10 + 8)
    (100, 3152, 272, 3, 0),         # ragged last K block in the last range, ragged columns
    (924, 1024, 320, 4, 0),         # two stages per range
    (130, 4096, 64, 16, 0),         # one narrow tile column, sixteen ranges
    (200, 128, 256, 4, 0),          # one K block cannot be split: the single launch
    (65, 48, 96, 2, 1),
])
def test_dense_splitk_equals_single_launch(tc, dtype, M, K, N, splits, epi):
    """Split-K (int32 partials per K range + reduce/epilogue kernel) gives the bits of the
    single-launch GEMM, whose epilogue it restates, and the int32 sums of the oracle."""
    A, B = _rand_i8((M, K), 31).to(DEV), _rand_i8((N, K), 32).to(DEV)
    g = torch.Generator().manual_seed(33)
    a_s = (torch.rand(M, generator=g) * 0.05 + 1e-3).to(DEV)
    w_s = (torch.rand(N, generator=g) * 1e-3 + 1e-5).to(dtype).to(DEV)
    bias = (torch.randn(N, generator=g) * 0.1).to(dtype).to(DEV)
    if splits is None:
        planned, nbytes = tc.dense_splitk_plan(M, N, K, epi)
        assert planned > 1 and nbytes == planned * ((M + 127) // 128 * 128) * N * 4
    one = tc.int8_gemm_tc(A, B, a_s, w_s, bias, out_dtype=dtype, epilogue=epi, splits=1)
    many = tc.int8_gemm_tc(A, B, a_s, w_s, bias, out_dtype=dtype, epilogue=epi, splits=splits)
    assert torch.equal(one, many)
    ref = O.epilogue(O.int32_matmul(A.cpu(), B.cpu()), a_s.cpu(), w_s.cpu(), bias.cpu(), dtype,
                     "gelu" if epi else "linear")
    assert O.rel_l2(many, ref) < 2e-3
    assert tc.device_status() == 0


@pytest.mark.parametrize("M,K,N,epi,splits", [
    (12288, 1280, 960, 0, 1), (49152, 1280, 320, 0, 1),      # pairs of 224 and 160 columns: seven and five slabs
    (3072, 768, 10240, 2, 1), (3072, 128, 10240, 1, 1),      # with a gate, and with K blocks too few to hide anything
    (27648, 128, 128, 0, 1),                                 # one slab a warp, one K block: wrong in some launches once
    (5000, 2048, 1360, 0, 3),                                # int32 partials: 16-column slabs
])
def test_staging_buffers_over_many_tiles_of_odd_slab_counts(tc, M, K, N, epi, splits):
    """Epilogue warps with an odd number of slabs in a tile and many tiles: the same bits as the direct stores that tile
    widths beside the slab take, over several launches."""
    g = torch.Generator(device=DEV).manual_seed(M + K + N)
    A = torch.randint(-127, 128, (M, K), generator=g, device=DEV, dtype=torch.int8)
    B = torch.randint(-127, 128, (N, K), generator=g, device=DEV, dtype=torch.int8)
    a_s = torch.rand(M, generator=g, device=DEV) * 0.02 + 1e-3
    w_s, b = ((torch.rand(N, generator=g, device=DEV) * 1e-2 + 1e-5).bfloat16() for _ in range(2))
    ref = tc.int8_gemm_tc(A, B, a_s, w_s, b, out_dtype=torch.bfloat16, epilogue=epi, cta_group=1, block_n=96 if epi == 2 else 80)
    for _ in range(40 if K == N else 4):
        assert torch.equal(tc.int8_gemm_tc(A, B, a_s, w_s, b, out_dtype=torch.bfloat16, epilogue=epi, splits=splits), ref)


def test_dense_splitk_plan_leaves_the_unet_shapes_alone(tc):
    for M, K, N in [(49152, 320, 320), (12288, 640, 5120), (3072, 5120, 1280), (924, 1024, 1280)]:
        assert tc.dense_splitk_plan(M, N, K)[0] == 1


@pytest.mark.parametrize("M,K,N,gemm,layer", [
    (257, 6144, 1536, False, False), (358, 5760, 4480, False, False), (123, 3520, 3392, False, False),
    (59, 4096, 64, True, False), (109, 8064, 752, True, True), (298, 7936, 384, True, True),
])
def test_dense_splitk_plans_split_where_it_is_faster(tc, M, K, N, gemm, layer):
    """Shapes of which the split form was measured more than 5 % slower or faster than the single launch, as a GEMM and
    as a layer: us of the GEMM 9.0 and 9.6 split, 11.7 and 15.0, 7.5 and 8.5; 7.7 and 6.6 (layer 10.8 and 10.3),
    12.7 and 7.8, 9.3 and 8.1."""
    for of_layer, want in ((False, gemm), (True, layer)):
        splits, nbytes = tc.dense_splitk_plan(M, N, K, layer=of_layer)
        assert (splits > 1) == want and nbytes == (splits * ((M + 127) // 128 * 128) * N * 4 if want else 0)


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("M,K,N,block_t,ks", [
    (1, 64, 16, 16, 1),            # smallest problem, one ragged K unit
    (16, 128, 128, 16, 1),         # a full 16-token block
    (12, 1280, 640, 16, 5),        # K split over a cluster
    (31, 2688, 1296, 32, 7),       # ragged ranges, ragged weight rows, more units than pipeline stages
    (33, 448, 272, 32, 2),         # second token block of one row
    (100, 1024, 320, 64, 3),       # ranges of unequal length
    (257, 512, 160, 96, 1),
    (300, 192, 96, 160, 1),
    (256, 256, 64, 256, 2),        # widest block
    (5, 2816, 7872, 16, 2)])       # few tokens, more weight tiles than half the SMs
def test_one_launch_layer_equals_two_launches(tc, sp, sparse, M, K, N, block_t, ks):
    """The one-launch layer (codes written straight to the operand tiles, K ranges over a cluster) against
    quantiser + GEMM: same codes, same integer sums, same epilogue, so the same bits."""
    if sparse and ks > 1 and (ks - 1) * -(-(-(-K // 256)) // ks) >= -(-K // 256):
        pytest.skip("a range would be empty")
    g = torch.Generator(device=DEV).manual_seed(M + K)
    wq = torch.randint(-127, 128, (N, K), generator=g, device=DEV, dtype=torch.int8)
    comp, meta = sp.sparse_prune_and_pack(wq) if sparse else (wq, None)
    for dtype in (torch.bfloat16, torch.float16):
        x = torch.randn(M, K, generator=g, device=DEV).to(dtype)
        ws = (torch.rand(N, generator=g, device=DEV) * 1e-3).to(dtype)
        b = torch.randn(N, generator=g, device=DEV).to(dtype)
        code = 1 if dtype == torch.bfloat16 else 0
        q, s = tc._quantize(x)
        for epi in (0, 1, 2):
            if epi == 2 and N % 32:
                continue
            ref = (sp.sparse_int8_gemm(q, s, comp, meta, ws, b, out_dtype=dtype, epilogue=epi) if sparse
                   else tc.int8_gemm_tc(q, wq, s, ws, b, out_dtype=dtype, epilogue=epi))
            out = torch.full_like(ref, float("nan"))
            rc = tc._lib.hy3d_linear_w8a8_cluster(
                x.data_ptr(), code, K, comp.data_ptr(), meta.data_ptr() if sparse else None, meta.shape[1] if sparse else 0,
                ws.data_ptr(), code, b.data_ptr(), code, out.data_ptr(), M, N, K, epi, block_t, ks,
                torch.cuda.current_stream().cuda_stream)
            assert rc == 0 and torch.equal(out, ref)


@pytest.mark.parametrize("M,K,N,one", [
    (7, 3200, 9632, True), (4, 2368, 6160, True), (10, 2048, 9456, True), (2, 7680, 7520, True), (7, 1216, 9760, True),
    (12, 1280, 640, True), (924, 1024, 2560, False), (257, 6144, 1536, False), (53, 4544, 3728, False),
])
def test_dense_layers_take_the_shorter_form(tc, M, K, N, one):
    """One launch or two by what was measured, us: 10.7 and 15.9, 9.0 and 12.5, 8.5 and 11.4, 15.0 and 19.6, 7.1 and 10.6;
    7.1 and 7.6; two where one takes 14.7 against 12.1, or has no plan."""
    assert _runs_as_one_launch(tc, M, N, K) == one


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gelu_epilogue_over_its_whole_range(tc, dtype):
    """Pre-activations from -14 to 14 in steps of 1/512 (accumulator k, scale 1/512): v * Phi(v) in double
    precision, plus the 5e-7 the fp32 form may add, plus the output type's unit roundoff (8 / 11 significant
    bits: 2^-8 / 2^-11 of the value, and half of fp16's spacing of 2^-24 below its normal range)."""
    a = torch.zeros(128, 64, dtype=torch.int8, device=DEV)
    w = torch.zeros(64, 64, dtype=torch.int8, device=DEV)
    v = torch.arange(-7168, 7169, device=DEV)[: 128 * 112].reshape(-1)
    for chunk in v.split(128):
        a.zero_()
        n = chunk.numel()
        a[:n, 0] = torch.div(chunk, 64, rounding_mode="floor").to(torch.int8)     # chunk = 64 * a0 + a1
        a[:n, 1] = (chunk % 64).to(torch.int8)
        w[:, 0], w[:, 1] = 64, 1
        y = tc.int8_gemm_tc(a, w, torch.full((128,), 1.0 / 512, device=DEV), torch.ones(64, device=DEV), None,
                            out_dtype=dtype, epilogue=1)[:n, 0].double()
        x = chunk.double() / 512
        ref = x * torch.special.ndtr(x)
        u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
        tol = ref.abs() * u + 5e-7 + (2.0 ** -25 if dtype == torch.float16 else 0.0)
        assert bool(((y - ref).abs() <= tol).all())


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("M,K,N", [(200, 64, 32), (333, 320, 640), (1000, 1280, 480)])
def test_bf16_gate_rounds_as_the_erf_form(tc, sp, sparse, M, K, N):
    """The GEGLU epilogue computes most gates by another formula than 0.5 * g * (1 + erf(g / sqrt 2)) but
    must round every bf16 output as that one does: torch's fp32 ops on the raw accumulators, bit for bit
    (gates between about -10 and 10; without a bias the rescaled accumulator is one rounded product)."""
    g = torch.Generator(device=DEV).manual_seed(K + N)
    q = torch.randint(-127, 128, (M, K), generator=g, device=DEV, dtype=torch.int8)
    w = torch.randint(-127, 128, (N, K), generator=g, device=DEV, dtype=torch.int8)
    comp, meta = sp.sparse_prune_and_pack(w) if sparse else (w, None)
    s = torch.rand(M, generator=g, device=DEV) * 2 + 0.5
    ws = (torch.rand(N, generator=g, device=DEV) + 0.5) * 3.0 / (73.0 * 73.0 * K ** 0.5 * 1.25)
    if sparse:
        acc = sp.sparse_int8_gemm(q, None, comp, meta, None, None, out_dtype=torch.int32)
        y = sp.sparse_int8_gemm(q, s, comp, meta, ws, None, out_dtype=torch.bfloat16, epilogue=2)
    else:
        acc = tc.int8_gemm_tc(q, w, None, None, None, out_dtype=torch.int32)
        y = tc.int8_gemm_tc(q, w, s, ws, None, out_dtype=torch.bfloat16, epilogue=2)
    v = (acc.double() * (s[:, None] * ws[None, :]).double()).float().view(M, N // 32, 2, 16)
    value, gate = v[:, :, 0].reshape(M, -1), v[:, :, 1].reshape(M, -1)
    ref = (value * (0.5 * gate * (1.0 + torch.erf(gate * 0.70710678118654752440)))).bfloat16()
    assert torch.equal(y, ref)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [(1, 8, 1, 1), (2, 24, 5, 7), (3, 320, 9, 16), (1, 2560, 4, 3), (2, 1032, 33, 17)])
def test_nhwc_steps_equal_the_separate_torch_ops(qu, dtype, shape):
    """Bias / residual sums, concatenation, upsampling and the normalisation's pre-added terms against torch's
    separate ops, bit for bit (values over many binades, so that small addends round away and ties occur)."""
    nat = qu._load_native()
    B, C, H, W = shape
    g = torch.Generator(device=DEV).manual_seed(C + H)

    def rand(*s):
        return (torch.randn(*s, generator=g, device=DEV) * torch.exp2(torch.randint(-12, 6, s, generator=g, device=DEV).float())).to(dtype)
    cl = torch.channels_last
    x, h = rand(*shape).contiguous(memory_format=cl), rand(*shape).contiguous(memory_format=cl)
    bx, bh = rand(C), rand(C)
    col = lambda b: b[:, None, None]   # noqa: E731
    assert torch.equal(nat.add_bias(x, bx, None, None), x + col(bx))
    assert torch.equal(nat.add_bias(x, None, h, bh), x + (h + col(bh)))
    assert torch.equal(nat.add_bias(x, bx, h, bh), (x + col(bx)) + (h + col(bh)))
    other = rand(B, 16, H, W).contiguous(memory_format=cl)
    y = nat.concat_nhwc(x, other)
    assert torch.equal(y, torch.cat([x, other], 1)) and y.is_contiguous(memory_format=cl)
    y = nat.upsample2x_nhwc(x)
    assert torch.equal(y, torch.nn.functional.interpolate(x, scale_factor=2.0, mode="nearest")) and y.is_contiguous(memory_format=cl)
    assert nat.add_bias(x.contiguous(memory_format=cl).float(), bx, None, None) is None
    # the normalisation with a bias and a strided (B, C) term equals normalising the sum made beforehand
    groups = 8 if C % 64 == 0 else 1
    terms = rand(B, C + 24)[:, 8:8 + C]
    norm = __import__("importlib").import_module("hunyuan3d-tools_b200.unet").GroupNormNHWC(groups, C).to(DEV).to(dtype)
    norm.requires_grad_(False).fused = True
    x1 = ((x + col(bx)) + terms[:, :, None, None]).contiguous(memory_format=cl)
    assert torch.equal(nat.groupnorm_call(norm, x, terms, bx), norm(x1))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K", [(1, 64), (33, 320), (257, 640), (1000, 1088), (5, 1280), (300, 2048), (70, 5120)])
def test_residual_quantisers_equal_adding_first(qu, ik, dtype, M, K):
    nat = qu._load_native()
    g = torch.Generator(device=DEV).manual_seed(M + K)
    x, h = (torch.randn(M, K, generator=g, device=DEV).to(dtype) for _ in range(2))
    q, s = ik.fused_quantize_activation(x + h)
    got = nat.add_quantize(x, h)
    assert torch.equal(got.q, q) and torch.equal(got.scale, s) and got.shape == x.shape and got.dtype == dtype
    if K <= 2048:
        ln = torch.nn.LayerNorm(K, device=DEV, dtype=dtype)
        ln.weight.data.copy_(1 + 0.2 * torch.randn(K, generator=g, device=DEV))
        norm = qu.Int8LayerNorm(ln)
        total, z = nat.norm_call(norm, x, h)
        ref = norm(x + h)
        assert torch.equal(total, x + h) and torch.equal(z.q, ref.q) and torch.equal(z.scale, ref.scale)


@pytest.mark.parametrize("M,K,N", [(298, 7936, 384), (173, 8448, 640)])
def test_planned_split_takes_parameters_at_any_address(qu, tc, M, K, N):
    """Scales and bias that do not start on 16 bytes: the reduction behind a split K refuses them, so a shape the
    plan would split runs as one launch, with the same bits.  With parameters that do it runs split, here and in the
    native path."""
    assert tc.dense_splitk_plan(M, N, K)[0] > 1 and tc.dense_splitk_plan(M, N, K, layer=True)[0] > 1
    assert not _runs_as_one_launch(tc, M, N, K)
    g = torch.Generator(device=DEV).manual_seed(K)
    x = torch.randn(M, K, generator=g, device=DEV).bfloat16()
    w = torch.randint(-127, 128, (N, K), generator=g, device=DEV, dtype=torch.int8)
    ws, b = (torch.rand(N + 1, generator=g, device=DEV).bfloat16() for _ in range(2))
    q, s = tc._quantize(x)
    ref = tc.int8_gemm_tc(q, w, s, ws[1:].clone(), b[1:].clone(), out_dtype=torch.bfloat16, splits=1)
    native = qu._load_native()
    for scale, bias in ((ws[1:].clone(), b[1:].clone()), (ws[1:], b[1:]), (ws[1:].clone(), b[1:]), (ws[1:], b[1:].clone())):
        assert torch.equal(tc.int8_linear_tc(x, w, scale, bias), ref)
        assert torch.equal(tc.int8_gemm_tc(q, w, s, scale, bias, out_dtype=torch.bfloat16), ref)
        assert torch.equal(native.gemm_dense(q, s, w, scale, bias, 1, 0, (M, K)), ref)


@pytest.mark.parametrize("sparse", [False, True])
@pytest.mark.parametrize("M,K,N,block", [(3000, 64, 640, 97), (2500, 320, 2560, 400), (700, 1280, 96, 33)])
def test_bf16_gate_keeps_its_bits_when_the_gates_width_changes(tc, sp, sparse, M, K, N, block):
    """Warps that meet many strongly negative gates go over to the erf form and come back where the gates are narrow:
    blocks of rows with gates of a standard deviation of 0.2, 2 and 12 in turn, the same bits throughout."""
    g = torch.Generator(device=DEV).manual_seed(K + N)
    q = torch.randint(-127, 128, (M, K), generator=g, device=DEV, dtype=torch.int8)
    w = torch.randint(-127, 128, (N, K), generator=g, device=DEV, dtype=torch.int8)
    comp, meta = sp.sparse_prune_and_pack(w) if sparse else (w, None)
    s = torch.tensor([0.2, 2.0, 0.2, 12.0], device=DEV)[torch.arange(M, device=DEV) // block % 4]
    ws = (torch.rand(N, generator=g, device=DEV) + 0.5) / (73.0 * 73.0 * K ** 0.5)
    if sparse:
        acc = sp.sparse_int8_gemm(q, None, comp, meta, None, None, out_dtype=torch.int32)
        y = sp.sparse_int8_gemm(q, s, comp, meta, ws, None, out_dtype=torch.bfloat16, epilogue=2)
    else:
        acc = tc.int8_gemm_tc(q, w, None, None, None, out_dtype=torch.int32)
        y = tc.int8_gemm_tc(q, w, s, ws, None, out_dtype=torch.bfloat16, epilogue=2)
    v = (acc.double() * (s[:, None] * ws[None, :]).double()).float().view(M, N // 32, 2, 16)
    value, gate = v[:, :, 0].reshape(M, -1), v[:, :, 1].reshape(M, -1)
    ref = (value * (0.5 * gate * (1.0 + torch.erf(gate * 0.70710678118654752440)))).bfloat16()
    assert torch.equal(y, ref)


def test_gelu_and_erf_form_stay_within_the_gates_bound(ik):
    """What the settled bf16 gate rests on, for every fp32 gate: 253 binades of two signs, none further from the erf
    form than 2.1e-7 |g| -- and the count does notice a bound that does not hold."""
    compared, outside = ik.gelu_enum_check(2.1e-7)
    assert compared == 2 * 253 * 2 ** 23 and outside == 0
    assert ik.gelu_enum_check(2.0e-7)[1] > 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,K,N", [(5, 128, 144), (300, 128, 144), (1500, 64, 256), (298, 7936, 384)])
def test_gelu_of_infinite_pre_activations(qu, tc, dtype, M, K, N):
    """+infinity stays, -infinity and NaN give NaN, as in torch, and the columns beside them keep their bits: one launch,
    two and three (split K), direct and bulk stores, dense and 2:4 sparse."""
    if K == 7936:
        assert tc.dense_splitk_plan(M, N, K, 1, layer=True)[0] > 1 and not _runs_as_one_launch(tc, M, N, K)
    torch.manual_seed(K)
    lin = torch.nn.Linear(K, N).to(DEV).to(dtype)
    x = torch.randn(M, K, device=DEV).to(dtype)
    special = [float("inf"), float("-inf"), float("nan"), 3e4, -3e4]
    for make in (qu.Int8Linear.from_linear, qu.Int8Linear.from_linear_sparse):
        layer = make(lin)
        layer.epilogue = "gelu"
        ref = layer(x)
        layer.bias = layer.bias.clone()
        layer.bias[:5] = torch.tensor(special, device=DEV).to(dtype)
        y = layer(x)
        assert torch.equal(y[:, 5:], ref[:, 5:])
        assert bool((y[:, 0] == float("inf")).all()) and bool(y[:, 1:3].isnan().all())
        assert bool((y[:, 3] > 2.9e4).all()) and bool((y[:, 4] == 0).all())


@pytest.mark.parametrize("alias", ["x", "h"])
def test_bias_pass_may_write_over_its_input(tc, alias):
    torch.manual_seed(3)
    x, h = (torch.randn(2, 40, 33, 17, device=DEV).bfloat16().contiguous(memory_format=torch.channels_last) for _ in range(2))
    b = torch.randn(40, device=DEV).bfloat16()
    ref = (x + b[:, None, None]) + (h + b[:, None, None])
    y = x if alias == "x" else h
    assert tc._lib.hy3d_add_bias_nhwc(x.data_ptr(), b.data_ptr(), h.data_ptr(), b.data_ptr(), 1, y.data_ptr(), 2 * 33 * 17, 40,
                                      torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(y, ref)
