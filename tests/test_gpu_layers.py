"""GPU tests of the host-side module (Int8Linear, model surgery), following the reference's
own integration checks (tools/test_sparse_tc.py:613-693, tools/test_sparse_numerics.py,
tools/test_int8_memory.py) plus parity with vectors from the reference's CPU code."""
import pytest
import torch
import torch.nn as nn

from oracle import oracle as O
from conftest import as_half

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _pruned_dense_weight(layer, sp, w_int8):
    """As tools/test_sparse_numerics.py:39-50: expand the kernel's compressed weight."""
    comp, meta_raw = sp.sparse_prune_compress(w_int8)
    N, K = w_int8.shape
    G = K // 4
    vals = comp.view(N, G, 2).float()
    nib = meta_raw.view(N, G).to(torch.int64)
    idx = torch.stack([nib & 3, (nib >> 2) & 3], dim=-1)
    dense = torch.zeros(N, G, 4, device=w_int8.device)
    dense.scatter_(2, idx, vals)
    assert torch.equal(comp, layer.weight_sparse_comp), "compressed weight mismatch"
    return dense.view(N, K) * layer.weight_scale.float()[:, None]


def test_dense_layer_matches_reference_golden(qu, golden):
    """Same fp16 Linear and inputs the reference's CPU path was run on."""
    for tag, (K, N) in {"a": (320, 128), "b": (128, 256), "c": (1024, 64)}.items():
        lin = nn.Linear(K, N).half()
        lin.weight.data = as_half(golden[f"{tag}_weight"])
        lin.bias.data = as_half(golden[f"{tag}_bias"])
        layer = qu.Int8Linear.from_linear(lin).to(DEV)      # quantised where the reference was: on the CPU
        assert torch.equal(layer.weight_int8_nk.cpu(), torch.from_numpy(golden[f"{tag}_weight_int8_nk"]))
        assert torch.equal(layer.weight_scale.cpu(), as_half(golden[f"{tag}_weight_scale"]))
        y = layer(as_half(golden[f"{tag}_x"]).to(DEV))
        y_ref = as_half(golden[f"{tag}_y_int_mm"])
        assert y.dtype == torch.float16 and y.shape == y_ref.shape
        assert O.rel_l2(y, y_ref) < 1e-2           # output gate against the reference's W8A8 path
        assert O.rel_l2(y, y_ref) < 1e-3           # observed: one fp16 rounding apart
        assert O.rel_l2(y, as_half(golden[f"{tag}_y_dequant"])) < 2e-2


@pytest.mark.parametrize("K,N,M", [(1280, 1280, 64), (1280, 1280, 4096), (320, 1280, 4096),
                                   (1280, 320, 64), (640, 5120, 777)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_dense_layer_close_to_fp_linear(qu, K, N, M, dtype):
    """tools/test_int8_memory.py:17-31: rel-L2 < 2 % against the unquantised layer."""
    torch.manual_seed(0)
    lin = nn.Linear(K, N).to(DEV).to(dtype)
    layer = qu.Int8Linear.from_linear(lin)
    x = torch.randn(M, K, device=DEV, dtype=dtype)
    y, ref = layer(x), lin(x)
    assert O.rel_l2(y, ref) < 0.02
    assert O.rel_l2(y, O.linear_w8a8(x.cpu(), layer.weight_int8_nk.cpu(), layer.weight_scale.cpu(),
                                     lin.bias.data.cpu())) < 1e-3


def test_layer_handles_3d_input_and_no_bias(qu):
    """tools/test_sparse_tc.py:646-672."""
    torch.manual_seed(1)
    lin = nn.Linear(640, 1280, bias=False).to(DEV).half()
    for make in (qu.Int8Linear.from_linear, qu.Int8Linear.from_linear_sparse):
        layer = make(lin)
        x = torch.randn(2, 77, 640, device=DEV, dtype=torch.float16)
        y = layer(x)
        assert y.shape == (2, 77, 1280) and not torch.isnan(y).any()
        assert torch.equal(y.view(-1, 1280), layer(x.view(-1, 640)))


def test_sparse_layer_buffers_and_stats(qu, sp):
    """tools/test_sparse_tc.py:628-679: buffer shapes of a 640->1280 layer and the stats of
    quantize_model_sparse on a two-layer MLP."""
    torch.manual_seed(2)
    lin = nn.Linear(640, 1280).to(DEV).half()
    layer = qu.Int8Linear.from_linear_sparse(lin)
    assert layer.mode == "sparse"
    assert tuple(layer.weight_sparse_comp.shape) == (1280, 320)
    assert tuple(layer.weight_sparse_meta.shape) == (1280, 20)      # K/32 words per row
    assert layer.weight_sparse_meta.dtype == torch.int32
    assert layer.weight_int8_nk.numel() == 0
    mlp = nn.Sequential(nn.Linear(640, 1280), nn.GELU(), nn.Linear(1280, 640)).to(DEV).half()
    stats = qu.quantize_model_sparse(mlp, verbose=False)
    assert stats["num_replaced"] == 2 and stats["sparse_eligible"] == 2 and stats["kept_fp16"] == 0
    out = mlp(torch.randn(300, 640, device=DEV, dtype=torch.float16))
    assert out.shape == (300, 640) and not torch.isnan(out).any()
    small = nn.Sequential(nn.Linear(320, 640)).to(DEV).half()
    s2 = qu.quantize_model_sparse(small, verbose=False)
    assert s2["kept_fp16"] == 1 and isinstance(small[0], nn.Linear)


@pytest.mark.parametrize("K,N,M", [(640, 640, 4096), (1280, 1280, 9216), (640, 5120, 2048),
                                   (2560, 640, 4096), (5120, 1280, 1024), (1024, 320, 2772),
                                   (1280, 1280, 3), (1536, 1536, 257), (4096, 1536, 257)])
def test_sparse_layer_numerics(qu, sp, K, N, M):
    """tools/test_sparse_numerics.py:53-76: rel-L2 < 2 % against fp32 math on the pruned
    weights (reduced M for the largest shapes), at M and at 64 rows."""
    torch.manual_seed(0)
    lin = nn.Linear(K, N).to(DEV).half()
    layer = qu.Int8Linear.from_linear_sparse(lin)
    w32 = lin.weight.float()
    scale = w32.abs().amax(dim=1).clamp(min=1e-8) / 127.0
    w_int8 = (w32 / scale[:, None]).round().clamp(-128, 127).to(torch.int8).contiguous()
    w_pruned = _pruned_dense_weight(layer, sp, w_int8)
    for m in sorted({M, 64}):
        x = torch.randn(m, K, device=DEV, dtype=torch.half)
        y = layer(x).float()
        ref = x.float() @ w_pruned.t() + lin.bias.float()
        assert float((y - ref).norm() / ref.norm()) < 0.02
    # and bit-level agreement of the packed buffers with the oracle
    co, no = O.prune_compress(w_int8.cpu())
    assert torch.equal(layer.weight_sparse_comp.cpu(), co)
    assert torch.equal(layer.weight_sparse_meta.cpu(), O.pack_metadata(no, layer.weight_sparse_meta.shape[1]))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("N,K", [(16, 64), (19, 96), (640, 320), (77, 2048), (33, 2080), (48, 6144), (1, 16384)])
def test_weight_conversion_equals_the_torch_expressions(qu, sp, dtype, N, K):
    """One kernel against the operation-by-operation torch form on the same device: codes, scales,
    survivors and metadata bit for bit (rows at both sides of every thread-group size, ragged metadata
    padding, an all-zero row, tiny and huge rows)."""
    torch.manual_seed(N + K)
    lin = nn.Linear(K, N, device=DEV, dtype=dtype)
    lin.weight.data.copy_(torch.randn(N, K, device=DEV) * 0.02)
    lin.weight.data[0] = 0
    lin.weight.data[-1] *= 1e4
    lin.weight.data[N // 2] *= 1e-5
    w = lin.weight.data.float()
    amax = w.abs().amax(dim=1)
    dt = dtype if dtype != torch.float32 else torch.float16
    for make, scale in ((qu.Int8Linear.from_linear, (amax / 127.0).clamp(min=1e-8)),
                        (qu.Int8Linear.from_linear_sparse, amax.clamp(min=1e-8) / 127.0)):
        layer = make(lin)
        codes = (w / scale[:, None]).round().clamp(-128, 127).to(torch.int8)
        assert torch.equal(layer.weight_scale, scale.to(dt))
        if layer.mode == "sparse":
            comp, meta = sp.sparse_prune_and_pack(codes)
            assert torch.equal(layer.weight_sparse_comp, comp) and torch.equal(layer.weight_sparse_meta, meta)
            assert layer.weight_int8_nk.numel() == 0
        else:
            assert torch.equal(layer.weight_int8_nk, codes)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("K", [768, 16384 + 512])      # kept in registers, read again
def test_weight_conversion_at_the_ties(qu, dtype, K):
    """Codes of weights around every half-integer multiple of the scale: rows of every significand of the largest weight (127
    divides some), of a scale at its floor in either form and below the type's normal range; the neighbours on both sides of
    each tie."""
    bits = 7 if dtype == torch.bfloat16 else 10
    plain = torch.cat([1 + torch.arange(2 ** bits) / 2 ** bits, torch.tensor([1.27e-6, 1.2e-6, 3e-7, 6e-8, 1e-3, 254 / 4096])]).to(dtype)
    dense_floor, sparse_floor = torch.tensor([1.2e-6, 3e-7, 6e-8, 1e-8]).to(dtype), torch.tensor([9.9e-9, 9e-9, 1e-9, 5e-11]).to(dtype)
    amax = torch.cat([plain, dense_floor, sparse_floor])      # the last four are zero in fp16
    unit = torch.cat([plain.double() / 127, torch.full((4,), 1e-8, dtype=torch.double), torch.full((4,), 1e-8 / 127, dtype=torch.double)])
    k = torch.arange(127)
    tie = (unit[:, None] * (2 * k + 1) / 2).to(dtype)
    near = torch.cat([tie, torch.nextafter(tie, torch.zeros_like(tie)), torch.nextafter(tie, amax[:, None].expand_as(tie))], 1)
    near = torch.cat([near, -near, amax[:, None], -amax[:, None]], 1)
    w = torch.zeros(amax.numel(), K, dtype=dtype)
    w[:, :near.shape[1]] = torch.minimum(near.abs(), amax[:, None]).copysign(near)
    lin = torch.nn.Linear(K, w.shape[0], bias=False, dtype=dtype, device=DEV)
    lin.weight.data.copy_(w)
    wf, am = w.to(DEV).float(), w.to(DEV).float().abs().amax(1, keepdim=True)
    dense = qu.Int8Linear.from_linear(lin)
    assert torch.equal(dense.weight_int8_nk, torch.round(wf / (am / 127.0).clamp(min=1e-8)).clamp(-128, 127).to(torch.int8))
    codes = torch.round(wf / (am.clamp(min=1e-8) / 127.0)).clamp(-128, 127).to(torch.int8)
    comp, _ = O.prune_compress(codes.cpu())
    assert torch.equal(qu.Int8Linear.from_linear_sparse(lin).weight_sparse_comp.cpu(), comp)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("N,K", [(9, 32), (40, 544), (24, 1312), (17, 2560), (3, 16416)])
def test_weight_conversion_in_registers_and_with_values_that_are_not_finite(qu, sp, dtype, N, K):
    """Rows of one round, of three and six of the five and eight that a thread keeps, of more threads than a warp, and
    rows too long to keep; a row with a NaN, one with an infinity, one whose only value is the last."""
    g = torch.Generator(device=DEV).manual_seed(N + K)
    w = (torch.randn(N, K, device=DEV, generator=g) * 0.02).to(dtype)
    w[0, K // 3], w[1, K - 1] = float("nan"), float("inf")
    w[2] = 0
    w[2, K - 1] = -0.5
    f = w.float()
    amax = f.abs().amax(dim=1)
    native = qu._load_native()
    for sparse, scale in ((False, (amax / 127.0).clamp(min=1e-8)), (True, amax.clamp(min=1e-8) / 127.0)):
        got = native.quantize_weight(w, sparse)
        codes = torch.nan_to_num((f / scale[:, None]).round()).clamp(-128, 127).to(torch.int8)
        assert torch.equal(torch.nan_to_num(got[-1]), torch.nan_to_num(scale.to(torch.float16 if dtype == torch.float32 else dtype)))
        assert torch.equal(torch.isnan(got[-1]), torch.isnan(scale))
        if sparse:
            comp, meta = sp.sparse_prune_and_pack(codes)
            assert torch.equal(got[0], comp) and torch.equal(got[1], meta)
        else:
            assert torch.equal(got[0], codes)


def test_geglu_fused_layer(qu):
    torch.manual_seed(3)
    lin = nn.Linear(320, 2560).to(DEV).bfloat16()
    x = torch.randn(1000, 320, device=DEV, dtype=torch.bfloat16)
    plain = qu.Int8Linear.from_linear(lin)
    fused = qu.Int8Linear.from_linear(lin).interleave_geglu_rows()
    v, g = plain(x).float().chunk(2, dim=-1)
    y = fused(x)
    assert y.shape == (1000, 1280)
    # the unfused path rounds value and gate to bf16 first
    assert O.rel_l2(y, v * torch.nn.functional.gelu(g)) < 1e-2


@pytest.mark.parametrize("M", [1000, 3072])
def test_geglu_fused_sparse_layer(qu, M):
    """Row interleaving commutes with 2:4 pruning (which acts along K inside a row), so a
    sparse up-projection can be switched to the fused GEGLU epilogue after conversion; M = 3072
    takes the CTA-pair variant of the sparse kernel."""
    torch.manual_seed(5)
    lin = nn.Linear(1280, 2560).to(DEV).bfloat16()
    x = torch.randn(M, 1280, device=DEV, dtype=torch.bfloat16)
    plain = qu.Int8Linear.from_linear_sparse(lin)
    fused = qu.Int8Linear.from_linear_sparse(lin).interleave_geglu_rows()
    assert fused.mode == "sparse" and fused.epilogue == "geglu"
    v, g = plain(x).float().chunk(2, dim=-1)
    y = fused(x)
    assert y.shape == (M, 1280)
    assert O.rel_l2(y, v * torch.nn.functional.gelu(g)) < 1e-2


def test_mixed_model_surgery(qu):
    torch.manual_seed(4)
    model = nn.Sequential(nn.Linear(320, 1280), nn.Linear(1280, 320), nn.Linear(320, 64)).to(DEV).half()
    stats = qu.quantize_model_mixed(model, sparse_min_k=640, verbose=False)
    assert stats["sparse_layers"] == 1 and stats["dense_layers"] == 1
    assert model[0].mode == "tc" and model[1].mode == "sparse" and isinstance(model[2], nn.Linear)
    y = model(torch.randn(500, 320, device=DEV, dtype=torch.float16))
    assert y.shape == (500, 64) and not torch.isnan(y).any()


def test_kernels_run_on_the_current_stream_and_capture(qu):
    """A layer call is capturable in a CUDA graph (everything is launched on the current
    stream and nothing synchronises)."""
    torch.manual_seed(5)
    layer = qu.Int8Linear.from_linear(nn.Linear(640, 640).to(DEV).half())
    x = torch.randn(512, 640, device=DEV, dtype=torch.float16)
    eager = layer(x)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        layer(x)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            y = layer(x)
    torch.cuda.current_stream().wait_stream(s)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, eager)


def test_sparse_state_dict_roundtrip(qu):
    """A pruned + packed layer reloads into a fresh module without re-pruning (the reference
    cannot: its sparse buffers are registered as None)."""
    torch.manual_seed(7)
    lin = nn.Linear(1280, 640).to(DEV).bfloat16()
    a = qu.Int8Linear.from_linear_sparse(lin)
    sd = {k: v.cpu() if torch.is_tensor(v) else v for k, v in a.state_dict().items()}
    b = qu.Int8Linear(1280, 640, bias=True)
    b.load_state_dict(sd)
    b = b.to(DEV)
    assert b.mode == "sparse" and b.weight_int8_nk.numel() == 0
    assert torch.equal(a.weight_sparse_comp, b.weight_sparse_comp)
    assert torch.equal(a.weight_sparse_meta, b.weight_sparse_meta)
    x = torch.randn(300, 1280, device=DEV, dtype=torch.bfloat16)
    assert torch.equal(a(x), b(x))


def test_host_pipeline_matches_direct_calls(qu, pkg):
    """Layers fed from pinned host memory through the three-stream pipeline return the same
    bits as direct calls on device tensors."""
    import importlib
    host_io = importlib.import_module(pkg.__name__ + ".host_io")
    torch.manual_seed(4)
    shapes = [(1000, 320, 640), (513, 640, 320), (2048, 1280, 1280)]
    layers, hx, hy, ref = [], [], [], []
    for M, K, N in shapes:
        lin = torch.nn.Linear(K, N, device=DEV, dtype=torch.bfloat16)
        L = qu.Int8Linear.from_linear(lin)
        x = torch.randn(M, K).bfloat16()
        layers.append(L)
        hx.append(x.pin_memory())
        hy.append(torch.empty(M, N, dtype=torch.bfloat16).pin_memory())
        ref.append(L(x.to(DEV)).cpu())
    pipe = host_io.HostPipeline(DEV)
    for _ in range(2):
        pipe.run(layers, hx, hy)
    pipe.synchronize()
    for a, b in zip(hy, ref):
        assert torch.equal(a, b)


def test_direct_calls_leave_hooks_and_overrides_alone(qu):
    """Calling a layer takes a direct way to the kernels; a hook, a replaced or overridden `forward` and a
    keyword argument must still go through nn.Module."""
    torch.manual_seed(5)
    lin = nn.Linear(128, 64).to(DEV).bfloat16()
    x = torch.randn(9, 128, device=DEV).bfloat16()
    for make in (qu.Int8Linear.from_linear, qu.Int8Linear.from_linear_sparse):
        layer = make(lin)
        y = layer(x)
        assert torch.equal(y, layer(x=x)) and torch.equal(y, layer.forward(x))
        h = layer.register_forward_hook(lambda m, a, out: out + 1)
        assert torch.equal(layer(x), y + 1)
        h.remove()
        h = layer.register_forward_pre_hook(lambda m, a: (a[0] * 0,))
        assert torch.equal(layer(x), layer.forward(x * 0))
        h.remove()
        h = nn.modules.module.register_module_forward_hook(lambda m, a, out: out * 2)
        assert torch.equal(layer(x), y * 2)
        h.remove()
        layer.forward = lambda t: t
        assert layer(x) is x
        del layer.forward
        assert torch.equal(layer(x), y)

    class Doubled(qu.Int8Linear):
        def forward(self, t):
            return super().forward(t) * 2
    d = Doubled(128, 64, dtype=torch.bfloat16)
    d.load_state_dict(qu.Int8Linear.from_linear(lin).state_dict())
    assert torch.equal(d.to(DEV)(x), qu.Int8Linear.from_linear(lin)(x) * 2)
    ln = qu.Int8LayerNorm(nn.LayerNorm(128).to(DEV).bfloat16())
    seen = []
    h = ln.register_forward_hook(lambda m, a, out: seen.append(out))
    a = ln(x)
    h.remove()
    b = ln(x)
    assert seen == [a] and torch.equal(a.q, b.q) and torch.equal(a.scale, b.scale)
    assert b.shape == x.shape and b.dtype == x.dtype and torch.equal(layer(a), layer(b))


@pytest.mark.parametrize("sparse", [False, True])
def test_quantised_activation_of_another_shape_is_refused(qu, sparse):
    """The output is allocated from the activation's shape while the kernel writes one row per code row, so a
    shape that does not describe the codes has to raise instead of reaching the kernel."""
    torch.manual_seed(8)
    layer = (qu.Int8Linear.from_linear_sparse if sparse else qu.Int8Linear.from_linear)(nn.Linear(128, 64).to(DEV).bfloat16())
    act = qu.Int8LayerNorm(nn.LayerNorm(128).to(DEV).bfloat16())(torch.randn(24, 128, device=DEV).bfloat16())
    y = layer(act)
    for shape in ((4, 6, 128), (24, 1, 128), (2, 3, 4, 128)):
        assert torch.equal(layer(act.view(*shape)), y.view(*shape[:-1], 64))
    for shape in ((1, 128), (23, 128), (4, 5, 128), (25, 128), (48, 128), (0, 128), (128,), (24, 2, 128)):
        with pytest.raises(RuntimeError):
            layer(qu.QuantizedActivation(act.q, act.scale, shape, act.dtype))
    native = qu._load_native()
    w, meta = (layer.weight_sparse_comp, (layer.weight_sparse_meta,)) if sparse else (layer.weight_int8_nk, ())
    gemm = native.gemm_sparse if sparse else native.gemm_dense
    for shape in ((24, 64), (-24, 128), (1 << 70, 128), (24, 1 << 70), (1 << 62, 1 << 62, 24, 128), (), ("24", 128)):
        assert gemm(act.q, act.scale, w, *meta, layer.weight_scale, layer.bias, 1, 0, shape) is None
    assert torch.equal(layer(act), y)
