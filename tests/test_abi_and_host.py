"""CPU-side checks: the C-ABI library loads and exports every symbol the header declares,
argument validation answers without a GPU, and the host-side module logic (lambda warm-up,
the straight-through training formula, state_dict compatibility) behaves as the reference's."""
import ctypes
import os
import re

import numpy as np
import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def header_symbols():
    text = open(os.path.join(ROOT, "include", "wf_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(wf_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol(wf):
    lib = ctypes.CDLL(wf._lib.LIB_PATH)
    names = header_symbols()
    assert len(names) >= 12
    for n in names:
        assert hasattr(lib, n), f"{n} declared in include/wf_b200.h but not exported"
    assert sorted(wf._lib.exported_symbols()) == names  # the Python binding covers the whole header


def test_argument_errors_need_no_gpu(wf):
    lib = wf._lib.lib()
    assert lib.wf_version() >= 100
    rc = lib.wf_pack_ternary(None, 0, 4, 64, 64, 0, 1e-5, None, None, None, 0, None)
    assert rc == 1 and b"null pointer" in lib.wf_last_error()
    assert lib.wf_pack_scratch_bytes(1536, 576) >= 8
    assert lib.wf_prefill_workspace_bytes(512, 2560) >= 512 * 2560 + 512 * 4
    buf = (ctypes.c_char * 4096)()
    p = ctypes.addressof(buf)
    p = (p + 255) // 256 * 256
    # K not a multiple of 64 is rejected before anything is launched
    rc = lib.wf_bitlinear_decode(p, 2, 48, None, p, 0, None, 1.0, None, 0, p, 0, 16, None, 1, 16, 48, 1e-5, 0, None)
    assert rc == 1 and b"multiple of 64" in lib.wf_last_error()
    rc = lib.wf_bitlinear_decode(p, 2, 64, None, p, 1, None, 1.0, None, 0, p, 0, 16, None, 1, 16, 64, 1e-5, 0, None)
    assert rc == 1 and b"128" in lib.wf_last_error()


def test_no_cpu_fallback(wf):
    if torch.cuda.is_available():
        pytest.skip("checks the behaviour of a machine without a GPU")
    assert not wf.check_kernel_available()
    with pytest.raises(RuntimeError):
        wf.pack_ternary(torch.zeros(4, 64))
    layer = wf.BitLinear(64, 8)
    with pytest.raises(RuntimeError), torch.no_grad():
        layer(torch.zeros(1, 64))


def test_training_formula_and_lambda(wf):
    torch.manual_seed(0)
    layer = wf.BitLinear(64, 16, bias=True)
    x = torch.randn(3, 64, requires_grad=True)
    # lambda = 1: forward == F.linear(aq(x), wq(W)) (test_paper_verification.py:365-377)
    y = layer(x)
    want = torch.nn.functional.linear(layer.activation_quant(x), layer.weight_quant(layer.weight), layer.bias)
    assert torch.allclose(y, want, atol=1e-5)
    y.sum().backward()
    assert x.grad is not None and layer.weight.grad is not None  # straight-through gradients
    # lambda = 0: plain linear (test_paper_verification.py:353-363)
    warm = wf.LambdaWarmup(warmup_steps=10)
    wf.set_global_lambda_warmup(warm)
    try:
        assert wf.get_current_lambda() == 0.0
        assert torch.allclose(layer(x), torch.nn.functional.linear(x, layer.weight, layer.bias), atol=1e-6)
        for _ in range(5):
            warm.step()
        assert wf.get_current_lambda() == pytest.approx(0.5)
        for _ in range(5):
            warm.step()
        assert warm.is_warmup_complete() and wf.get_current_lambda() == 1.0
        st = warm.state_dict()
        w2 = wf.LambdaWarmup(warmup_steps=3)
        w2.load_state_dict(st)
        assert w2.lambda_val == 1.0 and w2.warmup_steps == 10
    finally:
        wf.set_global_lambda_warmup(None)
    # quantizer formulas (test_paper_verification.py:24-48, 87-110)
    w = torch.randn(16, 64)
    s = w.abs().mean()
    assert torch.allclose(layer.weight_quant(w), (w / s).round().clamp(-1, 1) * s, atol=1e-6)
    aq = layer.activation_quant(x.detach())
    ints = aq * (127.0 / x.detach().abs().max(dim=-1, keepdim=True).values)
    assert torch.allclose(ints, ints.round(), atol=1e-3) and ints.abs().max() <= 128


def test_state_dict_and_conversion(wf):
    lin = torch.nn.Sequential(torch.nn.Linear(64, 32, bias=True), torch.nn.ReLU(), torch.nn.Linear(32, 8, bias=False))
    ref_sd = {k: v.clone() for k, v in lin.state_dict().items()}
    wf.convert_linear_to_bitlinear(lin)
    assert isinstance(lin[0], wf.BitLinear) and isinstance(lin[2], wf.BitLinear)
    assert set(lin.state_dict()) == set(ref_sd)  # weight / bias only: nn.Linear checkpoints load unchanged
    for k, v in ref_sd.items():
        assert torch.equal(lin.state_dict()[k], v)
    other = wf.BitLinear(64, 32, bias=True)
    other.load_state_dict({"weight": ref_sd["0.weight"], "bias": ref_sd["0.bias"]})
    x = torch.randn(2, 64)
    na = wf.BitLinearNoActivationQuant(64, 32)
    na.weight.data.copy_(ref_sd["0.weight"])
    assert torch.allclose(na(x), torch.nn.functional.linear(x, na.weight_quant(na.weight)), atol=1e-6)


def test_linear_method_shapes_on_cpu(wf):
    m = wf.BitNetLinearMethod(wf.BitNetConfig.from_config({"block_size": 128}))
    layer = torch.nn.Module()
    m.create_weights(layer, 256, [64, 64], 256, 128, torch.bfloat16, weight_loader="loader")
    assert layer.qweight.shape == (128, 64) and layer.qweight.dtype == torch.uint8
    assert layer.qweight.input_dim == 1 and layer.qweight.output_dim == 0 and layer.qweight.packed_dim == 1
    assert layer.qweight.weight_loader == "loader" and layer.scale.shape == (1,)
    assert wf.BitNetConfig.get_name() == "bitnet"
    with pytest.raises(RuntimeError):
        if torch.cuda.is_available():
            raise RuntimeError("skip")
        m.apply(layer, torch.zeros(1, 256))


def test_torch_operators_are_registered_with_fake_shapes(wf):
    """torch.ops.wf_b200.* exist with the reference's operator argument lists, and their shape-only
    implementations answer without a GPU (cpu_graph_runner.py:340-354 registers the same for the CPU operators)."""
    from torch._subclasses.fake_tensor import FakeTensorMode

    for name in wf.torch_ops.OPERATORS:
        assert hasattr(torch.ops.wf_b200, name)
    with FakeTensorMode():
        pw = torch.empty(64, 32, dtype=torch.uint8, device="cuda")
        a = torch.empty(5, 128, dtype=torch.int8, device="cuda")
        out = torch.ops.wf_b200.bitnet_gemm(pw, a, 0.5)
        assert out.shape == (5, 64) and out.dtype == torch.float32
        assert torch.ops.wf_b200.bitnet_gemv(pw, a[0], 0.5).shape == (64,)
        q, s = torch.ops.wf_b200.bitnet_quantize_activations(torch.empty(5, 128, device="cuda"))
        assert q.dtype == torch.int8 and q.shape == (5, 128) and s.shape == (1,)
        x = torch.empty(2, 3, 128, dtype=torch.bfloat16, device="cuda")
        y = torch.ops.wf_b200.bitlinear(x, pw, torch.empty(2, device="cuda"), None, 0, 1e-5)
        assert y.shape == (2, 3, 64) and y.dtype == torch.bfloat16
        c, sc = torch.ops.wf_b200.pack_ternary(torch.empty(16, 256, device="cuda"), 0, 1e-5)
        assert c.shape == (16, 64) and c.dtype == torch.uint8 and sc.shape == (2,)


def test_model_conversion_inserts_subln(wf):
    """convert_model_to_bitnet (stage1.py:169-214): q/k/v/gate/up become BitLinear with the same parameters,
    o_proj / down_proj become Sequential(SubLN, BitLinear); excluded names are left alone."""
    nn = torch.nn

    class Attn(nn.Module):
        def __init__(self):
            super().__init__()
            self.q_proj, self.k_proj, self.v_proj = nn.Linear(64, 64, bias=False), nn.Linear(64, 32), nn.Linear(64, 32)
            self.o_proj = nn.Linear(64, 64, bias=False)

    class Mlp(nn.Module):
        def __init__(self):
            super().__init__()
            self.gate_proj, self.up_proj, self.down_proj = nn.Linear(64, 128), nn.Linear(64, 128), nn.Linear(128, 64)

    class Layer(nn.Module):
        def __init__(self):
            super().__init__()
            self.self_attn, self.mlp = Attn(), Mlp()

    class Model(nn.Module):
        def __init__(self):
            super().__init__()
            self.embed_tokens = nn.Embedding(10, 64)
            self.layers = nn.ModuleList([Layer(), Layer()])
            self.lm_head = nn.Linear(64, 10, bias=False)

    m = Model()
    before = {k: v.clone() for k, v in m.state_dict().items()}
    wf.convert_model_to_bitnet(m, hidden_size=64, intermediate_size=128)
    for layer in m.layers:
        for name in ("q_proj", "k_proj", "v_proj"):
            assert isinstance(getattr(layer.self_attn, name), wf.BitLinear)
        assert isinstance(layer.self_attn.o_proj, nn.Sequential) and isinstance(layer.self_attn.o_proj[0], wf.SubLN)
        assert isinstance(layer.self_attn.o_proj[1], wf.BitLinear) and layer.self_attn.o_proj[0].hidden_size == 64
        assert isinstance(layer.mlp.down_proj[0], wf.SubLN) and layer.mlp.down_proj[0].hidden_size == 128
        assert isinstance(layer.mlp.gate_proj, wf.BitLinear) and isinstance(layer.mlp.down_proj[1], wf.BitLinear)
    assert type(m.lm_head) is nn.Linear
    assert torch.equal(m.layers[1].mlp.down_proj[1].weight, before["layers.1.mlp.down_proj.weight"])
    assert torch.equal(m.layers[0].self_attn.k_proj.bias, before["layers.0.self_attn.k_proj.bias"])
    x = torch.randn(3, 128)
    sub = m.layers[0].mlp.down_proj[0]
    assert torch.allclose(sub(x), x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6), atol=1e-6)
    assert wf.create_bitnet_config(block_size=128).block_size == 128


def _reference_checkout():
    from oracle.clib import reference_root

    return reference_root()


@pytest.mark.skipif(_reference_checkout() is None, reason="needs a checkout of the reference project")
def test_drop_in_inside_the_reference_tree(wf, monkeypatch):
    """The swap a maintainer makes: the reference's own callers (BitNetFFN, BitNetAttention, the stage-1 converter)
    import `wrinklefree.models.bitlinear`; with that module's classes replaced by the drop-in they build drop-in
    layers, `isinstance` checks hold, and the lambda schedule the reference's trainer installs in ITS module is the
    one the drop-in reads."""
    import importlib
    import sys

    ref = _reference_checkout()
    monkeypatch.syspath_prepend(os.path.join(ref, "packages", "training", "src"))
    for name in [n for n in sys.modules if n == "wrinklefree" or n.startswith("wrinklefree.")]:
        monkeypatch.delitem(sys.modules, name)
    ref_bl = importlib.import_module("wrinklefree.models.bitlinear")
    ref_forward_cls = ref_bl.BitLinear
    for name in ("BitLinear", "BitLinearNoActivationQuant", "convert_linear_to_bitlinear"):
        monkeypatch.setattr(ref_bl, name, getattr(wf, name))
    for name in ("wrinklefree.models.ffn", "wrinklefree.models.attention", "wrinklefree.models"):
        sys.modules.pop(name, None)
    ffn_mod = importlib.import_module("wrinklefree.models.ffn")
    att_mod = importlib.import_module("wrinklefree.models.attention")
    ref_lw = importlib.import_module("wrinklefree.quantization.lambda_warmup")

    torch.manual_seed(1)
    ffn = ffn_mod.BitNetFFN(64, 128, hidden_act="relu2")
    att = att_mod.BitNetAttention(64, 4, 2, 16, max_position_embeddings=16)
    assert isinstance(ffn.gate_proj, wf.BitLinear) and isinstance(att.o_proj, wf.BitLinear)
    # same numbers as the reference's own class on the training formula (gradient enabled -> torch formula on CPU)
    x = torch.randn(2, 5, 64, requires_grad=True)
    twin = ref_forward_cls(64, 128)
    twin.weight.data.copy_(ffn.gate_proj.weight.data)
    assert torch.allclose(ffn.gate_proj(x), twin(x), atol=1e-6)
    y = ffn(x)
    y.sum().backward()
    assert y.shape == (2, 5, 64) and ffn.down_proj.weight.grad is not None
    # the trainer's call (training/stage2.py): the schedule goes into the reference module's global
    warm = ref_lw.LambdaWarmup(warmup_steps=4)
    ref_lw.set_global_lambda_warmup(warm)
    try:
        assert wf.get_current_lambda() == 0.0  # the drop-in sees it
        plain = torch.nn.functional.linear(x, ffn.gate_proj.weight)
        assert torch.allclose(ffn.gate_proj(x), plain, atol=1e-6)  # lambda = 0: no quantization
        warm.step()
        warm.step()
        assert wf.get_current_lambda() == pytest.approx(0.5)
        lam_half = ffn.gate_proj(x)
        assert torch.allclose(lam_half, twin(x), atol=1e-6)  # the reference class mixes with the same lambda
        with torch.no_grad():  # lambda < 1 keeps the drop-in off the packed path even without gradients
            assert torch.allclose(ffn.gate_proj(x.detach()), lam_half.detach(), atol=1e-6)
    finally:
        ref_lw.set_global_lambda_warmup(None)
    assert wf.get_current_lambda() == 1.0
    # and the other direction: a schedule installed through the drop-in's module reaches the reference's global
    wf.set_global_lambda_warmup(wf.LambdaWarmup(warmup_steps=2))
    try:
        assert ref_lw.get_current_lambda() == 0.0
    finally:
        wf.set_global_lambda_warmup(None)
    assert ref_lw.get_global_lambda_warmup() is None


def test_packed_weight_cache_invalidation(wf):
    layer = wf.BitLinear(64, 8)
    layer._packed[torch.float32] = ("stale",)
    layer.load_state_dict({"weight": torch.zeros(8, 64)})
    assert not layer._packed  # loaders write through .data: load_state_dict drops the packed copies
    layer._packed[torch.float32] = ("stale",)
    layer.invalidate_packed()
    assert not layer._packed


def test_host_extension_belongs_to_its_torch(wf, monkeypatch, tmp_path):
    """The extension of the per-call host path is built against torch's C++ interface: it is built again when torch is another
    one, and one that was built for another torch is refused when it is loaded."""
    import importlib.util
    import subprocess

    import torch

    L = wf._lib
    spec = importlib.util.spec_from_file_location("_wf_build_under_test", os.path.join(L.HERE, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    compiled = []
    real_run = subprocess.run

    def run(cmd, **kw):
        if not any(str(c).endswith("wf_host.cpp") for c in cmd):
            return real_run(cmd, **kw)
        compiled.append(cmd)
        open(build.HOST_LIB, "w").close()
        return subprocess.CompletedProcess(cmd, 0, "", "")

    monkeypatch.setattr(build, "HOST_LIB", str(tmp_path / "wf_host.so"))
    monkeypatch.setattr(build.subprocess, "run", run)
    build.build_host_extension()
    build.build_host_extension()
    assert len(compiled) == 1
    assert L.host().torch_version == torch.__version__.split("+")[0]
    monkeypatch.setattr(torch, "__version__", "99.0.0+other")
    build.build_host_extension()
    build.build_host_extension()
    assert len(compiled) == 2
    monkeypatch.setattr(L, "_host", None)
    with pytest.raises(RuntimeError, match="build it again for torch 99.0.0"):
        L.host()
    (tmp_path / "broken.so").write_bytes(b"not a library")
    monkeypatch.setattr(L, "HOST_PATH", str(tmp_path / "broken.so"))
    with pytest.raises(RuntimeError, match="does not load; build it again"):
        L.host()


def test_flags_match_the_header_and_the_stack_rule(wf):
    """The flag values of the Python binding are those of include/wf_b200.h, wf_prefill_quantize validates its
    arguments without a GPU, and the rule that sends a stack of layers to the contraction is monotonic in the token
    count."""
    text = open(os.path.join(ROOT, "include", "wf_b200.h")).read()
    defs = {k: int(v) for k, v in re.findall(r"#define\s+(WF_FLAG_[A-Z_]+)\s+(\d+)u", text)}
    L = wf._lib
    assert defs["WF_FLAG_PDL"] == L.FLAG_PDL and defs["WF_FLAG_X_READY"] == L.FLAG_X_READY
    assert defs["WF_FLAG_WS_READY"] == L.FLAG_WS_READY
    assert defs["WF_FLAG_PREFILL_PAIR"] == L.FLAG_PREFILL_PAIR and defs["WF_FLAG_PREFILL_SINGLE"] == L.FLAG_PREFILL_SINGLE
    assert len(set(defs.values())) == len(defs)  # distinct bits
    lib = L.lib()
    assert lib.wf_prefill_quantize(None, 2, 64, 4, 64, 1e-5, None, 0, 0, None) == 1
    assert b"wf_prefill_quantize" in lib.wf_last_error()
    for k in (2560, 4096, 6912, 14336):
        uses = [wf.stack_uses_contraction(m, k) for m in range(1, 65)]
        assert uses == sorted(uses) and uses[-1] and not uses[0]  # once on the contraction, always from there on
    assert wf.stack_uses_contraction(4, 6912) and not wf.stack_uses_contraction(4, 2560) and wf.stack_uses_contraction(8, 2560)


@pytest.fixture
def launches(wf, monkeypatch):
    """The calls that the operators make into the library, recorded instead of made: (name, arguments)."""
    import contextlib

    from wrinklefree_monorepo_b200 import ops

    calls = []

    class Recorder:
        def __getattr__(self, name):
            return lambda *a: calls.append((name, a)) or 0

    monkeypatch.setattr(ops, "_need_cuda", lambda *ts: None)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops.L, "lib", lambda: Recorder())
    monkeypatch.setattr(torch.cuda, "device", lambda d: contextlib.nullcontext())
    return calls


def test_rope_of_a_prompt_takes_rows_only(wf, launches):
    """The row strides that the launch gets: those of contiguous tensors of any shape and of rows inside wider ones; a tensor whose rows
    lie otherwise is refused, where its first stride was once taken for a row's (and memory far behind the tensor read and written)."""
    from wrinklefree_monorepo_b200 import ops

    b, s, nq, nkv, d, t = 2, 5, 6, 2, 64, 9
    cos = torch.zeros(t, d // 2)
    cache = torch.zeros(b, nkv, t, d, dtype=torch.bfloat16)
    z = lambda *shape: torch.zeros(*shape, dtype=torch.bfloat16)  # noqa: E731
    q, k, v = z(b * s, (nq + 2 * nkv) * d).split([nq * d, nkv * d, nkv * d], 1)
    call = lambda q, k, v: ops.rope_kv_prompt_(q, k, v, cos, cos, cache, cache, s)  # noqa: E731
    good = [((z(b * s, nq * d), z(b * s, nkv * d), z(b * s, nkv * d)), nq * d, nkv * d), ((q, k, v), (nq + 2 * nkv) * d, (nq + 2 * nkv) * d),
            ((z(b, s, nq * d), z(b, s, nkv, d), z(b, s, nkv * d)), nq * d, nkv * d), ((z(b, s, nq, d), z(b * s, nkv * d), z(b, s, nkv, d)), nq * d, nkv * d),
            ((z(b * s * nq * d), k, v), nq * d, (nq + 2 * nkv) * d)]
    for args, ldq, ldk in good:
        del launches[:]
        call(*args)
        (name, a), = launches
        assert name == "wf_rope_kv_prompt_ld_bf16" and a[1] == ldq and a[4] == ldk and a[9:15] == (b, s, nq, nkv, d, t), args[0].shape
    wide = z(b, 2 * s, nq * d)[:, :s]
    for bad in ((wide, z(b * s, nkv * d), z(b * s, nkv * d)), (q, k, v.contiguous()), (q, k.contiguous(), v), (z(b * s, nq * d), z(nkv * d, b * s).t(), z(b * s, nkv * d)),
                (z(b * s, nq * d), z(b * s, nkv * d), z(b * s - 1, nkv * d)), (q.expand(b * s, nq * d).float(), k, v), (z(nq * d).expand(b * s, nq * d), k, v)):
        del launches[:]
        with pytest.raises(ValueError):
            call(*bad)
        assert not launches


def test_gate_activation_takes_rows_only(wf, launches):
    """gate and up share one row stride: contiguous ones in any shape of up, rows of wider tensors when both are; up was once read at
    gate's stride whatever its own."""
    from wrinklefree_monorepo_b200 import ops

    m, i = 5, 64
    z = lambda *shape: torch.zeros(*shape, dtype=torch.bfloat16)  # noqa: E731
    g, u = z(m, 2 * i).split(i, 1)
    q, scale = torch.zeros(m, i, dtype=torch.int8), torch.zeros(m)
    for gate, up, ld, rows in ((z(m, i), z(m, i), i, m), (z(m, i), z(m * i), i, m), (g, u, 2 * i, m), (g[:1], u[:1], i, 1), (g[::2], u[::2], 4 * i, 3)):
        del launches[:]
        ops.act_mul_quant(gate, up, q, scale)
        (name, a), = launches
        assert name == "wf_act_mul_quant_ld_bf16" and a[2] == ld and a[6:8] == (rows, i)
    for gate, up in ((g, u.contiguous()), (g.contiguous(), u), (z(i, m).t(), z(i, m).t()), (g, u[::2]), (z(m, i), z(m - 1, i)), (g.float(), u.float()),
                     (z(1, i).expand(m, i), z(1, i).expand(m, i))):
        del launches[:]
        with pytest.raises(ValueError):
            ops.act_mul_quant(gate, up, q, scale)
        assert not launches


def test_argmax_increments_an_int64_scalar_only(wf, launches):
    """`pos` is written as one int64: another type or length, or another device's tensor, is refused."""
    from wrinklefree_monorepo_b200 import ops

    x, out = torch.zeros(3, 8, dtype=torch.bfloat16), torch.zeros(3, dtype=torch.long)
    for pos in (None, torch.zeros((), dtype=torch.long), torch.zeros(1, dtype=torch.long)):
        ops.argmax_(x, out, pos)
    assert len(launches) == 3
    for pos in (torch.zeros((), dtype=torch.int32), torch.zeros(()), torch.zeros(0, dtype=torch.long), torch.zeros(2, dtype=torch.long),
                torch.zeros((), dtype=torch.long, device="meta")):
        with pytest.raises(ValueError):
            ops.argmax_(x, out, pos)
    with pytest.raises(ValueError):
        ops.argmax_(x, out.to("meta"))
    assert len(launches) == 3


def test_projections_side_by_side_take_their_scales_and_workspace_only(wf, launches):
    """What the launch reads by address alone: the scale of each token and row, and the workspace by its bytes."""
    from wrinklefree_monorepo_b200 import ops

    m, n, k = 3, 10, 64
    good = dict(x=torch.zeros(m, k, dtype=torch.int8), x_scale=torch.zeros(m), codes=torch.zeros(n, k // 4, dtype=torch.uint8), row_scale=torch.zeros(n),
                out=torch.zeros(m, n + 2)[:, :n], workspace=torch.zeros(4096, dtype=torch.uint8))
    ops.bitlinear_rows(**good)
    assert len(launches) == 1 and launches[0][1][8:11] == (m, n, k)
    for name, bad in (("x_scale", torch.zeros(m - 1)), ("x_scale", torch.zeros(m).half()), ("x_scale", torch.zeros(2 * m)[::2]), ("row_scale", torch.zeros(2 * n)[::2]),
                      ("codes", torch.zeros(n, k // 4)), ("workspace", torch.zeros(4096)), ("workspace", good["workspace"].to("meta")), ("x_scale", torch.zeros(m, device="meta"))):
        with pytest.raises(ValueError):
            ops.bitlinear_rows(**{**good, name: bad})
    assert len(launches) == 1


def test_prompt_attention_takes_rows_only(wf, launches):
    """q in rows of its own or of a wider tensor, whole caches and output: the launch writes B * s rows of out and reads as many of q."""
    from wrinklefree_monorepo_b200 import ops

    b, s, nq, nkv, d, t = 2, 5, 6, 2, 64, 9
    z = lambda *shape: torch.zeros(*shape, dtype=torch.bfloat16)  # noqa: E731
    good = dict(q=z(b * s, nq * d), kcache=z(b, nkv, t, d), vcache=z(b, nkv, t, d), out=z(b * s, nq * d), s=s)
    for q, ld in ((good["q"], nq * d), (z(b * s, nq * d + 16)[:, :nq * d], nq * d + 16), (z(b, s, nq * d), nq * d)):
        del launches[:]
        ops.attn_prompt(**{**good, "q": q})
        (name, a), = launches
        assert name == "wf_attn_prompt_bf16" and a[1] == ld and a[5:11] == (b, s, nq, nkv, d, t)
    del launches[:]
    for name, bad in (("q", z(b, 2 * s, nq * d)[:, :s]), ("q", z(b * s - 1, nq * d)), ("q", good["q"].float()), ("out", z(b * s - 1, nq * d)), ("out", z(b * s, nq * d + 8)[:, :nq * d]),
                      ("out", z(b * s, (nq + 1) * d)), ("out", good["out"].float()), ("kcache", z(b, nkv, 2 * t, d)[:, :, :t]), ("vcache", z(b, nkv, t - 1, d)),
                      ("vcache", good["vcache"].to("meta"))):
        with pytest.raises(ValueError):
            ops.attn_prompt(**{**good, name: bad})
    assert not launches


def test_layers_in_one_launch_take_their_shapes_only(wf, launches):
    """The launch has nothing but addresses: what lies behind each is looked at when the descriptors are made, and at each run."""
    from wrinklefree_monorepo_b200 import ops

    B, hidden, nq, nkv, d, inter, t = 2, 128, 4, 2, 64, 192, 5
    z = lambda *shape, dtype=torch.bfloat16: torch.zeros(*shape, dtype=dtype)  # noqa: E731
    shapes = ((nq * d, hidden), (nkv * d, hidden), (nkv * d, hidden), (hidden, nq * d), (inter, hidden), (inter, hidden), (hidden, inter))

    def layer(**other):
        return {**dict(codes=[z(n, k // 4, dtype=torch.uint8) for n, k in shapes], scales=[torch.zeros(2) for _ in shapes], norms=[z(hidden), z(hidden)],
                       caches=[z(B, nkv, t, d), z(B, nkv, t, d)]), **other}

    def make(*layers, norm_f=z(hidden), cos=torch.zeros(t, d // 2)):
        return ops.DecodeLayers(list(layers), hidden, nq, nkv, inter, "silu", 1e-5, norm_f, cos, torch.zeros(t, d // 2), 16)

    good = make(layer(), layer())
    h, pos = z(B, hidden), torch.zeros((), dtype=torch.long)
    good.run(h, h, pos)
    assert len(launches) == 1 and launches[0][1][8:15] == (B, hidden, nq, nkv, d, inter, t)
    for bad in ((h[:1], h, pos), (h.float(), h, pos), (h, z(B, 2 * hidden)[:, :hidden], pos), (h, h, pos.int()), (h, h, torch.zeros(2, dtype=torch.long)), (h, h, pos.to("meta"))):
        with pytest.raises(ValueError):
            good.run(*bad)
    assert len(launches) == 1
    codes = layer()["codes"]
    for bad in (dict(caches=[z(B, nkv, t + 1, d), z(B, nkv, t + 1, d)]), dict(caches=[z(B, nkv, t, d), z(B, nkv, t, d).float()]), dict(norms=[z(hidden), z(inter)]),
                dict(codes=codes[:6] + codes[:1]), dict(codes=[c.to(torch.int16) for c in codes]), dict(scales=[torch.zeros(2, dtype=torch.float64)] * 7), dict(scales=[torch.zeros(1)] * 6)):
        with pytest.raises(ValueError):
            make(layer(), layer(**bad))
    for bad in (dict(norm_f=z(inter)), dict(norm_f=torch.zeros(hidden)), dict(cos=torch.zeros(t - 1, d // 2)), dict(cos=torch.zeros(t, d // 2, dtype=torch.float64))):
        with pytest.raises(ValueError):
            make(layer(), **bad)


def test_native_prompt_loop_takes_its_shapes_only(wf):
    """The loop over the layers has the types and shapes of all it is given looked at before anything else: tensors that pass it on
    the CPU are refused for not being on the GPU, others for what they are."""
    B, S, nq, nkv, d, inter, t = 2, 3, 4, 2, 64, 192, 5
    hidden, qd, kvd, m = 128, nq * d, nkv * d, B * S
    z = lambda *shape, dtype=torch.bfloat16: torch.zeros(*shape, dtype=dtype)  # noqa: E731
    codes = lambda n, k: z(n, k // 4, dtype=torch.uint8)  # noqa: E731

    def layer(**other):
        one = dict(qkv=codes(qd + 2 * kvd, hidden), qkv_s=torch.zeros(qd + 2 * kvd), o=codes(hidden, qd), o_s=torch.zeros(2), gu=codes(2 * inter, hidden), gu_s=torch.zeros(2 * inter),
                   down=codes(hidden, inter), down_s=torch.zeros(2), n1=z(hidden), n2=z(hidden), kc=z(B, nkv, t, d), vc=z(B, nkv, t, d))
        return tuple({**one, **other}.values())

    def call(*layers, **other):
        a = dict(h=z(m, hidden), cos=torch.zeros(t, d // 2), sin=torch.zeros(t, d // 2), xq=z(m * qd, dtype=torch.int8), aq=z(m, inter, dtype=torch.int8), scale=torch.zeros(m),
                 qkv=z(m, qd + 2 * kvd), gu=z(m, 2 * inter), att=z(m, qd), res=z(m, hidden), ws=z(4096, dtype=torch.uint8))
        wf._lib.host().prompt_layers(list(layers), *{**a, **other}.values(), B, S, nq, nkv, d, 0, 1e-5, 64, 16, 4096)

    with pytest.raises(RuntimeError, match="CUDA"):
        call(layer(), layer())
    for bad in (dict(h=torch.zeros(m, hidden)), dict(res=torch.zeros(m, hidden)), dict(qkv=z(m, qd + 2 * kvd).half()), dict(scale=torch.zeros(m).double()), dict(ws=torch.zeros(4096)),
                dict(cos=torch.zeros(S - 1, d // 2)), dict(aq=z(m, inter, dtype=torch.uint8)), dict(att=z(m - 1, qd))):
        with pytest.raises(ValueError):
            call(layer(), **bad)
    for bad in (dict(kc=z(B, nkv, t, d).float(), vc=z(B, nkv, t, d).float()), dict(kc=z(B, nkv, t - 1, d), vc=z(B, nkv, t - 1, d)), dict(n1=torch.zeros(hidden)),
                dict(o=codes(hidden, qd).to(torch.int8)), dict(o_s=torch.zeros(0)), dict(down_s=torch.zeros(2).half()), dict(kc=z(B * nkv, t, d)), dict(gu_s=torch.zeros(2 * inter + 1))):
        with pytest.raises(ValueError):
            call(layer(), layer(**bad))


def test_decode_step_with_embeddings_that_require_gradients(wf):
    """A decoder made of a model's named_parameters holds an embedding that requires gradients; a step gathers its rows all the same."""
    from wrinklefree_monorepo_b200.decoder import SMOLLM2_135M, TernaryDecoder

    m = object.__new__(TernaryDecoder)
    m.cfg, m.B, m.masked, m.attention = SMOLLM2_135M, 2, True, "kernel"
    m.embed, m.tok, m.h = torch.randn(5, 8, requires_grad=True), torch.tensor([3, 1]), torch.empty(2, 8)
    m.resident = type("Resident", (), {"run": lambda *a, **k: None, "holds": lambda *a: True})()
    m.xf = m.head_out = m.pos = m.layers = m.norm_f = m.cos = m.sin = None
    m._head, m._greedy = lambda *a, **k: None, lambda *a, **k: None
    m._decode_step()
    assert torch.equal(m.h, m.embed[[3, 1]]) and not m.h.requires_grad


@pytest.mark.parametrize("name", ["norm_f", "cos", "sin", "n1", "n2", "kc", "vc", "layers", None])
def test_decode_step_takes_tensors_put_in_place_of_others(wf, launches, monkeypatch, name):
    """The one launch for all layers has the addresses of what the decoder was built with.  Rotary tables, a norm weight or a cache that a
    caller has put in another's place are what the next step computes with: it takes the separate launches then."""
    from wrinklefree_monorepo_b200 import ops
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    B, hidden, nq, nkv, d, inter, t = 2, 128, 4, 2, 64, 192, 5
    z = lambda *shape, dtype=torch.bfloat16: torch.zeros(*shape, dtype=dtype)  # noqa: E731
    shapes = dict(q=(nq * d, hidden), k=(nkv * d, hidden), v=(nkv * d, hidden), o=(hidden, nq * d), gate=(inter, hidden), up=(inter, hidden), down=(hidden, inter))
    m = object.__new__(TernaryDecoder)
    m.cfg = DecoderConfig(layers=2, hidden=hidden, n_q=nq, n_kv=nkv, head_dim=d, intermediate=inter, vocab=7)
    m.B, m.T, m.tp, m.prefetch, m._fuse_opt, m.dtype, m.dev = B, t, 1, False, None, torch.bfloat16, "cpu"
    m.masked, m.attention, m.fused, m.head_out = True, "kernel", True, None
    m.layers = [{**{n: (z(r, k // 4, dtype=torch.uint8), torch.zeros(2)) for n, (r, k) in shapes.items()}, "n1": z(hidden), "n2": z(hidden),
                 "kc": z(B, nkv, t, d), "vc": z(B, nkv, t, d)} for _ in range(2)]
    m.norm_f, m.cos, m.sin = z(hidden), torch.zeros(t, d // 2), torch.zeros(t, d // 2)
    m.embed, m.tok, m.pos, m.h, m.xf = z(7, hidden), torch.zeros(B, dtype=torch.long), torch.zeros((), dtype=torch.long), z(B, hidden), z(B, hidden)
    cluster = type("Lib", (), {"wf_decode_layers_cluster": lambda *a: 16, "__getattr__": lambda s, n: lambda *a: launches.append((n, a)) or 0})()
    monkeypatch.setattr(ops.L, "lib", lambda: cluster)
    m.resident = m._resident_layers()
    m._head, m._greedy, m._decode_step_fused = lambda *a, **k: None, lambda *a, **k: None, lambda: launches.append(("separate", ()))
    if name in ("norm_f", "cos", "sin"):
        setattr(m, name, getattr(m, name).clone())
    elif name == "layers":
        m.layers = m.layers[:1]
    elif name:
        m.layers[1][name] = m.layers[1][name].clone()
    m._decode_step()
    assert [n for n, _ in launches] == ["separate" if name else "wf_decode_layers_bf16"]


def test_which_prompts_the_attention_kernel_takes(wf):
    """Shapes that the launch refuses stay with the framework's attention: 65536 sequences of one token were sent to it."""
    from wrinklefree_monorepo_b200 import decoder

    takes = decoder._prompt_kernel_takes
    assert takes(1, 121, 9, 3, 64) and takes(65535, 1, 1, 1, 64) and not takes(65536, 1, 1, 1, 64)
    assert not takes(1, 8, 4, 2, 96) and not takes(1, 8, 4, 3, 64) and not takes(1, 1 << 14, 1, 1, 64)
