"""Decoder harness: the CUDA-graphed decode step (KV cache, RoPE, masking, grouped projections) must agree
with the prefill pass over the same tokens, which takes the other kernel path for every projection."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_stepwise_decode_matches_prefill(wf):
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    cfg = DecoderConfig(layers=2, hidden=256, n_q=4, n_kv=2, head_dim=64, intermediate=512, vocab=1000)
    dev = torch.device("cuda", 0)
    B, S, T = 3, 9, 16
    g = torch.Generator().manual_seed(5)
    ids = torch.randint(0, cfg.vocab, (B, S), generator=g).to(dev)

    m1 = TernaryDecoder(cfg, B, T, dev, seed=1)
    ref = m1.prefill(ids).float()
    assert int(m1.pos) == S

    m2 = TernaryDecoder(cfg, B, T, dev, seed=1)
    m2.capture(masked=True)
    assert int(m2.pos) == 0
    for t in range(S):
        m2.tok.copy_(ids[:, t])
        m2.graph.replay()
    torch.cuda.synchronize()
    got = m2.logits.float()
    assert int(m2.pos) == S
    err = float((got - ref).abs().max() / ref.abs().max())
    assert err < 3e-2, err
    assert (got.argmax(-1) == ref.argmax(-1)).float().mean() >= 2 / 3
    # the caches hold the same keys
    kerr = float((m1.layers[0]["kc"][:, :, :S].float() - m2.layers[0]["kc"][:, :, :S].float()).abs().max())
    assert kerr < 2e-2, kerr
    # greedy continuation runs and stays in range
    out = m2.decode(4)
    assert out.shape == (B, 4) and int(out.max()) < cfg.vocab
    wf.device_status()


@pytest.mark.parametrize("B", [1, 5, 20])
def test_graphed_step_reads_what_its_predecessor_wrote(wf, B):
    """In a replayed graph every launch starts while its predecessor still runs.  At widths whose projections read int8
    copies, made by kernels of their own, each step must use this step's activations and not the previous replay's: the
    graphed steps equal the same steps launched one by one, with other tokens in every step."""
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    cfg = DecoderConfig(layers=2, hidden=4096, n_q=32, n_kv=8, head_dim=128, intermediate=14336, vocab=1000)
    dev = torch.device("cuda", 0)
    ids = torch.randint(0, cfg.vocab, (B, 12), generator=torch.Generator().manual_seed(6)).to(dev)
    m = TernaryDecoder(cfg, B, 16, dev, seed=2)
    m.capture()
    assert m.qnorm and m.qact

    def steps(one):
        m.prefill(ids[:, :6])
        out = []
        for t in range(6, 12):
            m.tok.copy_(ids[:, t])
            one()
            torch.cuda.synchronize()
            out.append(m.logits.clone())
        return torch.stack(out)

    graphed = steps(lambda: m.graph.replay())
    plain = steps(lambda: m._decode_step())
    assert torch.equal(graphed, plain)
    wf.device_status()


@pytest.mark.parametrize("B,S,nq,nkv,D,T", [(1, 1, 1, 1, 16, 1), (2, 7, 9, 3, 64, 11), (1, 130, 32, 8, 128, 130), (3, 33, 4, 4, 48, 40)])
def test_rope_and_cache_write_of_a_prompt(wf, B, S, nq, nkv, D, T):
    """One launch for the rotation of q and k and the cache write of a prompt: bit for bit the operator chain it stands for;
    positions behind the prompt stay as they were."""
    from wrinklefree_monorepo_b200 import ops
    from wrinklefree_monorepo_b200.decoder import _rope

    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(B * 100 + S)
    q, k, v = (torch.randn(B * S, n * D, generator=g).bfloat16().to(dev) for n in (nq, nkv, nkv))
    ang = torch.rand(T, D // 2, generator=g).to(dev) * 6
    cos, sin = ang.cos(), ang.sin()
    kc, vc = (torch.full((B, nkv, T, D), 3.0, dtype=torch.bfloat16, device=dev) for _ in range(2))
    want_q, want_k = (_rope(t.view(B, S, n, D).transpose(1, 2), cos[:S], sin[:S]) for t, n in ((q, nq), (k, nkv)))
    ops.rope_kv_prompt_(q, k, v, cos, sin, kc, vc, S)
    assert torch.equal(q.view(B, S, nq, D).transpose(1, 2), want_q) and torch.equal(kc[:, :, :S], want_k)
    assert torch.equal(vc[:, :, :S], v.view(B, S, nkv, D).transpose(1, 2))
    assert bool((kc[:, :, S:] == 3.0).all()) and bool((vc[:, :, S:] == 3.0).all())


def test_fused_elementwise_kernels(wf):
    from wrinklefree_monorepo_b200 import ops

    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(3)
    M, K = 5, 576
    h = torch.randn(M, K, generator=g).bfloat16().to(dev)
    delta = torch.randn(M, K, generator=g).bfloat16().to(dev)
    w = (1 + 0.1 * torch.randn(K, generator=g)).bfloat16().to(dev)
    want_h = (h + delta)
    v = want_h.float()
    want_y = (v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + 1e-5)).to(torch.bfloat16) * w
    y = torch.empty_like(h)
    h2 = h.clone()
    ops.add_rmsnorm_(h2, delta, w, y, 1e-5)
    assert torch.equal(h2, want_h)
    assert float((y.float() - want_y.float()).abs().max()) <= 2e-2 * float(want_y.float().abs().max())
    y0 = torch.empty_like(h)
    ops.add_rmsnorm_(h2, None, w, y0, 1e-5)
    assert torch.equal(y0, y)

    gate = torch.randn(4, 512, generator=g).bfloat16().to(dev)
    up = torch.randn(4, 512, generator=g).bfloat16().to(dev)
    out = torch.empty_like(gate)
    ops.act_mul(gate, up, out, "silu")
    ref = torch.nn.functional.silu(gate) * up
    assert float((out.float() - ref.float()).abs().max()) <= 2e-2 * float(ref.float().abs().max())
    ops.act_mul(gate, up, out, "relu2")
    ref = torch.relu(gate).pow(2) * up
    assert float((out.float() - ref.float()).abs().max()) <= 2e-2 * float(ref.float().abs().max())

    B, nq, nkv, D, T = 3, 4, 2, 64, 16
    q = torch.randn(B, nq * D, generator=g).bfloat16().to(dev)
    k = torch.randn(B, nkv * D, generator=g).bfloat16().to(dev)
    vv = torch.randn(B, nkv * D, generator=g).bfloat16().to(dev)
    inv = 1.0 / (1e4 ** (torch.arange(0, D, 2, dtype=torch.float32) / D))
    ang = torch.arange(T, dtype=torch.float32)[:, None] * inv[None, :]
    cos, sin = ang.cos().to(dev), ang.sin().to(dev)
    pos = torch.tensor(21, dtype=torch.long, device=dev)  # slot 21 % 16 = 5
    kc = torch.zeros(B, nkv, T, D, dtype=torch.bfloat16, device=dev)
    vc = torch.zeros_like(kc)

    def rope(x, c, s):
        x1, x2 = x[..., : D // 2].float(), x[..., D // 2 :].float()
        return torch.cat([x1 * c - x2 * s, x2 * c + x1 * s], -1).to(torch.bfloat16)

    want_q = rope(q.view(B, nq, D), cos[5], sin[5]).reshape(B, nq * D)
    want_k = rope(k.view(B, nkv, D), cos[5], sin[5])
    ops.rope_kv_(q, k, vv, cos, sin, pos, kc, vc)
    assert torch.equal(q, want_q)
    assert torch.equal(kc[:, :, 5], want_k) and torch.equal(vc[:, :, 5], vv.view(B, nkv, D))
    assert not kc[:, :, 4].any() and not kc[:, :, 6].any()


# ---------------------------------------------------------------- against the reference's own model
import os  # noqa: E402

import numpy as np  # noqa: E402

import inputs as gi  # noqa: E402

GOLD = os.path.join(os.path.dirname(__file__), "golden")


def _fixture_decoder(act, dtype, pack_mode):
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    c = gi.MODEL_CFG
    z = np.load(os.path.join(GOLD, f"model_{act}.npz"))
    weights, ids = gi.model_weights(), gi.model_ids()
    assert gi.sha(ids.numpy(), *[weights[k].numpy() for k in sorted(weights)]) == str(z["input_sha"])
    cfg = DecoderConfig(layers=c["layers"], hidden=c["hidden"], n_q=c["n_q"], n_kv=c["n_kv"], head_dim=c["head_dim"],
                        intermediate=c["intermediate"], vocab=c["vocab"], rope_theta=c["rope_theta"], act=act,
                        eps=c["norm_eps"], subln=True)
    dev = torch.device("cuda", 0)
    model = TernaryDecoder(cfg, gi.MODEL_BATCH, c["max_pos"], dev, dtype=dtype, weights=weights, pack_mode=pack_mode)
    return model, ids.to(dev), z


def _nerr(got, ref):
    return float(np.abs(got - ref).max() / np.abs(ref).max())


@pytest.mark.parametrize("act", ["relu2", "silu"])
def test_prefill_equals_reference_model_fp32(wf, act):
    """TernaryDecoder.prefill on the weights of the reference's BitNetLlama (2 layers at SmolLM2-135M widths, SubLN,
    GQA, interleaved RoPE) against the reference's own fp32 forward, per position, err = max|a-b| / max|b|.

    Rounding to int8 is discontinuous: an input that lands within a few 1e-7 of a rounding boundary is rounded the
    other way when the fp32 summation order of a norm differs, that one code moves the token's hidden state by
    ~1e-3, and the next quantizations amplify it to ~1e-2 at the logits.  The reference does this to itself: adding
    3e-7 relative noise to its embeddings left 44 of 54 positions within 5e-7 and moved the other 10 by 0.5-1.7 %.
    So: at least 60 % of the positions must agree to 1e-5 (the computation is the same one), and no position may be
    off by more than 3e-2 (a rounding cascade, not a different model)."""
    model, ids, z = _fixture_decoder(act, torch.float32, torch.float32)
    logits = model.prefill(ids, all_logits=True)
    got = logits[:, gi.MODEL_KEEP_FROM:].float().cpu().numpy()
    ref = z["logits_f32"]
    err = np.abs(got - ref).max(-1) / np.abs(ref).max()  # [batch, position]
    np.set_printoptions(precision=1, linewidth=250)
    print(f"fp32 {act}: per-position error\n{err}")
    # A position's result depends on every earlier position of its sequence through attention, so a cascade, once
    # started, reaches the later positions of that sequence.  Measured: 45 / 36 of the 54 positions (relu2 / silu)
    # agree to 1e-6, the others sit at 5e-4 .. 1.7e-2.
    assert (err <= 1e-5).mean() >= 0.6, (err <= 1e-5).mean()
    assert err.max() <= 3e-2, err.max()
    assert (got.argmax(-1) == ref.argmax(-1)).mean() >= 0.9
    wf.device_status()


@pytest.mark.parametrize("act", ["relu2", "silu"])
def test_bf16_prefill_and_decode_steps_follow_reference_model(wf, act):
    """bf16 end to end, weights ternarized by the cast-first rule of BitLinear.forward.  Held to the reference's bf16
    forward within max|a-b| / max|b| <= 6e-2 (measured 0.037-0.041): the reference evaluates its norms, residuals and
    attention in bf16 arithmetic, this decoder in fp32 with one rounding, so int8 codes near a rounding boundary differ
    and the random two-layer network amplifies that.  For scale: the reference's own bf16 and fp32 forwards differ by
    0.16 on this fixture, and this decoder must sit as close to the bf16 reference as that (checked as well).  The
    CUDA-graphed decode step (fused norm, RoPE + cache write, grouped projections) is then teacher-forced over the next
    positions and held to the same logits."""
    model, ids, z = _fixture_decoder(act, torch.bfloat16, torch.bfloat16)
    S, K0 = gi.MODEL_PROMPT, gi.MODEL_KEEP_FROM
    logits = model.prefill(ids[:, :S], all_logits=True)
    got = logits[:, K0:].float().cpu().numpy()
    e_bf16, e_f32 = _nerr(got, z["logits_bf16"][:, :S - K0]), _nerr(got, z["logits_f32"][:, :S - K0])
    print(f"prefill {act}: vs bf16 reference {e_bf16:.4f}, vs fp32 reference {e_f32:.4f}")
    ref_gap = _nerr(z["logits_bf16"], z["logits_f32"])  # what bf16 arithmetic alone costs the reference
    assert e_bf16 <= 6e-2 and e_bf16 < ref_gap / 2 and e_f32 <= 1.5 * ref_gap, (e_bf16, e_f32, ref_gap)
    model.capture(masked=True)
    for i in range(gi.MODEL_STEPS):
        model.tok.copy_(ids[:, S + i])
        model.graph.replay()
        torch.cuda.synchronize()
        step = model.logits.float().cpu().numpy()
        e1, e2 = _nerr(step, z["logits_bf16"][:, S - K0 + i]), _nerr(step, z["logits_f32"][:, S - K0 + i])
        print(f"step {i} {act}: vs bf16 reference {e1:.4f}, vs fp32 reference {e2:.4f}")
        assert e1 <= 6e-2 and e2 <= 1.5 * ref_gap, (i, e1, e2)
    wf.device_status()


@pytest.mark.parametrize("B,nq,nkv,D,T,pos", [(1, 32, 8, 128, 2080, 2047), (3, 9, 3, 64, 100, 37), (32, 32, 8, 128, 300, 299),
                                              (2, 4, 4, 64, 64, 0), (5, 8, 1, 128, 1000, None), (7, 6, 2, 64, 130, 128), (300, 8, 4, 128, 70, 69)])
def test_decode_attention_kernel(wf, B, nq, nkv, D, T, pos):
    """The decode-step attention kernel (grouped-query heads, context split over CTAs and merged in the launch, bf16
    cache) against fp32 softmax attention over the valid positions: max|a-b| / max|b| <= 1e-2 (the probabilities are
    rounded to bf16 in front of the second product, the output is bf16).  Positions beyond the valid length hold
    large garbage that must not leak in."""
    from wrinklefree_monorepo_b200 import ops

    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(B * 1000 + T)
    q = torch.randn(B, nq * D, generator=g).bfloat16().to(dev)
    kc = torch.randn(B, nkv, T, D, generator=g).bfloat16().to(dev)
    vc = torch.randn(B, nkv, T, D, generator=g).bfloat16().to(dev)
    n_valid = T if pos is None else pos + 1
    kc[:, :, n_valid:] = 1e4
    vc[:, :, n_valid:] = -1e4
    out = torch.empty(B, nq * D, dtype=torch.bfloat16, device=dev)
    pos_t = None if pos is None else torch.tensor(pos, dtype=torch.long, device=dev)
    for _ in range(2):  # the merge tickets must be reusable
        out.fill_(7)
        ops.attn_decode(q, kc, vc, pos_t, out)
        qf = q.float().view(B, nkv, nq // nkv, D)
        kf, vf = kc.float()[:, :, :n_valid], vc.float()[:, :, :n_valid]
        s = torch.einsum("bhgd,bhtd->bhgt", qf, kf) * D ** -0.5
        ref = torch.einsum("bhgt,bhtd->bhgd", torch.softmax(s, -1), vf).reshape(B, nq * D)
        err = float((out.float() - ref).abs().max() / ref.abs().max())
        assert err <= 1e-2, err


def test_attention_workspace_of_a_captured_step(wf):
    """A captured step keeps its own attention workspace: a later, larger attention call and tensors allocated after it leave
    the replays what the same steps are without a graph."""
    from wrinklefree_monorepo_b200 import ops
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    cfg = DecoderConfig(layers=2, hidden=256, n_q=4, n_kv=2, head_dim=64, intermediate=512, vocab=1000)
    dev = torch.device("cuda", 0)
    T = 520  # several tiles per unit: partial results that CTAs merge through the workspace
    ids = torch.randint(0, cfg.vocab, (1, T), generator=torch.Generator().manual_seed(4)).to(dev)
    want = []
    for graphed in (False, True):
        m = TernaryDecoder(cfg, 1, T, dev, seed=3)
        if graphed:
            m.capture()
            big = torch.zeros(64, 8, 1024, 128, dtype=torch.bfloat16, device=dev)
            q = torch.zeros(64, 32 * 128, dtype=torch.bfloat16, device=dev)
            ops.attn_decode(q, big, big, None, torch.empty_like(q))
            filled = [torch.full((1 << 18,), 255, dtype=torch.uint8, device=dev) for _ in range(64)]
        m.prefill(ids[:, : T - 6])
        for t in range(T - 6, T):
            m.tok.copy_(ids[:, t])
            m.graph.replay() if graphed else m._decode_step()
            torch.cuda.synchronize()
            if graphed:
                assert torch.equal(m.logits, want[t - T + 6]), t
            else:
                want.append(m.logits.clone())
    assert all(bool((f == 255).all()) for f in filled)
    wf.device_status()


def test_attention_calls_without_a_workspace(wf):
    """Calls on two streams never share partial results or tickets, a captured call owns its workspace, the kept ones are
    bounded, and a growing context replaces only its own stream's."""
    from wrinklefree_monorepo_b200 import ops

    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(1)
    ins = []
    for t in (640, 2048, 320, 4096):
        kc, vc = (torch.randn(1, 2, t, 64, generator=g, device=dev).bfloat16() for _ in range(2))
        ins.append((torch.randn(1, 4 * 64, generator=g, device=dev).bfloat16(), kc, vc))

    def call(i):
        q, kc, vc = ins[i % len(ins)]
        return ops.attn_decode(q, kc, vc, None, torch.empty_like(q))

    want = [call(i) for i in range(len(ins))]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(ops.ATTN_WORKSPACES + 4)]
    got = []
    for i in range(12 * len(streams)):
        with torch.cuda.stream(streams[i % len(streams)]):
            got.append((i, call(i + i // len(streams))))
    torch.cuda.synchronize()
    assert all(torch.equal(o, want[(i + i // len(streams)) % len(ins)]) for i, o in got)
    assert len(ops._attn_ws) <= ops.ATTN_WORKSPACES
    assert len({ws.data_ptr() for ws in ops._attn_ws.values()}) == len(ops._attn_ws)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = [call(i) for i in range(len(ins))]
    ops._attn_ws.clear()
    torch.cuda.empty_cache()
    for _ in range(2):
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out, want))


def test_fused_inputs_of_grouped_projections(wf, oracle_c):
    """The fused input modes of the grouped decode kernel against the unfused kernels of the library: rmsnorm(x + x2)
    in front of a q/k/v-like group (all three forms of the kernel: shared tokens, a single matrix, a streaming
    stack), and act(gate) * up in front of a down-like projection.  Activation modes: accumulators and outputs
    identical to the unfused chain.  Norm mode: the residual output identical; the projection outputs within 1e-2
    (the mean of squares is summed in another order, which may move single int8 codes)."""
    from wrinklefree_monorepo_b200 import ops

    dev = torch.device("cuda", 0)
    g = torch.Generator().manual_seed(11)
    for (m, k, ns) in ((1, 4096, (4096, 1024, 1024)), (5, 576, (576, 192, 192)), (3, 2560, (6912,)), (20, 640, (512, 512))):
        h = torch.randn(m, k, generator=g).bfloat16().to(dev)
        delta = torch.randn(m, k, generator=g).bfloat16().to(dev)
        w = (1 + 0.1 * torch.randn(k, generator=g)).bfloat16().to(dev)
        mats = [wf.pack_ternary((torch.randn(n, k, generator=g) * 0.02).to(dev)) for n in ns]
        for with_delta in (True, False):
            # unfused: norm kernel, then the group on its output
            h_ref = h.clone()
            xn = torch.empty_like(h)
            ops.add_rmsnorm_(h_ref, delta if with_delta else None, w, xn, 1e-5)
            ref = ops.DecodeGroup([dict(x=xn, codes=c, w_scale=s_, out_dtype=torch.float32) for c, s_ in mats]).run()
            h_out = torch.zeros_like(h)
            probs = [dict(x=h, x2=delta if with_delta else None, x_mode="norm", norm_w=w, norm_eps=1e-5, codes=c, w_scale=s_,
                          out_dtype=torch.float32, h_out=h_out if i == 0 else None) for i, (c, s_) in enumerate(mats)]
            grp = ops.DecodeGroup(probs)
            for pdl in (False, True):
                h_out.zero_()
                got = grp.run(pdl=pdl)
                assert torch.equal(h_out, h_ref), (m, k, with_delta)
                for a, b in zip(got, ref):
                    err = float((a - b).abs().max() / b.abs().max())
                    assert err <= 1e-2, (m, k, with_delta, err)
    # a streaming stack (thousands of row items) with the norm fused in
    m, k = 2, 1024
    h = torch.randn(m, k, generator=g).bfloat16().to(dev)
    w = (1 + 0.1 * torch.randn(k, generator=g)).bfloat16().to(dev)
    mats = [wf.pack_ternary((torch.randn(6000 + 16 * i, k, generator=g) * 0.02).to(dev)) for i in range(8)]
    xn = torch.empty_like(h)
    ops.add_rmsnorm_(h.clone(), None, w, xn, 1e-6)
    ref = ops.DecodeGroup([dict(x=xn, codes=c, w_scale=s_, out_dtype=torch.float32) for c, s_ in mats]).run()
    got = ops.DecodeGroup([dict(x=h, x_mode="norm", norm_w=w, norm_eps=1e-6, codes=c, w_scale=s_, out_dtype=torch.float32) for c, s_ in mats]).run(pdl=True)
    for a, b in zip(got, ref):
        assert float((a - b).abs().max() / b.abs().max()) <= 1e-2
    # activation modes: bit-exact against act_mul + projection; `few`: on the launch for one or two tokens
    for (m, k, n, mode, few) in ((1, 14336, 4096, "silu", False), (4, 1536, 576, "relu2", False), (9, 1024, 300, "silu", False),
                                 (33, 640, 128, "relu2", False), (1, 1536, 576, "silu", True), (1, 6912, 2560, "relu2", True),
                                 (1, 16384, 70, "silu", True), (2, 1536, 576, "relu2", True), (2, 4096, 2560, "silu", True), (2, 8192, 33, "relu2", True)):
        assert wf._lib.lib().wf_decode_fuses_quant(m, k, n * k, 1) == few
        gate = torch.randn(m, k, generator=g).bfloat16().to(dev)
        up = torch.randn(m, k, generator=g).bfloat16().to(dev)
        codes, sc = wf.pack_ternary((torch.randn(n, k, generator=g) * 0.02).to(dev))
        act = torch.empty_like(gate)
        ops.act_mul(gate, up, act, mode)
        y_ref, acc_ref = wf.bitlinear(act, codes, sc, out_dtype=torch.float32, want_acc=True, path="decode")
        grp = ops.DecodeGroup([dict(x=gate, x2=up, x_mode=mode, codes=codes, w_scale=sc, out_dtype=torch.float32, want_acc=True)])
        y = grp.run()[0]
        assert torch.equal(grp.accs[0], acc_ref) and torch.equal(y, y_ref), (m, k, n, mode)
    wf.device_status()


@pytest.mark.parametrize("m,k,ns", [(1, 576, (64, 64)), (2, 2560, (640, 200, 640)), (1, 576, (6912, 6000)), (3, 576, (6912, 6000)), (5, 2560, (6912, 6016)),
                                    (2, 256, (40000, 40000)), (1, 192, (64000, 64000)), (2, 256, (40000, 30000)), (3, 256, (17000,) * 5), (9, 640, (512, 512))])
def test_every_residual_output_of_a_group_is_written(wf, m, k, ns):
    """Problems of one group with a residual output of their own: the launch for one or two tokens, the forms where warps share
    an item or take whole ones, the streaming form with equal and with unequal problems.  The sum of two bf16 tensors rounded once:
    exact."""
    from wrinklefree_monorepo_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(m * 7 + k)
    h, d = (torch.randn(m, k, generator=g, device="cuda").bfloat16() for _ in range(2))
    w = torch.ones(k, device="cuda").bfloat16()
    codes = [torch.randint(0, 3, (n, k // 4), generator=g, device="cuda", dtype=torch.uint8) for n in ns]
    for which in (range(len(ns)), (0,), (len(ns) - 1,), (0, len(ns) - 1)):
        outs = {i: torch.zeros_like(h) for i in which}
        grp = ops.DecodeGroup([dict(x=h, x2=d, x_mode="norm", norm_w=w, codes=c, w_scale=0.01, h_out=outs.get(i)) for i, c in enumerate(codes)])
        for kw in (dict(), dict(pdl=True), dict(pdl=True, x_ready=True)):
            for o in outs.values():
                o.zero_()
            grp.run(**kw)
            assert all(torch.equal(o, h + d) for o in outs.values()), (list(which), kw)
    wf.device_status()


@pytest.mark.parametrize("B", [1, 2, 3])
def test_fused_decode_step_equals_unfused(wf, B):
    """The six-launch decode step (fused inputs) against the ten-launch step of the same model; one and two sequences of a narrow
    model take it by default, on the launch for so few tokens."""
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    cfg = DecoderConfig(layers=3, hidden=256, n_q=4, n_kv=2, head_dim=64, intermediate=512, vocab=1000)
    dev = torch.device("cuda", 0)
    S, T = 7, 16
    assert TernaryDecoder(cfg, B, T, dev, seed=2).fused == (B <= 2)
    ids = torch.randint(0, cfg.vocab, (B, S), generator=torch.Generator().manual_seed(6)).to(dev)
    outs = []
    for fuse in (True, False):
        m = TernaryDecoder(cfg, B, T, dev, seed=2, fuse=fuse)
        assert m.fused == fuse
        m.capture(masked=True)
        steps = []
        for t in range(S):
            m.tok.copy_(ids[:, t])
            m.graph.replay()
            steps.append(m.logits.float().clone())
        outs.append(torch.stack(steps))
    err = float((outs[0] - outs[1]).abs().max() / outs[1].abs().max())
    assert err <= 2e-2, err
    assert (outs[0].argmax(-1) == outs[1].argmax(-1)).float().mean() >= 0.9
    wf.device_status()


@pytest.mark.parametrize("B,hidden,n_q,n_kv,d,mlp,fused", [(1, 576, 9, 3, 64, 16384, True), (1, 2560, 20, 5, 128, 9600, True), (1, 2560, 20, 5, 128, 11008, False),
                                                           (1, 2048, 16, 4, 128, 14336, False), (1, 4096, 32, 8, 128, 4096, False), (2, 1024, 16, 4, 64, 4096, True),
                                                           (2, 1024, 16, 4, 64, 8192, False), (2, 576, 9, 3, 64, 9600, False), (3, 576, 9, 3, 64, 1536, False)])
def test_default_step_is_fused_only_where_its_launches_take_it(wf, B, hidden, n_q, n_kv, d, mlp, fused):
    """The rule on widths alone chose the fused step for MLPs whose launches then ran, with the norm or the activation in every
    block, on the kernel for stacks (up to a third slower per layer)."""
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    cfg = DecoderConfig(layers=1, hidden=hidden, n_q=n_q, n_kv=n_kv, head_dim=d, intermediate=mlp, vocab=100)
    assert TernaryDecoder(cfg, B, 8, torch.device("cuda", 0)).fused == fused


def test_prefetch_that_was_asked_for_is_used(wf):
    """A model whose default is the fused step, which has no prefetch: asking for one selects the separate launches, and their
    descriptors carry the ranges."""
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    cfg = DecoderConfig(layers=2, hidden=576, n_q=9, n_kv=3, head_dim=64, intermediate=1536, vocab=500)
    dev = torch.device("cuda", 0)
    assert TernaryDecoder(cfg, 1, 8, dev, seed=2).fused
    m = TernaryDecoder(cfg, 1, 8, dev, seed=2, prefetch=True)
    assert not m.fused
    got = [p.prefetch_bytes for p in m.layers[0]["g_qkv"]._host] + [p.prefetch_bytes for p in m.layers[0]["g_gu"]._host]
    want = [m.layers[0][n][0].numel() for n in ("o", "gate", "up", "down")] + [m.layers[1]["q"][0].numel()]
    assert got == want


@pytest.mark.parametrize("m,n,k", [(1, 1000, 576), (3, 130, 72), (32, 5000, 4096), (256, 3000, 4096), (300, 1100, 1024), (17, 128, 8)])
@pytest.mark.parametrize("out_dtype", [torch.bfloat16, torch.float32])
def test_linear_bf16_output_head(wf, m, n, k, out_dtype):
    """The bf16 linear kernel (the decoder's output head) against an fp32 matmul of the same bf16 operands: the products
    are exact in fp32, only the order of the fp32 additions differs (tolerance 1e-3 of the largest output for f32, one
    bf16 rounding step more for bf16 outputs); row tails, token tails, K tails, more than 256 tokens."""
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(m * 1000 + n + k)
    x = torch.randn(m, k, generator=g, device=dev).bfloat16()
    w = (torch.randn(n, k, generator=g, device=dev) * 0.05).bfloat16()
    ref = x.float() @ w.float().t()
    y = wf.linear_bf16(x, w, out_dtype=out_dtype)
    assert y.shape == (m, n) and y.dtype == out_dtype
    tol = 1e-3 if out_dtype == torch.float32 else 1e-2
    err = float((y.float() - ref).abs().max() / ref.abs().max())
    assert err < tol, err
    # strided views: rows of a wider buffer on both sides, and into a wider output
    if k >= 64:
        xw = torch.zeros(m, k + 16, dtype=torch.bfloat16, device=dev)
        xw[:, :k] = x
        ww = torch.zeros(n, k + 8, dtype=torch.bfloat16, device=dev)
        ww[:, :k] = w
        out = torch.full((m, n + 5), 7.0, dtype=out_dtype, device=dev)
        wf.linear_bf16(xw[:, :k], ww[:, :k], out=out[:, :n])
        assert torch.equal(out[:, :n], y) and bool((out[:, n:] == 7.0).all())
    wf.device_status()


def test_linear_bf16_rejects_what_it_cannot_run(wf):
    dev = torch.device("cuda", 0)
    x = torch.zeros(2, 64, dtype=torch.bfloat16, device=dev)
    w = torch.zeros(8, 64, dtype=torch.bfloat16, device=dev)
    with pytest.raises(ValueError):
        wf.linear_bf16(x.float(), w)
    with pytest.raises(RuntimeError):
        wf.linear_bf16(x[:, :60], w[:, :60])  # K not a multiple of 8


@pytest.mark.parametrize("m,k", [(1, 4096), (5, 576), (3, 14336), (2, 16384), (33, 2048)])
def test_norm_and_activation_with_fused_quantization(wf, m, k):
    """The residual add + RMSNorm and the gate activation that quantize their own result: int8 codes, per-token multipliers,
    the updated residual stream and the optional bf16 copy equal the unfused chain (kernel, then act_quant_i8) bit for bit."""
    from wrinklefree_monorepo_b200 import ops

    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(m * 100 + k)
    h0 = torch.randn(m, k, generator=g, device=dev).bfloat16()
    delta = torch.randn(m, k, generator=g, device=dev).bfloat16()
    w = (torch.rand(k, generator=g, device=dev) + 0.5).bfloat16()
    for d in (delta, None):
        h_ref, y_ref = h0.clone(), torch.empty_like(h0)
        ops.add_rmsnorm_(h_ref, d, w, y_ref, 1e-5)
        q_ref, s_ref = wf.act_quant_i8(y_ref, eps=1e-5)
        h_f, y_f = h0.clone(), torch.empty_like(h0)
        q = torch.empty(m, k, dtype=torch.int8, device=dev)
        s = torch.empty(m, dtype=torch.float32, device=dev)
        ops.add_rmsnorm_quant_(h_f, d, w, q, s, 1e-5, out=y_f)
        assert torch.equal(h_f, h_ref) and torch.equal(y_f, y_ref) and torch.equal(q, q_ref) and torch.equal(s, s_ref)
        q2, s2 = torch.empty_like(q), torch.empty_like(s)
        ops.add_rmsnorm_quant_(h0.clone(), d, w, q2, s2, 1e-5)  # without the bf16 copy
        assert torch.equal(q2, q_ref) and torch.equal(s2, s_ref)
    up = torch.randn(m, k, generator=g, device=dev).bfloat16()
    for mode in ("silu", "relu2"):
        a_ref = ops.act_mul(h0, up, torch.empty_like(h0), mode)
        q_ref, s_ref = wf.act_quant_i8(a_ref, eps=1e-5)
        q = torch.empty(m, k, dtype=torch.int8, device=dev)
        s = torch.empty(m, dtype=torch.float32, device=dev)
        out = torch.empty_like(h0)
        ops.act_mul_quant(h0, up, q, s, mode, out=out)
        assert torch.equal(out, a_ref) and torch.equal(q, q_ref) and torch.equal(s, s_ref)


@pytest.mark.parametrize("B,hidden,n_q,n_kv,d,mlp,act,S,steps", [
    (1, 64, 1, 1, 64, 64, "silu", 3, 4),        # one row group per CTA, one head
    (3, 256, 4, 2, 64, 512, "relu2", 0, 20),    # from an empty cache, across the edge of a tile
    (1, 576, 9, 3, 64, 1536, "silu", 76, 8),    # across the edge of a round of tiles (80 positions per CTA)
    (7, 576, 9, 3, 64, 1536, "silu", 15, 4),    # every cluster that fits
    (2, 512, 8, 2, 128, 1024, "silu", 250, 4),  # sixteen lanes per position, several rounds
    (12, 320, 4, 4, 64, 192, "silu", 9, 3)])    # clusters of eight
def test_all_layers_in_one_launch(wf, B, hidden, n_q, n_kv, d, mlp, act, S, steps):
    """The step that runs all layers in one launch against the separate launches, teacher-forced: logits within the 3e-2 that int8
    codes on a rounding edge move them (norm and softmax sums run in another order), caches of the first layer likewise, nothing
    written behind the position."""
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    cfg = DecoderConfig(layers=3, hidden=hidden, n_q=n_q, n_kv=n_kv, head_dim=d, intermediate=mlp, vocab=500, act=act)
    dev = torch.device("cuda", 0)
    T = S + steps + 2
    ids = torch.randint(0, cfg.vocab, (B, S + steps), generator=torch.Generator().manual_seed(B + hidden)).to(dev)
    ms = [TernaryDecoder(cfg, B, T, dev, seed=2, fuse=fuse) for fuse in (None, False)]
    assert ms[0].resident is not None and ms[1].resident is None and ms[0].resident.cluster == (8 if B > 8 else 16)
    outs = []
    for m in ms:
        m.capture()
        for L in m.layers:  # the warm-up steps wrote position 0 and later ones
            L["kc"].zero_()
            L["vc"].zero_()
        if S:
            m.prefill(ids[:, :S])
        got = []
        for t in range(S, S + steps):
            m.tok.copy_(ids[:, t])
            m.graph.replay()
            got.append(m.logits.float().clone())
        assert int(m.pos) == S + steps
        assert torch.equal(m.next_tok, m.logits.argmax(-1))
        assert not any(bool(L[c][:, :, S + steps:].any()) for L in m.layers for c in ("kc", "vc"))
        outs.append(torch.stack(got))
    err = float((outs[0] - outs[1]).abs().max() / outs[1].abs().max())
    assert err <= 3e-2, err
    for c in ("kc", "vc"):
        a, b = (m.layers[0][c].float() for m in ms)
        assert float((a - b).abs().max() / b.abs().max()) <= 2e-2, c
    wf.device_status()


@pytest.mark.parametrize("B,V", [(1, 1), (3, 7), (2, 1000), (1, 49152), (5, 40001)])
def test_argmax_of_the_head(wf, B, V):
    """As torch.argmax: ties go to the first, zeros of both signs tie, a NaN is the largest; odd lengths and row strides."""
    from wrinklefree_monorepo_b200 import ops

    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(V)
    rows = torch.randn(B, V + 9, generator=g, device=dev).bfloat16()
    inputs = [rows[:, :V], rows[:, 1:V + 1], rows[:, :V].contiguous(), torch.zeros(B, V, device=dev).bfloat16() * -1, torch.full((B, V), float("-inf"), device=dev).bfloat16()]
    inputs.append(inputs[3].clone())
    inputs[-1][:, V // 2] = 0.0
    for at in (V - 1, V // 3):
        x = inputs[2].clone()
        x[:, at:] = float("nan")
        inputs.append(x)
    for i, x in enumerate(inputs):
        out, pos = torch.full((B,), -1, dtype=torch.long, device=dev), torch.tensor(41, device=dev)
        ops.argmax_(x, out, pos)
        assert torch.equal(out, x.argmax(-1)) and int(pos) == 42, i


@pytest.mark.parametrize("B,S,nq,nkv,D,T,wide", [(1, 1, 1, 1, 64, 1, 0), (2, 63, 9, 3, 64, 70, 0), (1, 64, 4, 1, 128, 64, 64), (3, 65, 6, 2, 64, 200, 384),
                                                 (1, 130, 32, 8, 128, 140, 0), (2, 512, 2, 2, 64, 512, 8)])
def test_prompt_attention_kernel(wf, B, S, nq, nkv, D, T, wide):
    """Causal attention of a prompt over the caches against fp32 softmax attention: max|a-b| / max|b| <= 1e-2 (probabilities are rounded
    to bf16 in front of the second product, the output is bf16); positions behind the prompt hold garbage that must not leak in;
    query rows inside wider rows."""
    from wrinklefree_monorepo_b200 import ops

    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(S * 10 + D)
    q = torch.randn(B * S, nq * D + wide, generator=g, device=dev).bfloat16()[:, :nq * D]
    kc, vc = (torch.randn(B, nkv, T, D, generator=g, device=dev).bfloat16() for _ in range(2))
    kc[:, :, S:] = 1e4
    vc[:, :, S:] = float("nan")
    out = torch.full((B * S, nq * D), 7.0, dtype=torch.bfloat16, device=dev)
    ops.attn_prompt(q, kc, vc, out, S)
    qf = q.float().reshape(B, S, nkv, nq // nkv, D)
    s = torch.einsum("bshgd,bhtd->bhgst", qf, kc[:, :, :S].float()) * D ** -0.5
    s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device=dev).triu(1), float("-inf"))
    ref = torch.einsum("bhgst,bhtd->bshgd", torch.softmax(s, -1), vc[:, :, :S].float()).reshape(B * S, nq * D)
    err = float((out.float() - ref).abs().max() / ref.abs().max())
    assert err <= 1e-2, err


@pytest.mark.parametrize("m,ns,k", [(1, (64, 64, 64), 64), (17, (100, 28, 130), 576), (64, (576, 192), 128), (65, (576, 192, 192), 576), (121, (1536, 1536), 576),
                                    (300, (200, 7), 1536), (1000, (1024, 256, 256), 1024)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_projections_side_by_side(wf, m, ns, k, dtype):
    """Several projections of the same tokens as one contraction with a scale per row: the bits of the separate calls."""
    from wrinklefree_monorepo_b200 import ops

    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(m + k)
    packed = [wf.pack_ternary(torch.randn(n, k, generator=g, device=dev) * 0.02 * (i + 1)) for i, n in enumerate(ns)]
    q, s = ops.act_quant_i8(torch.randn(m, k, generator=g, device=dev).bfloat16(), eps=1e-5)
    want = torch.cat([wf.bitlinear(q, c, w, x_scale=s, out_dtype=dtype) for c, w in packed], 1)
    codes, scales = torch.cat([c for c, _ in packed]), torch.cat([w[:1].expand(c.shape[0]) for c, w in packed])
    out = torch.full((m, sum(ns) + 8), 7.0, dtype=dtype, device=dev)
    ops.bitlinear_rows(q, s, codes, scales, out[:, :sum(ns)], ops.rows_workspace(m, [(sum(ns), k)], dev))
    assert torch.equal(out[:, :sum(ns)], want) and bool((out[:, sum(ns):] == 7.0).all())
    small = torch.empty(wf._lib.lib().wf_prefill_workspace_bytes(m, k), dtype=torch.uint8, device=dev)  # no room for expanded weights
    assert torch.equal(ops.bitlinear_rows(q, s, codes, scales, out[:, :sum(ns)], small), want)
    wf.device_status()


@pytest.mark.parametrize("B,S,hidden,n_q,n_kv,d,mlp,act", [(1, 1, 64, 1, 1, 64, 64, "silu"), (1, 7, 576, 9, 3, 64, 1536, "relu2"), (2, 33, 256, 4, 2, 128, 512, "silu"),
                                                           (1, 121, 576, 9, 3, 64, 1536, "silu"), (3, 20, 2048, 16, 4, 128, 2048, "silu")])
def test_prompt_layers_in_native_code(wf, monkeypatch, B, S, hidden, n_q, n_kv, d, mlp, act):
    """The native loop over the layers of a prompt makes the calls of the operators one by one: same bits, on either side of the token
    counts at which a projection changes its kernel."""
    from wrinklefree_monorepo_b200 import ops
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    def by_operators(layers, h, cos, sin, xbuf, aq, s1, qkv, gu, att, res, ws, b, s, nq, nkv, dim, mode, eps, *limits):
        m, k = h.shape
        xq, delta = xbuf[:m * k].view(m, k), None
        for qkv_c, qkv_s, o_c, o_s, gu_c, gu_s, down_c, down_s, n1, n2, kc, vc in layers:
            ops.add_rmsnorm_quant_(h, delta, n1, xq, s1, eps)
            ops.bitlinear_rows(xq, s1, qkv_c, qkv_s, qkv, ws)
            parts = qkv.split([nq * dim, nkv * dim, nkv * dim], 1)
            ops.rope_kv_prompt_(*parts, cos, sin, kc, vc, s)
            ops.attn_prompt(parts[0], kc, vc, att, s)
            ops.add_rmsnorm_quant_(h, ops.bitlinear(att, o_c, o_s), n2, xq, s1, eps)
            ops.bitlinear_rows(xq, s1, gu_c, gu_s, gu, ws)
            ops.act_mul_quant(gu[:, :gu.shape[1] // 2], gu[:, gu.shape[1] // 2:], aq, s1, mode="silu" if mode == 0 else "relu2")
            delta = res.copy_(ops.bitlinear(aq, down_c, down_s, x_scale=s1, out_dtype=h.dtype))

    cfg = DecoderConfig(layers=2, hidden=hidden, n_q=n_q, n_kv=n_kv, head_dim=d, intermediate=mlp, vocab=300, act=act)
    dev = torch.device("cuda", 0)
    ids = torch.randint(0, cfg.vocab, (B, S), generator=torch.Generator().manual_seed(S)).to(dev)
    m = TernaryDecoder(cfg, B, S + 3, dev, seed=4)
    native = m.prefill(ids, all_logits=True), [L[c].clone() for L in m.layers for c in ("kc", "vc")]
    monkeypatch.setattr(ops.L.host(), "prompt_layers", by_operators)
    assert torch.equal(m.prefill(ids, all_logits=True), native[0])
    assert all(torch.equal(a, b) for a, b in zip([L[c] for L in m.layers for c in ("kc", "vc")], native[1]))
    wf.device_status()
