"""The decoder's prompt pass and the launch for all layers of a step: scores that overflow, projections over several ring stages, long
contexts, rows side by side, and which form of a step or prompt runs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [64, 128])
def test_prompt_attention_behind_scores_that_overflow(wf, D):
    """A tile of keys whose scores are all -inf in fp32 counts for nothing once a later score is finite, as in softmax; the queries that
    see nothing else are NaN, as there.  The 1e-2 of the test above."""
    from wrinklefree_monorepo_b200 import ops

    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(D)
    S = 150
    q, kc, vc = (torch.randn(*shape, generator=g, device=dev).bfloat16() for shape in ((S, D), (1, 1, S, D), (1, 1, S, D)))
    q[:, 0], kc[:, :, :, 0] = 1e20, 0.0
    kc[:, :, :70, 0] = -1e30
    out = ops.attn_prompt(q, kc, vc, torch.zeros_like(q), S)
    s = (q.float() @ kc[0, 0].float().t() * D ** -0.5).masked_fill(torch.ones(S, S, dtype=torch.bool, device=dev).triu(1), float("-inf"))
    ref = torch.softmax(s, -1) @ vc[0, 0].float()
    assert bool(ref[:70].isnan().all()) and bool(ref[70:].isfinite().all())
    assert bool(out[:70].isnan().all())
    assert float((out[70:].float() - ref[70:]).abs().max() / ref[70:].abs().max()) <= 1e-2


def test_layer_launch_with_a_split_of_infinite_scores(wf):
    """Two CTAs share a head's positions, and all scores of one of them are -inf: its part counts for nothing, as in the framework's
    attention over the same cache.  The 3e-2 of the comparison with the separate launches."""
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    cfg = DecoderConfig(layers=1, hidden=256, n_q=2, n_kv=2, head_dim=64, intermediate=512, vocab=300)
    dev = torch.device("cuda", 0)
    ms = [TernaryDecoder(cfg, 1, 300, dev, seed=3, fuse=fuse) for fuse in (None, False)]
    assert ms[0].resident is not None
    ms[1].attention = "library"
    g = torch.Generator(device=dev).manual_seed(1)
    caches = [torch.randn(1, 2, 300, 64, generator=g, device=dev).bfloat16() for _ in range(2)]
    logits = []
    ms[1].pos.fill_(270)
    ms[1]._decode_step()
    q = ms[1].layers[0]["qkv"][0].view(2, 64)  # rotated in place
    for head in range(2):
        e = int(q[head].float().abs().argmax())
        for tile in range(1, 17, 2):  # seventeen tiles of 16 positions: the second CTA takes the odd ones
            caches[0][0, head, tile * 16:tile * 16 + 16, e] = -torch.sign(q[head, e]) * float("inf")
    for m in ms:
        for c, given in zip(("kc", "vc"), caches):
            m.layers[0][c].copy_(given)
        m.pos.fill_(270)
        m._decode_step()
        logits.append(m.logits.float())
    assert bool(logits[1].isfinite().all())
    assert float((logits[0] - logits[1]).abs().max() / logits[1].abs().max()) <= 3e-2
    wf.device_status()


@pytest.mark.parametrize("m,i", [(1, 8), (5, 192), (130, 6912)])
@pytest.mark.parametrize("mode", ["silu", "relu2"])
def test_gate_activation_of_rows_side_by_side(wf, m, i, mode):
    """gate and up as the halves of one contraction's rows, the activation as bf16 beside its codes: the bits of the plain activation of
    contiguous copies, as a prompt with sub-layer norms takes it."""
    from wrinklefree_monorepo_b200 import ops

    dev = torch.device("cuda", 0)
    rows = torch.randn(m, 2 * i, generator=torch.Generator(device=dev).manual_seed(i), device=dev).bfloat16()
    g, u = rows.split([i, i], 1)
    out, q, s = torch.empty(m, i, dtype=torch.bfloat16, device=dev), torch.empty(m, i, dtype=torch.int8, device=dev), torch.empty(m, device=dev)
    ops.act_mul_quant(g, u, q, s, mode=mode, out=out)
    want = ops.act_mul(g.contiguous(), u.contiguous(), torch.empty_like(out), mode)
    assert torch.equal(out, want)
    wq, ws = ops.act_quant_i8(want, eps=1e-5)
    assert torch.equal(q, wq) and torch.equal(s, ws.view(-1))


# ring stages of q/k/v, o, gate/up, down with the rows of a stage, by st_plan in csrc/wf_step.cu
@pytest.mark.parametrize("B,hidden,n_q,n_kv,d,mlp,cluster", [
    (2, 960, 15, 5, 64, 2560, 16),     # 1 x 100, 1 x 60, 54 + 54 + 52, 2 x 30
    (4, 1024, 16, 4, 64, 4096, 16),    # 1 x 96, 1 x 64, 4 x 64, 2 x 32
    (2, 1280, 10, 5, 64, 3456, 16),    # 1 x 80, 1 x 80, 4 x 44 + 40, 27 + 27 + 26: an odd number of rows
    (3, 1024, 8, 2, 128, 2816, 16),    # stages of 16 KB: 2 x 48, 1 x 64, 5 x 30 + 26, 22 + 22 + 20
    (1, 2560, 20, 5, 128, 6912, 16),   # 16 KB: 10 x 24, 6 x 23 + 22, 36 x 12, 17 x 9 + 7
    (9, 960, 15, 5, 64, 2560, 8)])     # q, k and v cut across stages: 2 x 100, 1 x 120, 5 x 64, 3 x 40
def test_layers_over_several_ring_stages(wf, monkeypatch, B, hidden, n_q, n_kv, d, mlp, cluster):
    """Projections of several ring stages against the separate launches, bit for bit: at position 0 a head has one weight, 1, and what is
    left are whole-number products and the same roundings (the squares of a norm are added in another order, which moves no bit of
    these inputs).  One width that the default leaves to the separate launches."""
    from wrinklefree_monorepo_b200 import ops
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    cfg = DecoderConfig(layers=1, hidden=hidden, n_q=n_q, n_kv=n_kv, head_dim=d, intermediate=mlp, vocab=500)
    dev = torch.device("cuda", 0)
    if hidden > 2048:
        monkeypatch.setattr(ops.L.lib(), "wf_decode_layers_cluster", lambda *shape: cluster)
    ms = [TernaryDecoder(cfg, B, 4, dev, seed=2, fuse=fuse) for fuse in (None, False)]
    assert ms[0].resident is not None and ms[1].resident is None and ms[0].resident.cluster == cluster
    for step in range(6):
        for m in ms:
            m.tok.copy_(torch.arange(B, device=dev) * 7 + step)
            m.pos.fill_(0)
            m._decode_step()
        assert torch.equal(ms[0].xf, ms[1].xf), step
        for c in ("kc", "vc"):
            assert torch.equal(ms[0].layers[0][c], ms[1].layers[0][c]), (step, c)
    wf.device_status()


@pytest.mark.parametrize("B,hidden,n_q,n_kv,d,mlp,S", [(2, 256, 4, 2, 64, 512, 3001), (1, 512, 8, 2, 128, 1024, 2500)])
def test_all_layers_in_one_launch_at_long_contexts(wf, B, hidden, n_q, n_kv, d, mlp, S):
    """As test_all_layers_in_one_launch, with the same bounds, where eight CTAs share a KV head through many rounds of tiles.  Then one step
    at a position behind the cache's end, which both steps take modulo its length."""
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    steps, T = 3, S + 6
    cfg = DecoderConfig(layers=2, hidden=hidden, n_q=n_q, n_kv=n_kv, head_dim=d, intermediate=mlp, vocab=500)
    dev = torch.device("cuda", 0)
    ids = torch.randint(0, cfg.vocab, (B, S + steps), generator=torch.Generator().manual_seed(S)).to(dev)
    ms = [TernaryDecoder(cfg, B, T, dev, seed=2, fuse=fuse) for fuse in (None, False)]
    assert ms[0].resident is not None and ms[1].resident is None
    outs = []
    for m in ms:
        m.prefill(ids[:, :S])
        got = []
        for t in range(S, S + steps + 1):
            m.tok.copy_(ids[:, t % S])
            m.pos.fill_(t if t < S + steps else T + 2)
            m._decode_step()
            got.append(m.logits.float().clone())
        assert int(m.pos) == T + 3
        assert not any(bool(L[c][:, :, S + steps:].any()) for L in m.layers for c in ("kc", "vc"))
        outs.append(torch.stack(got))
    err = float((outs[0] - outs[1]).abs().max() / outs[1].abs().max())
    assert err <= 3e-2, err
    for c in ("kc", "vc"):
        a, b = (m.layers[0][c].float() for m in ms)
        assert float((a - b).abs().max() / b.abs().max()) <= 2e-2, c
    wf.device_status()


@pytest.mark.parametrize("B,hidden,n_q,n_kv,d,mlp,options,resident,fused", [
    (1, 256, 4, 2, 64, 512, {}, True, True), (1, 256, 4, 2, 64, 512, dict(fuse=True), False, True), (2, 256, 4, 2, 64, 512, dict(fuse=False), False, False),
    (1, 256, 4, 2, 64, 512, dict(prefetch=True), False, False), (1, 256, 4, 2, 64, 512, dict(dtype=torch.float32), False, False),
    (1, 2560, 20, 5, 128, 6912, {}, False, True), (1, 4096, 32, 8, 128, 14336, {}, False, False)])
def test_which_step_a_decoder_runs(wf, B, hidden, n_q, n_kv, d, mlp, options, resident, fused):
    """All layers in one launch where nothing else is asked for and the width is small; what it replaces stays as it was chosen."""
    from wrinklefree_monorepo_b200.decoder import DecoderConfig, TernaryDecoder

    cfg = DecoderConfig(layers=1, hidden=hidden, n_q=n_q, n_kv=n_kv, head_dim=d, intermediate=mlp, vocab=64)
    m = TernaryDecoder(cfg, B, 8, torch.device("cuda", 0), **options)
    assert ((m.resident is not None), m.fused) == (resident, fused)


@pytest.mark.parametrize("hidden,n_q,n_kv,d,mlp,subln", [(576, 9, 3, 64, 1536, False), (512, 4, 2, 128, 1024, False), (512, 4, 2, 128, 1024, True)])
def test_prompts_with_the_frameworks_attention(wf, monkeypatch, hidden, n_q, n_kv, d, mlp, subln):
    """The same prompt with attention on this library's kernel and on the framework's, which takes q as a slice of the joint rows.  Keys and
    values of the first layer are the same bits, the logits within the 3e-2 of the comparisons of two attentions above."""
    from wrinklefree_monorepo_b200 import decoder

    cfg = decoder.DecoderConfig(layers=2, hidden=hidden, n_q=n_q, n_kv=n_kv, head_dim=d, intermediate=mlp, vocab=500, subln=subln)
    dev = torch.device("cuda", 0)
    ids = torch.randint(0, cfg.vocab, (2, 150), generator=torch.Generator().manual_seed(d)).to(dev)
    m = decoder.TernaryDecoder(cfg, 2, 160, dev, seed=4)
    own = m.prefill(ids, all_logits=True).float()
    first = [m.layers[0][c].clone() for c in ("kc", "vc")]
    for L in m.layers:
        L["kc"].zero_(), L["vc"].zero_()
    monkeypatch.setattr(decoder, "PROMPT_KERNEL_MAX", 0)
    other = m.prefill(ids, all_logits=True).float()
    assert all(torch.equal(a, m.layers[0][c]) for a, c in zip(first, ("kc", "vc")))
    assert float((own - other).abs().max() / other.abs().max()) <= 3e-2
