"""GPU test (-m gpu) of the fused layer forward (``natsl_layer_forward``) against the layers' general path (torch modules and
the ops one by one, which tests/test_gpu_layers.py ties to the oracle), and of its selection against torch's hard softmax.

Both paths round the same tensors to bf16 and differ in the order of fp32 sums and in the sigmoid's last two bits, so a
result may be off by the rounding flips of the tensors on its way: 2^-8 of the size of the largest entry for each of about
four roundings that do not cancel."""
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 4 * 2.0 ** -8


def _make(rule, hidden, heads, head_dim, expand_v, attn_heads, **kw):
    import neuralattentionsearchlinear_b200 as nat
    cls = nat.NeuralAttentionSearchLinearAttnGDN if rule == "gdn" else nat.NeuralAttentionSearchLinearAttnMamba
    args = dict(hidden_size=hidden, head_dim=head_dim, num_heads=heads, expand_v=expand_v, num_attn_heads=attn_heads,
                ops_for_incomplete_chunks="all", layer_idx=0, norm_eps=1e-6)
    args.update(kw)
    return cls(**args)


CASES = [
    ("gdn", dict(hidden=256, heads=4, head_dim=64, expand_v=1, attn_heads=4), 2, 64),
    ("gdn", dict(hidden=256, heads=2, head_dim=128, expand_v=1, attn_heads=2, conv_bias=True, allow_neg_eigval=True), 1, 131),
    ("gdn", dict(hidden=320, heads=3, head_dim=128, expand_v=2, attn_heads=6, nats_block_size=128), 2, 384),
    ("gdn", dict(hidden=256, heads=2, head_dim=192, expand_v=2, attn_heads=6, num_nats_head=2), 1, 193),
    ("gdn", dict(hidden=256, heads=4, head_dim=64, expand_v=2, attn_heads=4, attn_with_short_conv=False, nats_block_size=256), 2, 700),
    ("gdn", dict(hidden=256, heads=4, head_dim=64, expand_v=1, attn_heads=2, attn_qk_norm=False, outputs_are_weighted=False,
                 decay_for_non_gdn_blocks=False, num_nats_head=2), 3, 255),
    ("gdn", dict(hidden=256, heads=2, head_dim=64, expand_v=1, attn_heads=2, attn_qk_norm=False, attn_with_short_conv=False,
                 ops_for_incomplete_chunks="gated_delta_net"), 1, 129),
    ("mamba", dict(hidden=256, heads=2, head_dim=128, expand_v=0.5, attn_heads=2), 2, 65),
    ("mamba", dict(hidden=256, heads=40, head_dim=128, expand_v=0.5, attn_heads=40, nats_block_size=256), 1, 512),
    ("mamba", dict(hidden=256, heads=3, head_dim=128, expand_v=0.5, attn_heads=3, attn_with_short_conv=True), 2, 320),
    ("mamba", dict(hidden=256, heads=4, head_dim=128, expand_v=0.5, attn_heads=4, attn_with_short_conv=True, attn_qk_norm=True,
                   num_nats_head=2, nats_block_size=128), 1, 300),
    ("mamba", dict(hidden=256, heads=4, head_dim=128, expand_v=0.5, attn_heads=4, attn_qk_norm=True), 1, 128),
]


@pytest.mark.parametrize("rule,args,B,T", CASES)
@pytest.mark.parametrize("cached", [False, True])
def test_fused_forward_matches_the_general_path(rule, args, B, T, cached, monkeypatch):
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, natsl_attn_gdn, natsl_attn_mamba2
    if cached and args["head_dim"] == 192:
        pytest.skip("the general path has no chunk-inference op for these head dims")
    torch.manual_seed(T)
    layer = _make(rule, **args).cuda().bfloat16().eval()
    x = torch.randn(B, T, args["hidden"], generator=torch.Generator().manual_seed(B)).bfloat16().cuda()

    def run():
        cache = nat.NAtSCache() if cached else None
        with torch.no_grad():
            y = layer(x, past_key_values=cache)[0] if rule == "gdn" else layer(x, cache_params=cache)
        return y, layer.attn_fraction, (cache[0] if cached else None)

    ref_y, ref_f, ref_c = None, None, None
    y, f, c = run()
    took = []
    for mod in (natsl_attn_gdn, natsl_attn_mamba2):
        monkeypatch.setattr(mod, "layer_forward", lambda *a, **k: took.append(1))
    if args["head_dim"] == 192:                              # general path: the training op without gradients
        layer.train()
    ref_y, ref_f, ref_c = run()
    assert took or layer.training
    pairs = [("output", y, ref_y)]
    assert torch.equal(f, ref_f)
    if cached:
        assert (c.block_types is None) == (ref_c.block_types is None)
        if c.block_types is not None:
            assert torch.equal(c.block_types > 0.5, ref_c.block_types > 0.5)
        assert c.n_tokens == T
        pairs += [(n, getattr(c, n), getattr(ref_c, n)) for n in ("state", "state_block_start", "k_attn", "v_attn", "g_block", "pool_sum")]
        pairs += [("tails", torch.cat(c.conv_state, 1), torch.cat(ref_c.conv_state, 1))]
    for name, got, want in pairs:
        assert got.shape == want.shape, name
        got, want = got.float(), want.float()
        bound = TOL * max(float(want.abs().max()), 1e-3)
        err = float((got - want).abs().max())
        assert err <= bound, f"{name} off by {err:.3g} (bound {bound:.3g})"
    assert _lib.load().natsl_device_status() == 0


def test_selection_equals_torch_hard_softmax_bit_for_bit():
    """Blocks of 64 equal tokens make the pooled input, and one-hot selection weights the logits, any bf16 pair: random
    pairs, exact ties and pairs up to three units in the last place apart at every magnitude."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200.modules import hard_softmax
    B, TN = 64, 256
    gen = torch.Generator().manual_seed(0)
    n = B * TN
    l0 = torch.randn(n, generator=gen).bfloat16() * torch.logspace(-4, 2, n).bfloat16()
    step = torch.randint(-3, 4, (n,), generator=gen).to(torch.int16)
    l1 = (l0.view(torch.int16) + step).view(torch.bfloat16)
    l1[::5] = torch.randn(n, generator=gen).bfloat16()[::5]
    logits = torch.stack([l0, l1], -1).cuda()
    logits = torch.where(logits.isfinite(), logits, torch.zeros_like(logits))
    layer = _make("gdn", hidden=64, heads=1, head_dim=64, expand_v=1, attn_heads=1).cuda().bfloat16().eval()
    layer.nats_layer.weight.data.zero_()
    layer.nats_layer.weight.data[0, 0] = layer.nats_layer.weight.data[1, 1] = 1
    x = torch.zeros(B, TN, 64, 64, device="cuda", dtype=torch.bfloat16)
    x[..., :2] = logits.view(B, TN, 1, 2)
    with torch.no_grad():
        cache = nat.NAtSCache()
        layer(x.view(B, TN * 64, 64), past_key_values=cache)
        want = hard_softmax(logits.view(B, TN, 1, 2))
    assert torch.equal(cache[0].block_types.float(), torch.round(want.float()))


def test_silu_of_the_fused_convolution_rounds_like_the_separate_kernel():
    """Convolutions of one tap pass the projection on, so that the layer's keys are silu(k_raw): against float64 rounded to bf16
    they differ where the sigmoid's last fp32 bits flip a rounding, no more often than the convolution kernel's own
    (2^-24 in front of a rounding to 2^-9: a few in 10^5)."""
    import neuralattentionsearchlinear_b200 as nat
    torch.manual_seed(5)
    layer = _make("gdn", hidden=64, heads=4, head_dim=64, expand_v=1, attn_heads=4, attn_qk_norm=False).cuda().bfloat16().eval()
    for conv in (layer.q_conv1d, layer.k_conv1d, layer.v_conv1d):
        conv.weight.data.zero_()
        conv.weight.data[..., 3] = 1
    x = 40 * torch.randn(4, 4096, 64, generator=torch.Generator().manual_seed(0)).bfloat16().cuda()
    cache = nat.NAtSCache()
    with torch.no_grad():
        layer(x, past_key_values=cache)
        raw = layer.k_proj(x)
        separate = layer.k_conv1d(raw)[0]
        want = torch.nn.functional.silu(raw.double()).bfloat16()
    fused = cache[0].k_attn.reshape(want.shape)
    off = lambda t: int((t != want).sum())
    assert off(fused) <= off(separate) + 2e-6 * want.numel(), (off(fused), off(separate), want.numel())
    extreme = torch.tensor([0.0, -0.0, 88.0, -88.0, -200.0, 300.0, float("inf"), float("nan")])
    x[0, :8] = 0
    layer.k_proj.weight.data.zero_()
    layer.k_proj.weight.data[:, 0] = 1
    x[..., 0] = 0
    x[0, :8, 0] = extreme.to(x)
    with torch.no_grad():
        cache = nat.NAtSCache()
        layer(x, past_key_values=cache)
        want = layer.k_conv1d(layer.k_proj(x))[0][0, :8]
    assert torch.equal(torch.nan_to_num(cache[0].k_attn[0, :8].reshape(8, -1), 7.0), torch.nan_to_num(want, 7.0))
