"""GPU test (-m gpu) of the single-token layer kernel against the general cached path it stands for (torch projections,
``linear_recurrent_step``, masked attention, mixing), which tests/test_gpu_decode.py ties to the one-shot forward.

Both round the same tensors to bf16 (projections, convolutions, norms, branch outputs, mixing weights, result) and differ
only in the order of fp32 sums, so a result may be off by the rounding flips of the tensors on its way: 2^-8 of the size
of the largest entry for each of about four roundings that do not cancel."""
import copy

import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 4 * 2.0 ** -8


def _gdn(hidden, heads, head_dim, expand_v, attn_heads, **kw):
    from neuralattentionsearchlinear_b200 import NeuralAttentionSearchLinearAttnGDN
    args = dict(hidden_size=hidden, expand_v=expand_v, head_dim=head_dim, num_heads=heads, num_attn_heads=attn_heads,
                layer_idx=0, norm_eps=1e-6)
    args.update(kw)
    return NeuralAttentionSearchLinearAttnGDN(**args)


def _mamba(hidden, heads, head_dim, expand_v, attn_heads, **kw):
    from neuralattentionsearchlinear_b200 import NeuralAttentionSearchLinearAttnMamba
    args = dict(hidden_size=hidden, expand_v=expand_v, head_dim=head_dim, num_heads=heads, num_attn_heads=attn_heads,
                ops_for_incomplete_chunks="all", layer_idx=0, norm_eps=1e-6)
    args.update(kw)
    return NeuralAttentionSearchLinearAttnMamba(**args)


CASES = [
    # make, layer arguments, batch, prompt: around block ends, every batch grouping of the products, all head-dim pairs
    (_gdn, dict(hidden=256, heads=4, head_dim=64, expand_v=1, attn_heads=4), 1, 62),
    (_gdn, dict(hidden=256, heads=4, head_dim=64, expand_v=1, attn_heads=4, allow_neg_eigval=True), 9, 127),
    (_gdn, dict(hidden=320, heads=3, head_dim=128, expand_v=2, attn_heads=6, num_nats_head=3), 2, 700),
    (_gdn, dict(hidden=256, heads=2, head_dim=128, expand_v=1, attn_heads=2, conv_bias=True,
                ops_for_incomplete_chunks="gated_delta_net"), 17, 190),
    (_gdn, dict(hidden=256, heads=2, head_dim=128, expand_v=1, attn_heads=4, attn_qk_norm=False, outputs_are_weighted=False,
                decay_for_non_gdn_blocks=False), 33, 64),
    (_gdn, dict(hidden=256, heads=2, head_dim=256, expand_v=0.5, attn_heads=4, attn_with_short_conv=False), 64, 0),
    (_mamba, dict(hidden=256, heads=2, head_dim=128, expand_v=0.5, attn_heads=2, nats_block_size=128), 3, 380),
    (_mamba, dict(hidden=256, heads=4, head_dim=64, expand_v=1, attn_heads=4, attn_qk_norm=True, attn_with_short_conv=True), 1, 126),
    (_mamba, dict(hidden=256, heads=4, head_dim=64, expand_v=1, attn_heads=2, num_nats_head=2,
                  ops_for_incomplete_chunks="mamba", nats_block_size=256), 5, 255),
]


@pytest.mark.parametrize("make,args,B,T0", CASES)
def test_token_kernel_matches_the_general_path(make, args, B, T0):
    from neuralattentionsearchlinear_b200 import NAtSCache
    from neuralattentionsearchlinear_b200.decode_step import decode_token
    from neuralattentionsearchlinear_b200.decoding import forward_cached
    torch.manual_seed(T0 + B)
    layer = make(**args).cuda().bfloat16().eval()
    n_new = 70 if B <= 3 else 6
    gen = torch.Generator().manual_seed(B)
    x = torch.randn(B, T0 + n_new, args["hidden"], generator=gen).bfloat16().cuda()

    def general(piece, cache):
        return layer.mix(piece, *forward_cached(layer, piece, cache))

    with torch.no_grad():
        cache = NAtSCache()
        t = 0
        while t < T0:                                        # a prompt of 64 tokens or more at once, a shorter one in pieces
            n = T0 if T0 >= 64 else min(31, T0 - t)
            general(x[:, t:t + n], cache)
            t += n
        ref_cache = NAtSCache()
        ref_cache.layers = [copy.copy(c) for c in cache.layers]
        for i in range(n_new):
            tok = x[:, T0 + i:T0 + i + 1]
            y = decode_token(layer, tok, cache)
            assert y is not None, "the token kernel does not take this configuration"
            ref = general(tok, ref_cache)
            for name, got, want in (("output", y, ref), ("state", cache[0].state, ref_cache[0].state),
                                    ("block-start state", cache[0].state_block_start, ref_cache[0].state_block_start),
                                    ("keys", cache[0].k_attn, ref_cache[0].k_attn), ("values", cache[0].v_attn, ref_cache[0].v_attn),
                                    ("tails", torch.cat(cache[0].conv_state, 1), torch.cat(ref_cache[0].conv_state, 1)),
                                    ("decay", cache[0].g_block, ref_cache[0].g_block), ("pool", cache[0].pool_sum, ref_cache[0].pool_sum)):
                got, want = got.float(), want.float()
                bound = TOL * max(float(want.abs().max()), 1e-3)
                err = float((got - want).abs().max())
                assert err <= bound, f"token {i} (position {T0 + i}): {name} off by {err:.3g} (bound {bound:.3g})"
        assert cache[0].n_tokens == ref_cache[0].n_tokens == T0 + n_new


@pytest.mark.parametrize("make,args,B,T0", [
    (_gdn, dict(hidden=256, heads=4, head_dim=64, expand_v=1, attn_heads=4), 1, 8200),
    (_mamba, dict(hidden=256, heads=4, head_dim=128, expand_v=0.5, attn_heads=4, nats_block_size=256), 2, 1270),
    (_gdn, dict(hidden=256, heads=2, head_dim=128, expand_v=1, attn_heads=2), 3, 2090),
    (_gdn, dict(hidden=256, heads=16, head_dim=64, expand_v=1, attn_heads=16), 3, 3300),
    (_mamba, dict(hidden=256, heads=4, head_dim=128, expand_v=0.5, attn_heads=4, nats_block_size=128), 1, 4160),
    (_gdn, dict(hidden=256, heads=2, head_dim=128, expand_v=1, attn_heads=2), 1, 8230),
])
def test_token_kernel_over_many_units(make, args, B, T0):
    """Splits that take every S-th selected unit and unit of the current block (up to 32 units, and up to 64 over many splits),
    and ranges of units (beyond); the tokens cross the lines, and the end of a block of several units."""
    test_token_kernel_matches_the_general_path(make, args, B, T0)


@pytest.mark.parametrize("make,args,B,T0", [
    (_gdn, dict(hidden=256, heads=16, head_dim=128, expand_v=1, attn_heads=16), 17, 40),
    (_gdn, dict(hidden=256, heads=16, head_dim=128, expand_v=1, attn_heads=16), 17, 1500),
    (_gdn, dict(hidden=256, heads=16, head_dim=64, expand_v=1, attn_heads=16), 17, 700),
    (_mamba, dict(hidden=256, heads=16, head_dim=128, expand_v=0.5, attn_heads=16, nats_block_size=256), 17, 200),
])
def test_token_kernel_with_one_ring_slot(make, args, B, T0):
    """Grids of more CTAs than fit the SMs and few steps per split: none, one and several steps through a ring of one slot."""
    test_token_kernel_matches_the_general_path(make, args, B, T0)


def test_copied_cache_continues_on_its_own():
    from neuralattentionsearchlinear_b200 import NAtSCache
    torch.manual_seed(1)
    layer = _gdn(hidden=256, heads=4, head_dim=64, expand_v=1, attn_heads=4).cuda().bfloat16().eval()
    x = torch.randn(2, 200, 256, device="cuda").bfloat16()
    with torch.no_grad():
        cache = NAtSCache()
        layer(x[:, :150], past_key_values=cache)
        layer(x[:, 150:151], past_key_values=cache)
        fork = NAtSCache()
        fork.layers = [copy.copy(c) for c in cache.layers]
        first = [layer(x[:, t:t + 1], past_key_values=cache)[0] for t in range(151, 160)]
        layer(x[:, 170:171], past_key_values=cache)
        again = [layer(x[:, t:t + 1], past_key_values=fork)[0] for t in range(151, 160)]
    for a, b in zip(first, again):
        assert torch.equal(a, b)


@pytest.mark.parametrize("B,head_dim", [(1, 64), (2, 128)])
def test_infinite_keys_weigh_nothing(B, head_dim):
    """Keys that give every cached token a score of -inf: the new token alone counts, as in the general path."""
    from neuralattentionsearchlinear_b200 import NAtSCache
    from neuralattentionsearchlinear_b200.decode_step import decode_token
    from neuralattentionsearchlinear_b200.decoding import forward_cached
    torch.manual_seed(2)
    layer = _gdn(hidden=256, heads=2, head_dim=head_dim, expand_v=1, attn_heads=2).cuda().bfloat16().eval()
    x = torch.randn(B, 200, 256, device="cuda").bfloat16()
    with torch.no_grad():
        cache = NAtSCache()
        layer(x[:, :199], past_key_values=cache)
        c = cache[0]
        q = layer.project_qkv(x[:, 199:], conv_state=c.conv_state, want_conv_state=True)["q_attn"]
        keys = torch.zeros_like(c.k_attn)
        keys[..., 5] = torch.where(q[..., 5] > 0, -float("inf"), float("inf")).to(keys.dtype)
        c.k_attn = keys
        other = NAtSCache()
        other.layers = [copy.copy(c)]
        y = decode_token(layer, x[:, 199:], cache)
        want = layer.mix(x[:, 199:], *forward_cached(layer, x[:, 199:], other))
    assert bool(want.isfinite().all())
    assert float((y.float() - want.float()).abs().max()) <= TOL * float(want.float().abs().max())


@pytest.mark.parametrize("where", ["keys", "all keys", "values", "token"])
def test_nan_reaches_the_output(where):
    """A NaN that a token sees is in its output, as in the general path."""
    from neuralattentionsearchlinear_b200 import NAtSCache
    from neuralattentionsearchlinear_b200.decode_step import decode_token
    torch.manual_seed(2)
    layer = _gdn(hidden=256, heads=2, head_dim=64, expand_v=1, attn_heads=2).cuda().bfloat16().eval()
    x = torch.randn(1, 200, 256, device="cuda").bfloat16()
    with torch.no_grad():
        cache = NAtSCache()
        layer(x[:, :199], past_key_values=cache)
        c = cache[0]
        k, v, tok = c.k_attn.clone(), c.v_attn.clone(), x[:, 199:].clone()
        if where == "keys":
            k[:, 194, :, 3] = float("nan")
        elif where == "all keys":
            k.fill_(float("nan"))
        elif where == "values":
            v[:, 194] = float("nan")
        else:
            tok[0, 0, 7] = float("nan")
        c.k_attn, c.v_attn = k, v
        assert bool(decode_token(layer, tok, cache).isnan().all())
