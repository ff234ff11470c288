"""GPU test (-m gpu) of what the ops, the layers and the cache refuse or leave to their general paths, and of calls whose
results must not depend on the path that serves them."""
import pytest
import torch

from oracle import tables as otab
from tests.helpers import synth_gdn_inputs, synth_mamba_inputs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nat():
    import neuralattentionsearchlinear_b200 as n
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    return n


def op_inputs(rule, B, T, H, K, V, nbs, dtype=torch.bfloat16, seed=0):
    """(positional arguments up to the decays and betas, 0/1 block types with the last one forced, its own types)"""
    if rule == "gdn":
        q, k, v, g, beta, _ = (x.cuda() for x in synth_gdn_inputs(B, T, H, K, V, seed=seed, dtype=dtype))
        args = (q, k, v, q, k, v, None, g, beta)
    else:
        q, k, v, g, _ = (x.cuda() for x in synth_mamba_inputs(B, T, H, K, V, seed=seed, dtype=dtype))
        args = (q, k, v, q, k, v, None, g)
    raw = otab.synth_types(B, -(-T // nbs), H, 0.5, seed=seed, force_last=False)
    return args, otab.force_last_block(raw.clone()).cuda(), raw[:, -1].cuda()


@pytest.mark.parametrize("rule,K,V", [("gdn", 64, 64), ("mamba", 128, 64)])
@pytest.mark.parametrize("T", [100, 128])
@pytest.mark.parametrize("want", [False, True])
def test_chunk_inference_refuses_fp32(nat, rule, K, V, T, want):
    """The fp32 recurrence has no block-start state for a decoder: the op raises, with and without states asked for."""
    args, types, last = op_inputs(rule, 2, T, 2, K, V, 64, dtype=torch.float32)
    op, key = ((nat.nats_mixed_attn_gdn_chunk_inference, "output_final_state_gated_delta") if rule == "gdn" else
               (nat.nats_mixed_attn_mamba_chunk_inference, "output_final_state_mamba"))
    with pytest.raises(TypeError):
        op(*args, types, last, None, nats_block_size=64, ops_for_incomplete_chunks="all", **{key: want})


# ------------------------------------------------------------------------------------------------ layers and their caches
def make_layer(nat, rule="gdn", **kw):
    cls = nat.NeuralAttentionSearchLinearAttnGDN if rule == "gdn" else nat.NeuralAttentionSearchLinearAttnMamba
    args = dict(hidden_size=256, expand_v=1, head_dim=64, num_heads=4, num_attn_heads=4, ops_for_incomplete_chunks="all",
                layer_idx=0, norm_eps=1e-6)
    if rule == "mamba":
        args.update(head_dim=128, expand_v=0.5)
    args.update(kw)
    torch.manual_seed(3)
    return cls(**args).cuda().bfloat16().eval()


def call(layer, x, cache=None):
    if hasattr(layer, "b_proj"):
        return layer(x, past_key_values=cache)[0]
    return layer(x, cache_params=cache)


def tokens(B, T, hidden=256, seed=0):
    return torch.randn(B, T, hidden, generator=torch.Generator().manual_seed(seed)).bfloat16().cuda()


@pytest.mark.parametrize("rule", ["gdn", "mamba"])
def test_token_of_another_width_raises(nat, rule):
    """The first token and every later one: a wrong width raises and leaves the cache as it was."""
    layer, x = make_layer(nat, rule), tokens(2, 72)
    with torch.no_grad():
        cache = nat.NAtSCache()
        call(layer, x[:, :70], cache)
        for t in (70, 71):
            state = cache[0].state.clone()
            for hidden in (128, 320):
                with pytest.raises(RuntimeError):
                    call(layer, tokens(2, 1, hidden), cache)
            assert cache[0].n_tokens == t and torch.equal(cache[0].state, state)
            call(layer, x[:, t:t + 1], cache)
    assert cache[0].n_tokens == 72
