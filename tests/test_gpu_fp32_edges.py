"""GPU test (-m gpu) of the fp32 kernels at the edges of their tiles (groups of 32 or 16 tokens, 16 value columns; 16
queries x 64 keys) against the CPU oracle in float64.  Sums of at most a few hundred fp32 products: 1e-4 as in the parity
tests of the op."""
import pytest
import torch

from oracle import attn as oattn
from oracle import gdn as ogdn
from oracle import tables as otab
from tests.helpers import assert_close, synth_gdn_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,K,V,nbs", [(1, 64, 64, 64), (31, 32, 32, 64), (33, 96, 48, 64), (64, 128, 64, 64), (65, 192, 16, 64),
                                       (161, 256, 64, 128), (130, 64, 128, 128)])
def test_token_recurrence(T, K, V, nbs):
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    B, H = 2, 3
    q, k, v, g, beta, h0 = synth_gdn_inputs(B, T, H, K, V, seed=T + K, dtype=torch.float32)
    types = otab.synth_types(B, -(-T // nbs), H, 0.5, seed=T)
    cu = lambda x: x.cuda()
    tb = nat.build_selection_tables(cu(types), T, nbs)
    for rule in ("gdn", "mamba"):
        gdn = rule == "gdn"
        scale = K ** -0.5 if gdn else 1.0
        o, ht, _ = _ops.linear_recurrent(_lib.RULE_GDN if gdn else _lib.RULE_MAMBA, cu(q), cu(k), cu(v), cu(g), cu(beta) if gdn else None,
                                         tb, scale, cu(h0), True, gdn)
        ref, s = ogdn.linear_recurrent(q.double(), k.double(), v.double(), g.double(), beta.double() if gdn else None, types[..., 1],
                                       nbs=nbs, scale=scale, h0=h0.double(), decay=True, use_l2norm=gdn, rule=rule)
        assert_close(o, ref.float(), 1e-4, f"o {rule}")
        assert_close(ht, s.float(), 1e-4, f"state {rule}")


@pytest.mark.parametrize("T,D,nbs", [(1, 64, 64), (17, 32, 64), (65, 64, 64), (200, 128, 128)])
def test_fp32_attention(T, D, nbs):
    import neuralattentionsearchlinear_b200 as nat
    B, H = 2, 2
    q, k, v, g, beta, _ = synth_gdn_inputs(B, T, H, D, D, seed=T + D, dtype=torch.float32)
    types = otab.synth_types(B, -(-T // nbs), H, 0.5, seed=T)
    cu = lambda x: x.cuda()
    _, o, _ = nat.nats_mixed_attn_gdn(cu(q), cu(k), cu(v), cu(q), cu(k), cu(v), None, cu(g), cu(beta), cu(types), None,
                                      nats_block_size=nbs, ops_for_incomplete_chunks="all", decay_for_non_gdn_blocks=True)
    ref, _ = oattn.attn_sdpa(q.double(), k.double(), v.double(), oattn.attn_mask(types[..., 0], T, nbs, H))
    assert_close(o, ref.float(), 1e-4, "o")


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("where", ["v", "k"])
def test_non_finite_values_behind_the_mask(D, value, where):
    """A token that a query does not see changes nothing for it, whatever its key and value hold; it sees its own."""
    import neuralattentionsearchlinear_b200 as nat
    B, H, T, bad = 1, 2, 150, 101
    q, k, v, g, beta, _ = (x.cuda() for x in synth_gdn_inputs(B, T, H, D, D, seed=D, dtype=torch.float32))
    types = otab.synth_types(B, 3, H, 0.5, seed=1).cuda()
    k2, v2 = k.clone(), v.clone()
    (v2 if where == "v" else k2)[:, bad, :, 3] = value
    run = lambda kk, vv: nat.nats_mixed_attn_gdn(q, kk, vv, q, k, v, None, g, beta, types, None, nats_block_size=64,
                                                 ops_for_incomplete_chunks="all", decay_for_non_gdn_blocks=True)[1]
    clean, got = run(k, v), run(k2, v2)
    assert torch.equal(got[:, :bad], clean[:, :bad])
    if where == "v":
        assert not bool(got[:, bad, :, 3].isfinite().any()) and torch.equal(got[:, bad, :, 4:], clean[:, bad, :, 4:])
    sees = types[:, 1, :, 0] == 1                            # heads whose later queries see the token's block
    assert torch.equal(got[:, 128:][:, :, ~sees[0]], clean[:, 128:][:, :, ~sees[0]])


@pytest.mark.parametrize("rule", ["gdn", "mamba"])
def test_fp32_linear_branch_beside_a_bf16_softmax_branch(rule):
    """Each branch takes its own dtype: outputs in it, equal to those of the branch on its own; the other mix raises."""
    import neuralattentionsearchlinear_b200 as nat
    from tests.helpers import synth_mamba_inputs
    B, T, H, D = 2, 130, 2, 64
    if rule == "gdn":
        q, k, v, g, beta, _ = (x.cuda() for x in synth_gdn_inputs(B, T, H, D, D, seed=3, dtype=torch.float32))
        op, rest = nat.nats_mixed_attn_gdn, (None, g, beta)
    else:
        q, k, v, g, _ = (x.cuda() for x in synth_mamba_inputs(B, T, H, D, D, seed=3, dtype=torch.float32))
        op, rest = nat.nats_mixed_attn_mamba, (None, g)
    types = otab.synth_types(B, 3, H, 0.5, seed=3)
    low = [x.bfloat16() for x in (q, k, v)]
    run = lambda a, l: op(*a, *l, *rest, types.cuda(), None, nats_block_size=64, ops_for_incomplete_chunks="all")[:2]
    o_l, o_a = run(low, (q, k, v))
    assert o_l.dtype == torch.float32 and o_a.dtype == torch.bfloat16
    assert torch.equal(o_l, run((q, k, v), (q, k, v))[0])
    ref, _ = oattn.attn_sdpa(*(x.double().cpu() for x in low), oattn.attn_mask(types[..., 0], T, 64, H))
    assert_close(o_a, ref.float(), 2.0 ** -8, "o")           # one rounding of the output
    with pytest.raises(TypeError):
        run((q, k, v), low)
