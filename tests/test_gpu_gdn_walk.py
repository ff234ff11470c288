"""GPU test (-m gpu) of the fused gated-delta-rule walks (natsl_gdn_walk on mma.sync, natsl_gdn_walk_fused_ex on tcgen05)
with the block-start state they hand to a decoder, against the oracle's token recurrence with re-roll: every built pair of
head dims, ragged last chunks and blocks, block sizes above 64, a last block of its own type linear or not."""
import pytest
import torch

from oracle import gdn as ogdn
from oracle import tables as otab
from tests.helpers import assert_close, synth_gdn_inputs

pytestmark = pytest.mark.gpu
TOL = 1e-2

CASES = [  # K, V, T, nbs, heads, selection heads, decay, initial state, tcgen05
    (64, 64, 64, 64, 2, 2, True, True, False), (64, 64, 65, 64, 4, 2, True, False, False),
    (64, 128, 320, 128, 2, 2, False, True, False), (128, 64, 255, 64, 2, 1, True, True, False),
    (128, 128, 37, 64, 2, 2, True, False, False), (128, 128, 449, 256, 2, 2, True, True, False),
    (128, 128, 512, 256, 2, 2, False, False, False), (128, 256, 384, 64, 3, 3, True, True, False),
    (192, 384, 200, 64, 2, 2, True, True, False), (192, 384, 256, 128, 2, 2, True, False, False),
    (128, 128, 64, 64, 2, 2, True, True, True), (128, 128, 448, 64, 4, 2, True, False, True),
    (128, 128, 300, 64, 2, 2, False, True, True),
]


@pytest.mark.parametrize("K,V,T,nbs,H,HN,decay,use_h0,tc", CASES)
@pytest.mark.parametrize("wide", [False, True])
def test_walk_outputs_and_states(K, V, T, nbs, H, HN, decay, use_h0, tc, wide, monkeypatch):
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    if wide and (tc or K == 192):
        pytest.skip("one slicing only")
    monkeypatch.setattr(_ops, "WALK_MMA_MAX_HEADS", 0 if tc else 10 ** 9)
    B = 2 if not wide else -(-160 * 32 // (H * V))           # enough (batch, head) pairs for the 64-column slices
    q, k, v, g, beta, h0 = synth_gdn_inputs(B, T, H, K, V, seed=T + K + V, normalize_qk=False)
    TN = -(-T // nbs)
    raw = otab.synth_types(B, TN, HN, 0.5, seed=T + 3, force_last=False)
    types = otab.force_last_block(raw.clone())
    dev = torch.device("cuda")
    c = lambda x: x.to(dev)
    tb = nat.build_selection_tables(c(types), T, nbs)
    o, ht, inter = _ops.linear_fwd(_lib.RULE_GDN, c(q), c(k), c(v), c(g), c(beta), tb, K ** -0.5, c(h0) if use_h0 else None, decay,
                                   True, True, want_start=True, last_types=c(raw[:, -1].bfloat16()))
    keep = slice(0, 2) if not wide else slice(B - 1, B)      # the oracle on a sample of the batch
    f = lambda x: x[keep].float()
    kw = dict(nbs=nbs, h0=h0[keep].float() if use_h0 else None, decay=decay, use_l2norm=True, rule="gdn", scale=K ** -0.5)
    args = (f(q), f(k), f(v), g[keep], f(beta))
    o_ref, fin_ref = ogdn.linear_recurrent(*args, types[keep][..., 1], **kw)
    _, _, start_ref = ogdn.linear_recurrent(*args, (raw if T % nbs == 0 else types)[keep][..., 1], return_block_start=True, **kw)
    assert_close(o[keep], o_ref, TOL, "o")
    assert_close(ht[keep], fin_ref, TOL, "final state")
    assert_close(inter["start"][keep], start_ref, TOL, "block-start state")
    assert _lib.load().natsl_device_status() == 0


@pytest.mark.parametrize("T,decay", [(1, True), (63, True), (65, True), (127, False), (128, True), (1100, True)])
def test_tc_walk_at_chunk_edges(T, decay, monkeypatch):
    """The tcgen05 walk stores whole chunks by TMA, which clips the last one, and every chunk adds up its own run of skipped ones."""
    test_walk_outputs_and_states(128, 128, T, 64, 3, 3, decay, True, True, False, monkeypatch)


@pytest.mark.parametrize("T,nbs,decay", [(64, 64, True), (300, 64, True), (512, 128, False), (640, 256, True)])
def test_mamba_walk_block_start_state(T, nbs, decay):
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    from tests.helpers import synth_mamba_inputs
    B, H, K, V = 2, 3, 128, 64
    q, k, v, g, h0 = synth_mamba_inputs(B, T, H, K, V, seed=T)
    raw = otab.synth_types(B, -(-T // nbs), H, 0.5, seed=T, force_last=False)
    types = otab.force_last_block(raw.clone())
    c = lambda x: x.cuda()
    tb = nat.build_selection_tables(c(types), T, nbs)
    o, ht, inter = _ops.linear_fwd(_lib.RULE_MAMBA, c(q), c(k), c(v), c(g), None, tb, 1.0, c(h0), decay, False, True,
                                   want_start=True, last_types=c(raw[:, -1]))
    kw = dict(nbs=nbs, h0=h0.float(), decay=decay, use_l2norm=False, rule="mamba", scale=1.0)
    args = (q.float(), k.float(), v.float(), g, None)
    o_ref, fin_ref = ogdn.linear_recurrent(*args, types[..., 1], **kw)
    _, _, start_ref = ogdn.linear_recurrent(*args, (raw if T % nbs == 0 else types)[..., 1], return_block_start=True, **kw)
    assert_close(o, o_ref, TOL, "o")
    assert_close(ht, fin_ref, TOL, "final state")
    assert_close(inter["start"], start_ref, TOL, "block-start state")
    assert _lib.load().natsl_device_status() == 0


def test_walk_of_more_than_2_31_outputs():
    """T * H * V = 2^31: offsets of the output that do not fit 32 bits, against the two-kernel form on the last tokens."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    T, H, K, V = 65536, 128, 128, 256
    gen = torch.Generator(device="cuda").manual_seed(0)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda", dtype=torch.bfloat16)
    q, k, v, beta = rnd(1, T, H, K), rnd(1, T, H, K), rnd(1, T, H, V), rnd(1, T, H).sigmoid()
    g = -torch.nn.functional.softplus(rnd(1, T, H).float())
    types = otab.synth_types(1, T // 64, 1, 0.5, seed=0).cuda()
    o = _ops.linear_fwd(_lib.RULE_GDN, q, k, v, g, beta, nat.build_selection_tables(types, T, 64), K ** -0.5, None, True, True, True)[0]
    n = 4096                                                 # the decayed state forgets what lies further back
    tail = [x[:, -n:].contiguous() for x in (q, k, v, g, beta)]
    tb = nat.build_selection_tables(types[:, -n // 64:].contiguous(), n, 64)
    want = _ops.linear_fwd(_lib.RULE_GDN, *tail, tb, K ** -0.5, None, True, True, True, return_intermediates=True)[0]
    assert_close(o[:, -n // 2:], want[:, -n // 2:].float(), TOL, "o")
    assert _lib.load().natsl_device_status() == 0


@pytest.mark.parametrize("T,nbs,want", [(512, 64, False), (500, 64, True), (512, 256, True)])
def test_760m_head_dims_keep_fp32(T, nbs, want):
    """K = 192, V = 384 holds the state and its operands to fp32 precision between bf16 tensors: the output is off from float64 by
    its one rounding to bf16 (2^-9 of an entry at most), the states by a few roundings to fp32 (2^-24 each).  Op and
    chunk-inference op."""
    import neuralattentionsearchlinear_b200 as nat
    B, H, K, V = 1, 2, 192, 384
    q, k, v, g, beta, h0 = synth_gdn_inputs(B, T, H, K, V, seed=T, normalize_qk=True)
    raw = otab.synth_types(B, -(-T // nbs), H, 0.5, seed=nbs, force_last=False)
    types = otab.force_last_block(raw.clone())
    c = lambda x: x.cuda()
    qa, ka, va = (c(x).view(B, T, 3 * H, -1) for x in (q, k, v))
    args = (qa, ka, va, c(q), c(k), c(v), c(h0), c(g), c(beta), c(types))
    opts = dict(nats_block_size=nbs, ops_for_incomplete_chunks="all", output_final_state_gated_delta=True, decay_for_non_gdn_blocks=True)
    kw = dict(nbs=nbs, h0=h0.double(), decay=True, use_l2norm=True, rule="gdn", scale=K ** -0.5)
    ref_in = (q.double(), k.double(), v.double(), g.double(), beta.double())
    o_ref, fin_ref = ogdn.linear_recurrent(*ref_in, types[..., 1], **kw)
    rel = lambda a, b: float((a.double().cpu() - b).norm() / b.norm())
    if want:
        o, _, ht, start = nat.nats_mixed_attn_gdn_chunk_inference(*args, c(raw[:, -1]) if T % nbs == 0 else None, None, **opts)
        _, _, start_ref = ogdn.linear_recurrent(*ref_in, (raw if T % nbs == 0 else types)[..., 1], return_block_start=True, **kw)
        assert rel(start, start_ref) <= 8 * 2.0 ** -24
    else:
        o, _, ht = nat.nats_mixed_attn_gdn(*args, None, **opts)
    assert rel(o, o_ref) <= 2.0 ** -9
    assert rel(ht, fin_ref) <= 8 * 2.0 ** -24
