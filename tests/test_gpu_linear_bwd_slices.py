"""GPU test (-m gpu) of the reverse walk's two slicings (64 value columns where those fill the SMs, 32 otherwise) and of
the kernels around it: many heads at once equal the same heads a few at a time, bit for bit (a warp does the same
arithmetic in both), and the few are held against the oracle in tests/test_gpu_backward.py."""
import pytest
import torch

from oracle import tables as otab
from tests.helpers import synth_gdn_inputs, synth_mamba_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rule,K,V,H,T", [("gdn", 64, 64, 148, 129), ("gdn", 128, 128, 74, 200), ("gdn", 128, 64, 150, 64),
                                          ("gdn", 64, 128, 76, 1), ("mamba", 128, 64, 148, 320), ("mamba", 64, 64, 160, 63)])
def test_wide_slices_equal_narrow_ones(rule, K, V, H, T):
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    gdn = rule == "gdn"
    if gdn:
        q, k, v, g, beta, h0 = (x.cuda() for x in synth_gdn_inputs(1, T, H, K, V, seed=T + V, normalize_qk=False))
    else:
        q, k, v, g, h0 = (x.cuda() for x in synth_mamba_inputs(1, T, H, K, V, seed=T + V))
        beta = None
    NT = -(-T // 64)
    types = otab.synth_types(1, NT, H, 0.4, seed=T).cuda()
    gen = torch.Generator().manual_seed(T)
    do, dht = torch.randn(1, T, H, V, generator=gen).bfloat16().cuda(), (torch.randn(1, H, K, V, generator=gen) * 0.1).cuda()

    def grads(s):
        c = lambda x: x[:, :, s].contiguous()
        tb = nat.build_selection_tables(c(types), T, 64)
        return _ops.linear_bwd(_lib.RULE_GDN if gdn else _lib.RULE_MAMBA, c(q), c(k), c(v), c(g), None if beta is None else c(beta), tb,
                               K ** -0.5, h0[:, s].contiguous(), True, gdn, c(do), dht=dht[:, s].contiguous())
    wide = grads(slice(0, H))
    for s in (slice(0, 2), slice(H - 3, H)):
        few = grads(s)
        for name in ("dq", "dk", "dv", "dg", "dnats") + (("dbeta",) if gdn else ()):
            assert torch.isfinite(few[name]).all() and torch.equal(wide[name][:, :, s], few[name]), name
        assert torch.equal(wide["dh0"][:, s], few["dh0"])
    assert _lib.load().natsl_device_status() == 0
