"""GPU test (-m gpu) of the states that every chunk of the gated delta rule reads: the tcgen05 walk that many (batch, head) pairs
take against the mma.sync scan that few of them take, at the edges of its chunks and of its runs of skipped blocks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,p,with_h0,decay", [(256, 0.5, False, True), (257, 1.0, True, True), (319, 0.0, True, True), (640, 0.1, False, False),
                                               (1000, 0.5, True, True), (1024, 1.0, False, True)])
def test_states_of_many_pairs(T, p, with_h0, decay):
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib
    B, H, NT = 5, 16, -(-T // 64)
    gen = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    k = torch.nn.functional.normalize(rnd(B, T, H, 128), dim=-1).bfloat16()
    w, u = (0.05 * rnd(B, T, H, 128)).bfloat16(), rnd(B, T, H, 128).bfloat16()
    g = -0.1 * torch.rand(B, T, H, device="cuda", generator=gen)
    gcs = torch.cat([x.cumsum(1) for x in g.split(64, 1)], 1).contiguous()
    krs = 1 + 0.1 * torch.rand(B, T, H, device="cuda", generator=gen)
    types = (torch.rand(B, NT, H, 2, device="cuda", generator=gen) < p).float()
    h0 = rnd(B, H, 128, 128) if with_h0 else None

    def states(b0, b1):
        tb = nat.build_selection_tables(types[b0:b1].contiguous(), T, 64)
        h = torch.full((b1 - b0, NT, H, 128, 128), float("nan"), device="cuda", dtype=torch.bfloat16)
        carry = torch.full((b1 - b0, NT, H), float("nan"), device="cuda")
        at = lambda x: None if x is None else x[b0:b1].data_ptr()
        _lib.call("natsl_linear_fwd_h", _lib.RULE_GDN, at(k), at(w), at(u), at(gcs), at(krs), tb.types_i.data_ptr(), tb.indices.data_ptr(),
                  tb.n_blocks.data_ptr(), at(h0), h.data_ptr(), carry.data_ptr(), None, b1 - b0, T, H, H, 128, 128, 64,
                  _lib.FLAG_DECAY_SKIPPED if decay else 0, torch.cuda.current_stream().cuda_stream)
        return h, carry

    h, carry = states(0, B)
    for b in range(B):                                        # 16 pairs: the scan
        h1, c1 = states(b, b + 1)
        # the same roundings to bf16 at the same places; products that add up in another order may turn some of them, by 2^-8
        assert (h[b] - h1[0]).float().norm() <= 2 ** -8 * h1.float().norm()
        torch.testing.assert_close(carry[b], c1[0], rtol=1e-6, atol=1e-6)
    assert _lib.load().natsl_device_status() == 0
    again, _ = states(0, B)
    assert torch.equal(h, again)
