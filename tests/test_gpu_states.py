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


def _inputs(B, T, H, HN, p, size, with_h0, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    k = (size * torch.nn.functional.normalize(rnd(B, T, H, 128), dim=-1)).bfloat16()
    # (w is made of normalised keys whatever the size of k: with larger ones the recurrence grows, and roundings with it)
    w, u = (0.05 * rnd(B, T, H, 128)).bfloat16(), rnd(B, T, H, 128).bfloat16()
    g = -0.1 * torch.rand(B, T, H, device="cuda", generator=gen)
    gcs = torch.cat([x.cumsum(1) for x in g.split(64, 1)], 1).contiguous()
    krs = (1 + 0.1 * torch.rand(B, T, H, device="cuda", generator=gen)) / size
    types = (torch.rand(B, -(-T // 64), HN, 2, device="cuda", generator=gen) < p).float()
    return k, w, u, gcs, krs, types, (rnd(B, H, 128, 128) if with_h0 else None)


def _states(k, w, u, gcs, krs, types, h0, decay, quirk, b0, b1):
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib
    T, H, HN = k.shape[1], k.shape[2], types.shape[2]
    tb = nat.build_selection_tables(types[b0:b1].contiguous(), T, 64)
    h = torch.full((b1 - b0, -(-T // 64), H, 128, 128), float("nan"), device="cuda", dtype=torch.bfloat16)
    carry = torch.full((b1 - b0, -(-T // 64), H), float("nan"), device="cuda")
    at = lambda x: None if x is None else x[b0:b1].data_ptr()
    flags = (_lib.FLAG_DECAY_SKIPPED if decay else 0) | (0 if quirk else _lib.FLAG_NO_TRAILING_QUIRK)
    _lib.call("natsl_linear_fwd_h", _lib.RULE_GDN, at(k), at(w), at(u), at(gcs), at(krs), tb.types_i.data_ptr(), tb.indices.data_ptr(),
              tb.n_blocks.data_ptr(), at(h0), h.data_ptr(), carry.data_ptr(), None, b1 - b0, T, H, HN, 128, 128, 64, flags,
              torch.cuda.current_stream().cuda_stream)
    return h, carry


def _exact(k, w, u, gcs, krs, types, h0, decay, quirk):
    """S <- e^{g_last+carry} S + k^T ((u - e^{carry} w S) rstd e^{g_last-g}) over the selected chunks, in float64."""
    k, w, u, gcs, krs = (x.double() for x in (k, w, u, gcs, krs))
    B, T, H, _ = k.shape
    sel = types[..., 1].bool().repeat_interleave(H // types.shape[2], 2)
    last = torch.where(sel, torch.arange(sel.shape[1], device="cuda").view(1, -1, 1), -1).amax(1)
    S = torch.zeros(B, H, 128, 128, device="cuda", dtype=torch.float64) if h0 is None else h0.double()
    carry, hs, cs = torch.zeros(B, H, device="cuda", dtype=torch.float64), [], []
    for c in range(sel.shape[1]):
        at = slice(64 * c, min(64 * c + 64, T))
        kc, wc, uc, gc, rc = (x[:, at].transpose(1, 2) for x in (k, w, u, gcs, krs))
        hs.append(S)
        cs.append(carry)
        gl = gc[..., -1]
        v = uc - carry.exp()[..., None, None] * (wc @ S)
        new = (gl + carry).exp()[..., None, None] * S + kc.transpose(-1, -2) @ (v * (rc * (gl[..., None] - gc).exp())[..., None])
        S = torch.where(sel[:, c][..., None, None], new, S)
        skipped = carry + gl * ((c < last) | (not quirk)) if decay else carry
        carry = torch.where(sel[:, c], torch.zeros_like(carry), skipped)
    return torch.stack(hs, 1), torch.stack(cs, 1)


@pytest.mark.parametrize("B,H,HN,T,p,size,with_h0,decay,quirk", [
    (5, 16, 16, 255, 0.5, 1.0, True, True, True), (5, 16, 4, 256, 0.5, 1.0, False, True, True), (7, 9, 3, 1000, 0.7, 1.0, True, True, True),
    (8, 8, 8, 383, 0.5, 1.0, False, True, True), (8, 8, 2, 384, 0.5, 1.0, True, True, False), (4, 16, 8, 1000, 0.6, 30.0, True, True, False),
    (37, 4, 4, 256, 0.3, 1.0, False, False, True), (149, 1, 1, 320, 0.5, 0.03, True, True, True), (12, 16, 16, 4096, 0.8, 1.0, False, True, True)])
def test_states_at_the_lines_of_the_rule(B, H, HN, T, p, size, with_h0, decay, quirk):
    """Both kernels in turn (63 and 64, 80, 148 and 149 pairs, sequences at their lines; a sequence alone takes the scan): the same
    bits, so that a sequence does not depend on the batch around it, and the recurrence in float64."""
    from neuralattentionsearchlinear_b200 import _lib
    x = _inputs(B, T, H, HN, p, size, with_h0, T + H)
    h, carry = _states(*x, decay, quirk, 0, B)
    for b in sorted({0, B // 2, B - 1}):
        h1, c1 = _states(*x, decay, quirk, b, b + 1)
        assert torch.equal(h[b], h1[0]) and torch.equal(carry[b], c1[0])
        ref, cref = _exact(*(None if t is None else t[b:b + 1] for t in x), decay, quirk)
        # bf16 roundings (2^-9 each) of the state that w reads, of v'' and of the result; what the first two leave behind decays
        assert (h1.double() - ref).norm() <= 3 * 2 ** -9 * ref.norm()
        torch.testing.assert_close(c1.double(), cref, rtol=1e-5, atol=1e-5)
    assert _lib.load().natsl_device_status() == 0
