"""GPU test (-m gpu) of the tcgen05 softmax backward at the edges of its tiles: 128-query tiles, pairs of 64-key tiles
(one key tile in all, an odd number, pairs far apart, none or every block selected), query heads of a group with
selections of their own, against the CPU oracle in float64."""
import pytest
import torch

from oracle import grad as ograd
from oracle import tables as otab
from tests.test_gpu_backward import close_scaled

pytestmark = pytest.mark.gpu

CASES = [  # T, query heads, key/value heads, selection heads, DK, DV, block, share of softmax blocks, own block, compat
    (1, 2, 2, 2, 128, 128, 64, 0.5, True, False), (63, 2, 2, 2, 64, 64, 64, 0.5, True, False),
    (64, 2, 2, 2, 128, 64, 64, 0.5, False, False), (65, 2, 2, 2, 64, 128, 64, 0.5, True, False),
    (129, 2, 2, 2, 128, 128, 64, 1.0, True, False), (191, 4, 1, 4, 128, 128, 64, 0.4, True, False),
    (320, 4, 2, 4, 64, 64, 64, 0.0, True, False), (577, 4, 2, 2, 128, 64, 128, 0.5, True, True),
    (832, 2, 2, 2, 128, 128, 192, 0.3, False, False), (1000, 16, 1, 8, 64, 128, 64, 0.2, True, False),
    (2112, 1, 1, 1, 128, 128, 64, 0.1, True, False),
]


@pytest.mark.parametrize("T,HQ,HKV,HN,DK,DV,nbs,p,own,compat", CASES)
def test_softmax_backward_tiles(T, HQ, HKV, HN, DK, DV, nbs, p, own, compat):
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    B = 2
    gen = torch.Generator().manual_seed(T + DK + DV)
    rnd = lambda *s: torch.randn(*s, generator=gen).bfloat16()
    q, k, v, do = rnd(B, T, HQ, DK), rnd(B, T, HKV, DK), rnd(B, T, HKV, DV), rnd(B, T, HQ, DV)
    types = otab.synth_types(B, -(-T // nbs), HN, p, seed=T)
    tb = nat.build_selection_tables(types.cuda(), T, nbs)
    scale = DK ** -0.5
    c = [x.cuda() for x in (q, k, v)]
    o, lse = _ops.attn_fwd(*c, tb, scale, own)
    got = _ops.attn_bwd(*c, o, lse, do.cuda(), tb, scale, own, reference_compat=compat)
    ref = ograd.attn_grads(q.double(), k.double(), v.double(), types[..., 0], do.double(), nbs=nbs, scale=scale, own_chunk=own,
                           reference_compat=compat)
    # dq: delta = rowsum(o do) is summed from o rounded to bf16 (2^-9 of an entry at most, 2^-9 / sqrt(3) in the mean), so
    # it is off by 0.0011 sqrt(128) = 0.0128 in the mean for normal o and do, and dq by that times scale |k|: 0.0064 with
    # DK = 64 and |k| = 4; three times that, over the millions of entries here, is 2e-2
    for x, name in zip(got, ("dq", "dk", "dv", "dnats")):
        close_scaled(x, ref[name], name, tol=2e-2 if name == "dq" else 1e-2, scale="max" if name == "dnats" else "auto")
    assert _lib.load().natsl_device_status() == 0
    again = _ops.attn_bwd(*c, o, lse, do.cuda(), tb, scale, own, reference_compat=compat)
    assert all(torch.equal(x, y) for x, y in zip(got, again))


@pytest.mark.parametrize("B,T,HQ,HKV,DK,DV", [(3, 700, 12, 6, 128, 128), (5, 300, 14, 7, 64, 64)])
def test_query_blocks_over_several_groups_of_heads(B, T, HQ, HKV, DK, DV):
    """More blocks of 128 queries than SMs, more heads than the 32 whose blocks are interleaved: what a CTA takes over from the
    grid, and the last group of heads, which is a smaller one."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    gen = torch.Generator().manual_seed(T)
    rnd = lambda *s: torch.randn(*s, generator=gen).bfloat16()
    q, k, v, do = rnd(B, T, HQ, DK), rnd(B, T, HKV, DK), rnd(B, T, HKV, DV), rnd(B, T, HQ, DV)
    types = otab.synth_types(B, -(-T // 64), HQ, 0.4, seed=T)
    tb = nat.build_selection_tables(types.cuda(), T, 64)
    c = [x.cuda() for x in (q, k, v)]
    o, lse = _ops.attn_fwd(*c, tb, DK ** -0.5, True)
    got = _ops.attn_bwd(*c, o, lse, do.cuda(), tb, DK ** -0.5, True)
    ref = ograd.attn_grads(q.double(), k.double(), v.double(), types[..., 0], do.double(), nbs=64, scale=DK ** -0.5, own_chunk=True)
    for x, name in zip(got, ("dq", "dk", "dv", "dnats")):     # (the bounds above)
        close_scaled(x, ref[name], name, tol=2e-2 if name == "dq" else 1e-2, scale="max" if name == "dnats" else "auto")
    assert _lib.load().natsl_device_status() == 0


@pytest.mark.parametrize("B,T,H,DK,DV,p", [(8, 128, 32, 64, 64, 1.0), (16, 256, 16, 128, 64, 0.5), (4, 1000, 16, 128, 64, 0.5)])
def test_sums_of_short_pairs_repeat(B, T, H, DK, DV, p):
    """Many pairs of key tiles with one or two steps each, one behind the other on an SM: the sums of a pair are not touched by the
    next one, nor are its gradients.  Bit for bit the same in every run, and the oracle's."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    gen = torch.Generator().manual_seed(T + H)
    rnd = lambda *s: torch.randn(*s, generator=gen).bfloat16()
    q, k, v, do = rnd(B, T, H, DK), rnd(B, T, H, DK), rnd(B, T, H, DV), rnd(B, T, H, DV)
    types = otab.synth_types(B, -(-T // 64), H, p, seed=T)
    tb = nat.build_selection_tables(types.cuda(), T, 64)
    c = [x.cuda() for x in (q, k, v)]
    o, lse = _ops.attn_fwd(*c, tb, DK ** -0.5, True)
    runs = [_ops.attn_bwd(*c, o, lse, do.cuda(), tb, DK ** -0.5, True) for _ in range(30)]
    assert all(torch.equal(x, y) for r in runs[1:] for x, y in zip(runs[0], r))
    for b in (0, B - 1):                                      # of the last one's blocks most are taken over
        row = slice(b, b + 1)
        ref = ograd.attn_grads(q[row].double(), k[row].double(), v[row].double(), types[row, ..., 0], do[row].double(), nbs=64,
                               scale=DK ** -0.5, own_chunk=True)
        for x, name in zip(runs[0], ("dq", "dk", "dv", "dnats")):                             # (the bounds above)
            close_scaled(x[row], ref[name], name, tol=2e-2 if name == "dq" else 1e-2, scale="max" if name == "dnats" else "auto")
    assert _lib.load().natsl_device_status() == 0


@pytest.mark.parametrize("B,T,HQ,HKV,DK,DV", [(2, 100, 37, 37, 64, 64), (3, 128, 50, 25, 128, 128), (4, 65, 37, 37, 128, 64),
                                              (1, 100, 149, 149, 64, 128), (37, 200, 1, 1, 128, 128)])
def test_halved_blocks_of_small_grids(B, T, HQ, HKV, DK, DV):
    """74, 75, 148, 149 and 74 blocks of the dk, dv kernel: halves that fit the SMs at once, halves that are taken over, whole
    blocks; pairs of selected tiles, unselected ones, both or one of either in a block."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    gen = torch.Generator().manual_seed(T + HQ)
    rnd = lambda *s: torch.randn(*s, generator=gen).bfloat16()
    q, k, v, do = rnd(B, T, HQ, DK), rnd(B, T, HKV, DK), rnd(B, T, HKV, DV), rnd(B, T, HQ, DV)
    types = otab.synth_types(B, -(-T // 64), HQ, 0.4, seed=T)
    tb = nat.build_selection_tables(types.cuda(), T, 64)
    c = [x.cuda() for x in (q, k, v)]
    o, lse = _ops.attn_fwd(*c, tb, DK ** -0.5, True)
    got = _ops.attn_bwd(*c, o, lse, do.cuda(), tb, DK ** -0.5, True)
    ref = ograd.attn_grads(q.double(), k.double(), v.double(), types[..., 0], do.double(), nbs=64, scale=DK ** -0.5, own_chunk=True)
    # (the bounds above; dnats here are sums over as little as one query, T = 65, so that delta's error, 0.0011 sqrt(DV) = 0.009 to
    # 0.0125 in the mean, comes through whole instead of cancelling over many queries: three times that over a few hundred entries)
    for x, name in zip(got, ("dq", "dk", "dv", "dnats")):
        close_scaled(x, ref[name], name, tol={"dq": 2e-2, "dnats": 4e-2}.get(name, 1e-2), scale="max" if name == "dnats" else "auto")
    assert _lib.load().natsl_device_status() == 0


@pytest.mark.parametrize("T,HQ,HKV,DK,DV,own", [(700, 4, 4, 128, 128, True), (1000, 4, 2, 64, 64, True), (460, 2, 2, 128, 64, False)])
@pytest.mark.parametrize("what", ["k", "v", "q", "do"])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_what_an_infinite_or_undefined_entry_reaches(T, HQ, HKV, DK, DV, own, what, value):
    """One entry of a key, value, query or output gradient: nothing changes, in any bit, outside the tiles of 128 queries and 64 keys
    that see each other (of a pair of key tiles, the one that the queries do not see is kept out by the products' lane mask),
    nor in other rows than the key's own."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    B, G, at = 2, HQ // HKV, T // 3
    gen = torch.Generator().manual_seed(T)
    rnd = lambda *s: torch.randn(*s, generator=gen).bfloat16().cuda()
    x = dict(q=rnd(B, T, HQ, DK), k=rnd(B, T, HKV, DK), v=rnd(B, T, HKV, DV), do=rnd(B, T, HQ, DV))
    types = otab.synth_types(B, -(-T // 64), HQ, 0.3, seed=T)
    tb = nat.build_selection_tables(types.cuda(), T, 64)
    o, lse = _ops.attn_fwd(x["q"], x["k"], x["v"], tb, DK ** -0.5, own)
    run = lambda y: _ops.attn_bwd(y["q"], y["k"], y["v"], o, lse, y["do"], tb, DK ** -0.5, own)
    clean = dict(zip(("q", "k", "v", "n"), run(x)))
    y = {n: t.clone() for n, t in x.items()}
    head = 1
    y[what][0, at, head, 5] = value
    got = dict(zip(("q", "k", "v", "n"), run(y)))
    NT, NQ = -(-T // 64), -(-T // 128)
    sel = types[0, ..., 0].bool()                             # [key tile, query head]
    sees = torch.zeros(NQ, NT, HQ, dtype=torch.bool)          # query tile, key tile
    for i in range(NQ):
        for j in range(NT):
            later = 64 * (j + 1) < min(128 * (i + 1), T)
            mine = j // 2 == i and (own or what in ("k", "v"))           # (dq masks the own tiles, with `own` off too)
            sees[i, j] = (sel[j] & later) | mine
    may = {n: torch.zeros(t.shape, dtype=torch.bool) for n, t in clean.items()}
    if what in ("k", "v"):
        for hq in range(head * G, head * G + G):
            for i in sees[:, at // 64, hq].nonzero().flatten().tolist():
                may["q"][0, 128 * i:128 * i + 128, hq] = True
            may["n"][0, at // 64, hq] = True
        may["k"][0, at, head] = True
        may["v"][0, at, head] = what == "k"
    else:
        may["q"][0, at, head] = True
        for j in sees[at // 128, :, head].nonzero().flatten().tolist():
            may["k"][0, 64 * j:64 * j + 64, head // G] = True
            may["v"][0, 64 * j:64 * j + 64, head // G] = True
            may["n"][0, j, head] = True
    for n, t in clean.items():
        same = (got[n] == t).cpu()
        assert bool((same | may[n]).all()), f"d{n}: {int((~same & ~may[n]).sum())} entries changed outside"
        assert may[n].all() or bool(torch.isfinite(got[n].cpu()[~may[n]]).all())
    assert _lib.load().natsl_device_status() == 0
