"""The softmax branch's work items: lengths around the edges of 64-key units, 128-query tiles and 256-query items, block sizes
whose blocks do not line up with them, everything and nothing selected, and more items than SMs.  Against the oracle's dense
mask in fp32 on the same bf16 inputs; P is rounded to bf16 (2^-9 relative) and so is the output: 1e-2 covers both."""
from __future__ import annotations

import pytest
import torch

from helpers import assert_close
from oracle import attn as oattn

pytestmark = pytest.mark.gpu


def _inputs(B, T, HQ, HKV, DK, DV, nbs, p, seed):
    gen = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=gen).bfloat16()
    types = torch.zeros(B, -(-T // nbs), HKV, 2)
    types[..., 0] = (torch.rand(B, types.shape[1], HKV, generator=gen) < p).float()
    types[..., 1] = 1 - types[..., 0]
    types[:, -1] = 1
    return rnd(B, T, HQ, DK), rnd(B, T, HKV, DK), rnd(B, T, HKV, DV), types


def _both(q, k, v, types):
    """(o, lse, reference o, reference lse) on the CPU, blocks of 64."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _ops
    T, scale = q.shape[1], q.shape[3] ** -0.5
    o, lse = _ops.attn_fwd(q.cuda(), k.cuda(), v.cuda(), nat.build_selection_tables(types.cuda(), T, 64), scale, True)
    ref = oattn.attn_sdpa(q.float(), k.float(), v.float(), oattn.attn_mask(types[..., 0], T, 64, q.shape[2], own_chunk=True), scale)
    return o.cpu(), lse.cpu(), *ref


def _check(q, k, v, types, nbs, own=True):
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    T, HQ, scale = q.shape[1], q.shape[2], q.shape[3] ** -0.5
    tb = nat.build_selection_tables(types.cuda(), T, nbs)
    o, lse = _ops.attn_fwd(q.cuda(), k.cuda(), v.cuda(), tb, scale, own)
    o_ref, lse_ref = oattn.attn_sdpa(q.float(), k.float(), v.float(), oattn.attn_mask(types[..., 0], T, nbs, HQ, own_chunk=own), scale)
    assert_close(o, o_ref, 1e-2, "o_attn")
    assert_close(lse, lse_ref, 1e-2, "lse")
    assert _lib.load().natsl_device_status() == 0
    return o


@pytest.mark.parametrize("DK,DV", [(64, 64), (64, 128), (128, 64), (128, 128)])
@pytest.mark.parametrize("T", [1, 64, 65, 127, 129, 192, 193, 256, 257, 385, 700])
def test_lengths(T, DK, DV):
    _check(*_inputs(2, T, 4, 2, DK, DV, 64, 0.5, T), 64)


@pytest.mark.parametrize("own", [True, False])
@pytest.mark.parametrize("p", [0.0, 0.4, 1.0])
@pytest.mark.parametrize("nbs,T", [(128, 900), (192, 1000), (256, 1030), (320, 1400), (1024, 1500)])
def test_block_sizes(nbs, T, p, own):
    _check(*_inputs(1, T, 2, 2, 64, 64, nbs, p, nbs), nbs, own)
    _check(*_inputs(1, T, 2, 1, 128, 128, nbs, p, nbs), nbs, own)


@pytest.mark.parametrize("T,DK,DV", [(130, 64, 64), (515, 128, 128)])
def test_more_items_than_sms(T, DK, DV):
    """Each SM goes through several items; a sequence's result does not depend, bit for bit, on how many there are."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _ops
    q, k, v, types = _inputs(24, T, 16, 16, DK, DV, 64, 0.4, T)
    o = _check(q, k, v, types, 64)
    tb = nat.build_selection_tables(types[5:6].cuda(), T, 64)
    one, _ = _ops.attn_fwd(q[5:6].cuda(), k[5:6].cuda(), v[5:6].cuda(), tb, DK ** -0.5, True)
    assert torch.equal(one, o[5:6])


@pytest.mark.parametrize("nbs", [64, 128, 192, 256])
@pytest.mark.parametrize("DK,DV", [(64, 64), (64, 128), (128, 64), (128, 128)])
def test_one_tile_and_two_tile_items(DK, DV, nbs):
    """Few tiles: a block of the grid is one tile; many: two tiles that share their loads.  The same bits either way."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    q, k, v, types = (x.cuda() for x in _inputs(8, 643, 8, 4, DK, DV, nbs, 0.4, nbs))
    o, lse = _ops.attn_fwd(q, k, v, nat.build_selection_tables(types, 643, nbs), DK ** -0.5, True)
    for b in (0, 5):
        few = slice(b, b + 1)
        tb = nat.build_selection_tables(types[few].contiguous(), 643, nbs)
        o1, lse1 = _ops.attn_fwd(q[few], k[few], v[few], tb, DK ** -0.5, True)
        assert torch.equal(o1, o[few]) and torch.equal(lse1, lse[few])
    assert _lib.load().natsl_device_status() == 0


@pytest.mark.parametrize("q_off,nbs", [(128, 64), (384, 64), (384, 128), (640, 128)])
@pytest.mark.parametrize("DK,DV", [(64, 64), (128, 128)])
def test_window_on_an_odd_tile(q_off, nbs, DK, DV):
    """Queries from an odd multiple of 128 on: the items do not start where those of the whole sequence do."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _ops
    T = 900
    q, k, v, types = _inputs(2, T, 4, 2, DK, DV, nbs, 0.5, q_off)
    tb = nat.build_selection_tables(types.cuda(), T, nbs)
    o, lse = _ops.attn_fwd(q[:, q_off:].contiguous().cuda(), k.cuda(), v.cuda(), tb, DK ** -0.5, True, q_off=q_off)
    o_ref, lse_ref = oattn.attn_sdpa(q.float(), k.float(), v.float(), oattn.attn_mask(types[..., 0], T, nbs, 4, own_chunk=True), DK ** -0.5)
    assert_close(o, o_ref[:, q_off:], 1e-2, "o_attn")
    assert_close(lse, lse_ref[:, q_off:], 1e-2, "lse")


@pytest.mark.parametrize("DK,DV", [(64, 64), (128, 128)])
def test_infinite_scores(DK, DV):
    """A key whose score is +inf for half of the rows, -inf for the others: no weight and no effect where it is -inf, NaN (as
    softmax gives it) where it is +inf, and nothing of it where it is not visible."""
    q, k, v, types = _inputs(1, 400, 1, 1, DK, DV, 64, 0.0, 5)
    q[..., 0] = torch.where(torch.arange(400) % 2 == 0, 1.0, -1.0).bfloat16().view(1, 400, 1)
    types[:, 2] = 1                                        # keys 128..191: seen by every later block
    k[:, 130] = 0
    k[:, 130, :, 0] = float("inf")
    o, lse, o_ref, lse_ref = _both(q, k, v, types)
    hit = (torch.arange(400) >= 130) & (torch.arange(400) % 2 == 0)
    assert torch.isnan(o_ref[0, hit]).all() and torch.isnan(o[0, hit]).all()
    assert_close(o[0, ~hit], o_ref[0, ~hit], 1e-2, "o_attn")
    assert_close(lse[0, ~hit], lse_ref[0, ~hit], 1e-2, "lse")


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("DK,DV", [(64, 64), (128, 128)])
def test_keys_behind_the_mask(bad, DK, DV):
    """NaN or infinities in a key reach the rows that see it and no other: same bits as without."""
    q, k, v, types = _inputs(1, 512, 1, 1, DK, DV, 64, 0.0, 7)
    clean, clean_lse, _, _ = _both(q, k, v, types)
    k[:, 70] = bad                                         # block 1, seen by the rows 70..127
    o, lse, _, _ = _both(q, k, v, types)
    sees = (torch.arange(512) >= 70) & (torch.arange(512) < 128)
    assert torch.equal(o[0, ~sees], clean[0, ~sees]) and torch.equal(lse[0, ~sees], clean_lse[0, ~sees])
    assert torch.isnan(o[0, sees]).all()


def test_values_behind_the_mask():
    """NaN in the values of blocks that a query tile does not see at all are not in its output."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _ops
    q, k, v, types = _inputs(1, 512, 1, 1, 64, 64, 64, 0.0, 3)
    clean = _check(q, k, v, types, 64)
    v[:, 64:128] = float("nan")                            # block 1: seen by its own 64 rows alone
    tb = nat.build_selection_tables(types.cuda(), 512, 64)
    o, _ = _ops.attn_fwd(q.cuda(), k.cuda(), v.cuda(), tb, 0.125, True)
    assert torch.equal(o[:, 128:], clean[:, 128:]) and torch.isnan(o[:, 64:128]).all()


def test_output_on_sixteen_bytes():
    """An output that starts on 16 but not on 32 bytes takes the narrower stores."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib, _ops
    q, k, v, types = (x.cuda() for x in _inputs(1, 300, 2, 2, 64, 64, 64, 0.5, 9))
    tb = nat.build_selection_tables(types, 300, 64)
    ref, _ = _ops.attn_fwd(q, k, v, tb, 0.125, True)
    buf, lse = torch.zeros(ref.numel() + 8, dtype=ref.dtype, device="cuda"), torch.empty(1, 300, 2, device="cuda")
    o = buf[8:].view_as(ref)
    _lib.call("natsl_attn_fwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), tb.types_i.data_ptr(), tb.indices.data_ptr(),
              tb.attn_n_iters.data_ptr(), o.data_ptr(), lse.data_ptr(), 1, 300, 2, 2, 2, 64, 64, 64, 0.125,
              _lib.FLAG_ATTN_OWN_CHUNK, torch.cuda.current_stream().cuda_stream)
    assert torch.equal(o, ref)
