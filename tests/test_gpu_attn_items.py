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
