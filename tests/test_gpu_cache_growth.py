"""A cache's rows moved into a longer buffer: the copy kernel at sizes around its 16 KB pieces, and where it leaves the copy to torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,n,old,new,width", [(1, 1, 1, 64, 8), (3, 7, 7, 320, 64), (2, 64, 100, 384, 128), (5, 65, 65, 384, 128),
                                               (1, 1000, 1030, 1344, 96), (2, 9, 9, 64, 3)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_rows_are_copied(B, n, old, new, width, dtype):
    from neuralattentionsearchlinear_b200.cache import _copy_rows
    src = torch.randn(B, old, 2, width, device="cuda").to(dtype)
    dst = torch.full((B, new, 2, width), 7.0, device="cuda", dtype=dtype)
    _copy_rows(dst, src, n)
    assert torch.equal(dst[:, :n], src[:, :n]) and bool((dst[:, n:] == 7).all())


def test_strided_and_tracked_rows():
    from neuralattentionsearchlinear_b200.cache import _copy_rows
    src = torch.randn(2, 16, 4, 8, device="cuda").transpose(2, 3)
    dst = torch.zeros(2, 32, 8, 4, device="cuda")
    _copy_rows(dst, src, 16)
    assert torch.equal(dst[:, :16], src)
    leaf = torch.randn(2, 16, 8, 4, device="cuda", requires_grad=True)
    dst = torch.zeros(2, 32, 8, 4, device="cuda")
    _copy_rows(dst, leaf, 16)
    dst.sum().backward()
    assert torch.equal(leaf.grad, torch.ones_like(leaf))


def _appended(k, v):
    """Two rows appended to a cache of plain rows k, v, whose buffers have to grow for them."""
    from neuralattentionsearchlinear_b200 import NAtSCache
    layer = NAtSCache().layer(0, 64)
    layer.append_kv(k, v)
    layer.append_kv(k[:, :2] * 2, v[:, :2] * 3)
    return layer.k_attn, layer.v_attn


def test_tangents_of_the_rows_are_kept():
    k, v, dk, dv = (torch.randn(2, 16, 2, 8, device="cuda") for _ in range(4))
    (ko, vo), (dko, dvo) = torch.func.jvp(_appended, (k, v), (dk, dv))
    assert torch.equal(ko, torch.cat([k, k[:, :2] * 2], 1)) and torch.equal(dko, torch.cat([dk, dk[:, :2] * 2], 1))
    assert torch.equal(vo, torch.cat([v, v[:, :2] * 3], 1)) and torch.equal(dvo, torch.cat([dv, dv[:, :2] * 3], 1))


def test_rows_under_vmap_and_in_a_trace():
    k, v, k2, v2 = (torch.randn(3, 2, 16, 2, 8, device="cuda") for _ in range(4))
    assert torch.equal(torch.vmap(_appended)(k, v)[0], torch.cat([k, k[:, :, :2] * 2], 2))
    traced = torch.jit.trace(_appended, (k[0], v[0]))
    for got, want in zip(traced(k2[1], v2[1]), _appended(k2[1], v2[1])):
        assert torch.equal(got, want)


def test_copy_in_one_compiled_graph():
    from neuralattentionsearchlinear_b200.cache import _copy_rows

    def grown(src):
        dst = src.new_zeros(src.shape[0], 64, *src.shape[2:])
        _copy_rows(dst, src, 16)
        return dst

    src = torch.randn(2, 16, 2, 8, device="cuda")
    assert torch.equal(torch.compile(grown, backend="eager", fullgraph=True)(src), grown(src))
