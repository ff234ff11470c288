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
