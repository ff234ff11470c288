"""Edges of the row and convolution kernels: rows that do not fill a turn of the grid, one row, tensors that do not start on 16
bytes, channel counts between two tiles, blocks between two groups of loads; against the same formulas in float64."""
import pytest
import torch

from neuralattentionsearchlinear_b200 import _lib

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
EPS = 1e-6


def _rand(gen, *shape, off=0):
    """bf16 values; ``off`` elements behind an address that is a multiple of 16 bytes."""
    n = 1
    for s in shape:
        n *= s
    buf = torch.randn(n + 8, generator=gen, device="cuda").to(BF)
    return buf[off:off + n].view(shape)


def _st():
    return torch.cuda.current_stream().cuda_stream


def _close(got, ref, fp32=False):
    # bf16 outputs: one rounding (2^-9 of the value) and a few fp32 roundings of terms as large as the row's values;
    # fp32 sums over n rows: n roundings of 2^-24 of the sum of magnitudes, far below 1e-4 of the result's size here
    got, ref = got.double(), ref.double()
    scale = ref.pow(2).mean().sqrt().clamp_min(1e-6)
    tol = (1e-4 * scale if fp32 else 2 ** -8 * ref.abs() + 1e-5 * scale)
    assert bool(((got - ref).abs() <= tol).all()), float(((got - ref).abs() - tol).max())


@pytest.mark.parametrize("D", [64, 128, 256, 512, 1024, 2048])
@pytest.mark.parametrize("rows,add,w32", [(1, False, False), (7, True, True), (4 * 592 + 5, True, False)])
@pytest.mark.parametrize("off", [0, 1])
def test_rmsnorm_bwd(D, rows, add, w32, off):
    if off and D >= 256 and rows > 7:
        pytest.skip("one size is enough")
    g = torch.Generator(device="cuda").manual_seed(D + rows)
    s, dy, da = (_rand(g, rows, D, off=off) for _ in range(3))
    w = torch.randn(D, generator=g, device="cuda").to(torch.float32 if w32 else BF)
    n_part = min(-(-rows // 8), 592)
    dx, part = torch.empty(rows, D, dtype=BF, device="cuda"), torch.full((n_part, D), float("nan"), device="cuda")
    _lib.call("natsl_rmsnorm_bwd", s.data_ptr(), w.data_ptr(), _lib.DT_F32 if w32 else _lib.DT_BF16, dy.data_ptr(),
              da.data_ptr() if add else None, dx.data_ptr(), part.data_ptr(), n_part, rows, D, EPS, _st())
    x, gy, wd = s.double(), dy.double(), w.double()
    rstd = (x.pow(2).mean(-1, keepdim=True) + EPS).rsqrt()
    xh = x * rstd
    ref = rstd * (gy * wd - xh * (gy * wd * xh).mean(-1, keepdim=True)) + (da.double() if add else 0.0)
    _close(dx, ref)
    _close(part.sum(0), (gy * xh).sum(0), fp32=True)


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("rows,act,off", [(1, 0, 0), (35, 1, 1), (148 * 8 * 32 + 3, 0, 0)])
def test_norm_gate_mix(D, rows, act, off):
    g = torch.Generator(device="cuda").manual_seed(D + rows)
    x1, x2, gt, dy = (_rand(g, rows, D, off=off if i == 3 else 0) for i in range(4))
    xw = torch.rand(rows, 2, generator=g, device="cuda").to(BF)
    w1, w2 = (torch.randn(D, generator=g, device="cuda").to(BF) for _ in range(2))
    y = torch.empty(rows, D, dtype=BF, device="cuda")
    _lib.call("natsl_norm_gate_mix", x1.data_ptr(), x2.data_ptr(), gt.data_ptr(), xw.data_ptr(), 0, w1.data_ptr(), w2.data_ptr(), 0,
              y.data_ptr(), rows, D, EPS, act, _st())
    leaves = [t.double().requires_grad_(True) for t in (x1, x2, gt, xw, w1, w2)]
    a, b, c, m, u, v = leaves
    n1 = a * (a.pow(2).mean(-1, keepdim=True) + EPS).rsqrt() * u
    n2 = b * (b.pow(2).mean(-1, keepdim=True) + EPS).rsqrt() * v
    ref = (n1 * m[:, :1] + n2 * m[:, 1:]) * (c.sigmoid() * (1.0 if act else c))
    _close(y, ref.detach())
    ref.backward(dy.double())
    n_part = min(-(-rows // 8), 592)
    outs = [torch.empty(rows, D, dtype=BF, device="cuda") for _ in range(3)]
    dxw, part = torch.empty(rows, 2, device="cuda"), torch.full((n_part, 2, D), float("nan"), device="cuda")
    _lib.call("natsl_norm_gate_mix_bwd", x1.data_ptr(), x2.data_ptr(), gt.data_ptr(), xw.data_ptr(), 0, w1.data_ptr(), w2.data_ptr(), 0,
              dy.data_ptr(), *(o.data_ptr() for o in outs), dxw.data_ptr(), part.data_ptr(), n_part, rows, D, EPS, act, _st())
    for got, leaf in zip(outs, leaves[:3]):
        _close(got, leaf.grad)
    _close(dxw, m.grad, fp32=True)
    _close(part.sum(0), torch.stack([u.grad, v.grad]), fp32=True)


@pytest.mark.parametrize("B,T,D,off", [(1, 3, 8, 0), (2, 65, 136, 0), (1, 130, 256, 3), (3, 64, 40, 1)])
@pytest.mark.parametrize("silu", [0, 1])
def test_short_conv(B, T, D, off, silu):
    g = torch.Generator(device="cuda").manual_seed(T + D)
    x, dy, w, bias = _rand(g, B, T, D), _rand(g, B, T, D), _rand(g, D, 4, off=off), _rand(g, D)
    y, dx = torch.empty_like(x), torch.empty_like(x)
    part = torch.full((B * -(-T // 64), D, 5), float("nan"), device="cuda")
    _lib.call("natsl_short_conv_fwd", x.data_ptr(), w.data_ptr(), bias.data_ptr(), y.data_ptr(), B, T, D, 4, silu, _st())
    _lib.call("natsl_short_conv_bwd", x.data_ptr(), w.data_ptr(), bias.data_ptr(), dy.data_ptr(), dx.data_ptr(), part.data_ptr(), B, T, D, 4,
              silu, 64, _st())
    a, u, v = (t.double().requires_grad_(True) for t in (x, w, bias))
    ref = torch.nn.functional.conv1d(a.transpose(1, 2), u.unsqueeze(1), v, padding=3, groups=D)[..., :T].transpose(1, 2)
    ref = torch.nn.functional.silu(ref) if silu else ref
    _close(y, ref.detach())
    ref.backward(dy.double())
    _close(dx, a.grad)
    dw = part.sum(0)
    _close(dw[:, :4], u.grad, fp32=True)
    _close(dw[:, 4], v.grad, fp32=True)


@pytest.mark.parametrize("B,T,D,nbs", [(1, 15, 8, 64), (2, 81, 264, 64), (2, 300, 32, 256), (1, 64, 16, 16)])
def test_block_mean_adds_tokens_in_their_order(B, T, D, nbs):
    g = torch.Generator(device="cuda").manual_seed(T)
    x = _rand(g, B, T, D)
    NB = -(-T // nbs)
    y = torch.empty(B, NB, D, dtype=BF, device="cuda")
    _lib.call("natsl_block_mean", x.data_ptr(), y.data_ptr(), B, T, D, nbs, _st())
    for c in range(NB):
        acc = torch.zeros(B, D, device="cuda")
        rows = x[:, c * nbs:(c + 1) * nbs].float()
        for t in range(rows.shape[1]):
            acc = acc + rows[:, t]
        inv = (torch.ones((), device="cuda") / rows.shape[1])
        assert torch.equal(y[:, c], (acc * inv).to(BF))


@pytest.mark.parametrize("act", [0, 1])
def test_sigmoid_of_pairs_in_fp32(act):
    """The mixing weights' gradient is a sum over a row in fp32: with one feature that is not zero it is the gate's function itself, for
    every bf16 gate up to 80.  ``__expf`` is off by 2 + 1.173 |x| units of 2^-23 at most, the reciprocal with its step of Newton's
    iteration by one, the sum in front of it and the products by half a one each."""
    bits = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.uint16).view(BF)
    gate = bits[(bits.float().abs() <= 80) & ((bits.float().abs() >= 2 ** -60) | (bits == 0))]
    rows, D, j = gate.numel(), 64, 21
    one = torch.zeros(rows, D, dtype=BF, device="cuda")
    one[:, j] = 1
    gt = one * gate[:, None]
    xw = torch.ones(rows, 2, device="cuda")
    n_part = min(-(-rows // 8), 592)
    outs = [torch.empty(rows, D, dtype=BF, device="cuda") for _ in range(3)]
    dxw, part = torch.empty(rows, 2, device="cuda"), torch.empty(n_part, 2, D, device="cuda")
    _lib.call("natsl_norm_gate_mix_bwd", one.data_ptr(), one.data_ptr(), gt.data_ptr(), xw.data_ptr(), _lib.DT_F32, None, None, 0, one.data_ptr(),
              *(o.data_ptr() for o in outs), dxw.data_ptr(), part.data_ptr(), n_part, rows, D, 0.0, act, _st())
    x = gate.double()
    want = 8.0 * x.sigmoid() * (1.0 if act else x)            # x / sqrt(mean(x^2)) = 8, up to the two units of rsqrtf
    for got in dxw.double().unbind(1):
        assert bool(((got - want).abs() <= 2 ** -23 * (7 + 1.173 * x.abs()) * want.abs()).all())


@pytest.mark.parametrize("B,T,D,span", [(2, 131, 72, 32), (1, 300, 136, 100), (2, 64, 8, 7)])
def test_short_conv_bwd_over_other_spans(B, T, D, span):
    """Spans of other than 64 tokens per partial sum (a kernel of their own) give the same gradients."""
    g = torch.Generator(device="cuda").manual_seed(T)
    x, dy, w, bias = _rand(g, B, T, D), _rand(g, B, T, D), _rand(g, D, 4), _rand(g, D)
    got = []
    for s in (64, span):
        dx, part = torch.empty_like(x), torch.full((B * -(-T // s), D, 5), float("nan"), device="cuda")
        _lib.call("natsl_short_conv_bwd", x.data_ptr(), w.data_ptr(), bias.data_ptr(), dy.data_ptr(), dx.data_ptr(), part.data_ptr(), B, T, D, 4,
                  1, s, _st())
        got.append((dx, part.sum(0)))
    _close(got[1][0], got[0][0])
    _close(got[1][1], got[0][1], fp32=True)


def test_forward_kernels_refuse_tensors_between_their_loads():
    """What reads or writes whole vectors is refused on the host where a tensor starts between two of them."""
    t = torch.zeros(4096, dtype=BF, device="cuda")
    on, off = t.data_ptr(), t.data_ptr() + 2
    calls = {"natsl_rmsnorm_fwd": ([on, None, None, 0, on, None], (1, 64, EPS)), "natsl_norm_gate_mix": ([on, on, on, None, 0, None, None, 0, on], (1, 64, EPS, 0)),
             "natsl_short_conv_fwd": ([on, on, None, on], (1, 4, 8, 4, 1)), "natsl_short_conv_bwd": ([on, on, None, on, on, on], (1, 4, 8, 4, 1, 64)),
             "natsl_swiglu_fwd": ([on, on, on], (8,)), "natsl_swiglu_bwd": ([on] * 5, (8,)), "natsl_block_mean": ([on, on], (1, 4, 8, 64))}
    weights = {("natsl_short_conv_fwd", 1), ("natsl_short_conv_bwd", 1), ("natsl_short_conv_bwd", 5)}      # (and partial sums, fp32)
    for name, (tensors, sizes) in calls.items():
        for i, p in enumerate(tensors):
            if p == on and (name, i) not in weights:
                with pytest.raises(_lib.NatslError, match="does not start"):
                    _lib.call(name, *tensors[:i], off, *tensors[i + 1:], *sizes, _st())
