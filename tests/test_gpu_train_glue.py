"""The small steps of the layers' training path against the same formulas in float64: rows that do not fill a CTA, heads that do not
divide one, tensors that do not start on 16 bytes, gradients that are absent, every grouping of the partial sums."""
import pytest
import torch

from neuralattentionsearchlinear_b200 import _lib
from neuralattentionsearchlinear_b200.modules import L2Norm, _BlockMeanFn, _column_sums, layer_gates

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _close(got, ref, terms=1):
    # bf16 results: one rounding (2^-8 of the value covers it and the flip of a rounded factor); `terms`: fp32 sums of so many terms
    got, ref = got.double(), ref.double()
    scale = ref.pow(2).mean().sqrt().clamp_min(1e-9)
    tol = 2 ** -8 * ref.abs() + 2 ** -20 * terms * scale
    assert got.shape == ref.shape and bool(((got - ref).abs() <= tol).all()), float(((got - ref).abs() / (ref.abs() + scale)).max())


def _reference(a, b, v, A_log, dt_bias, neg):
    dt = torch.nn.functional.softplus(a + dt_bias)
    beta = None if b is None else b.sigmoid() * (2 if neg else 1)
    return -A_log.exp() * dt, beta, None if v is None else v * dt.unsqueeze(-1)


@pytest.mark.parametrize("B,T,H,V", [(1, 1, 1, None), (2, 77, 6, None), (3, 65, 16, 64), (1, 333, 40, 128), (2, 9, 256, 32), (1, 700, 7, 256)])
@pytest.mark.parametrize("with_b,neg,f32,off", [(True, False, True, 0), (False, False, False, 1), (True, True, False, 0)])
def test_gates(B, T, H, V, with_b, neg, f32, off):
    g = torch.Generator(device="cuda").manual_seed(B * T + H)

    def rnd(*s, off=0, scale=1.0):
        n = torch.Size(s).numel()
        return (torch.randn(n + 8, generator=g, device="cuda") * scale).to(BF)[off:off + n].view(s).requires_grad_(True)

    a, b, v = rnd(B, T, H, scale=4.0), rnd(B, T, H) if with_b else None, None if V is None else rnd(B, T, H, V, off=off)
    with torch.no_grad():
        a.view(-1)[0] = 30.0                                 # beyond the softplus' threshold
    pdt = torch.float32 if f32 else BF
    A_log, bias = (torch.randn(H, generator=g, device="cuda").to(pdt).requires_grad_(True) for _ in range(2))
    out = layer_gates(a, A_log, bias, b=b, v=v, neg_eigval=neg)
    ref_in = [None if t is None else t.detach().double().requires_grad_(True) for t in (a, b, v, A_log, bias)]
    ref = _reference(*ref_in, neg)
    got, want = [(x, y) for x, y in zip(out, ref) if x is not None], None
    assert [x is None for x in out] == [x is None for x in ref]
    grads = [torch.randn(x.shape, generator=g, device="cuda").to(x.dtype) for x, _ in got]
    for x, y in got:
        _close(x.detach(), y.detach(), 4)
    torch.autograd.backward([x for x, _ in got], grads)
    torch.autograd.backward([y for _, y in got], [x.double() for x in grads])
    for t, r in zip((a, v), (ref_in[0], ref_in[2])):
        if t is not None:
            _close(t.grad, r.grad, 64)                       # the step size enters da as a sum of V products
    if b is not None:
        # as torch does it for bf16, sigmoid's gradient y (1 - y) is formed from y rounded to bf16, off by 2^-9 y at most, which
        # moves it by 2^-9 |1 - 2 y| y <= 2^-9; the result itself is rounded once
        dbeta = grads[1].double().abs() * (2 if neg else 1)
        assert bool(((b.grad.double() - ref_in[1].grad).abs() <= 2 ** -8 * ref_in[1].grad.abs() + 2 ** -9 * dbeta).all())
    for t, r in zip((A_log, bias), ref_in[3:]):
        assert float((t.grad.double() - r.grad).abs().max()) <= (2 ** -8 if not f32 else 1e-4) * float(r.grad.abs().max()) + 1e-3


def test_gates_with_a_gradient_missing_and_where_torch_runs():
    a = torch.randn(2, 70, 4, device="cuda").to(BF).requires_grad_(True)
    v = torch.randn(2, 70, 4, 64, device="cuda").to(BF).requires_grad_(True)
    A, bias = torch.zeros(4, device="cuda", requires_grad=True), torch.zeros(4, device="cuda", requires_grad=True)
    g, _, vo = layer_gates(a, A, bias, v=v)
    vo.float().sum().backward()
    assert torch.isfinite(a.grad).all() and float(A.grad.abs().max()) == 0.0
    assert layer_gates(a.float(), A, bias) is None and layer_gates(a, A.half(), bias) is None and layer_gates(a.cpu(), A, bias) is None
    assert layer_gates(a, A, bias, v=v[..., :24]) is None and layer_gates(a, torch.zeros(3, device="cuda"), bias) is None


@pytest.mark.parametrize("with_b,neg,V", [(True, True, None), (True, False, 64), (False, False, 64)])
def test_gates_second_derivatives(with_b, neg, V):
    """Differentiable gradients (``create_graph``): first and second derivatives of a scalar of the three outputs, against float64."""
    gen = torch.Generator(device="cuda").manual_seed(7)
    rnd = lambda *s, dt=BF: torch.randn(*s, generator=gen, device="cuda").to(dt).requires_grad_(True)
    a, b, v = rnd(2, 70, 4), rnd(2, 70, 4) if with_b else None, None if V is None else rnd(2, 70, 4, V)
    with torch.no_grad():
        a.view(-1)[0] = 30.0
    ins = (a, b, v, rnd(4, dt=torch.float32), rnd(4, dt=torch.float32))
    refs = tuple(None if t is None else t.detach().double().requires_grad_(True) for t in ins)

    def derivatives(run, ins):
        some = [t for t in ins if t is not None]
        out = [x for x in run(*ins) if x is not None]
        first = torch.autograd.grad(sum(x.to(torch.float64).square().sum() for x in out), some, create_graph=True)
        return first, torch.autograd.grad(sum(x.to(torch.float64).square().sum() for x in first), some)

    got = derivatives(lambda a, b, v, A, bias: layer_gates(a, A, bias, b=b, v=v, neg_eigval=neg), ins)
    want = derivatives(lambda a, b, v, A, bias: _reference(a, b, v, A, bias, neg), refs)
    for order, g, w in ((1, got[0], want[0]), (2, got[1], want[1])):
        for x, y in zip(g, w):
            # every bf16 tensor on the way (outputs, gradients, their gradients: five at most) is rounded once, 2^-9 each
            assert (x.double() - y).norm() <= 5 * 2 ** -9 * order * y.norm(), (order, x.shape)


@pytest.mark.parametrize("what", ["l2norm", "block mean", "gates"])
def test_batched_gradients(what):
    """``is_grads_batched`` and ``vmap`` over a backward pass: the rows of one gradient at a time."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn(2, 70, 4 if what == "gates" else 64, generator=gen, device="cuda").to(BF).requires_grad_(True)
    A = torch.randn(4, generator=gen, device="cuda")
    y = L2Norm()(x) if what == "l2norm" else _BlockMeanFn.apply(x, 64) if what == "block mean" else layer_gates(x, A, A)[0]
    dys = torch.randn(3, *y.shape, generator=gen, device="cuda").to(y.dtype)
    one = lambda dy: torch.autograd.grad(y, x, dy, retain_graph=True)[0]
    want = torch.stack([one(dy) for dy in dys])
    for got in (torch.autograd.grad(y, x, dys, retain_graph=True, is_grads_batched=True)[0], torch.vmap(one)(dys)):
        _close(got, want, 64)


@pytest.mark.parametrize("shape", [(1, 64), (7, 5, 128), (3, 41, 2, 256)])
def test_l2norm(shape):
    x = torch.randn(*shape, device="cuda").to(BF).requires_grad_(True)
    dy = torch.randn(*shape, device="cuda").to(BF)
    y = L2Norm()(x)
    y.backward(dy)
    r = x.detach().double().requires_grad_(True)
    want = r * (r.pow(2).sum(-1, keepdim=True) + 1e-6).rsqrt()
    want.backward(dy.double())
    _close(y.detach(), want.detach(), 4)
    _close(x.grad, r.grad, 16)
    # the gradient's own gradient, and forward mode, as torch operations give them
    z = torch.randn(2, 64, device="cuda").to(BF).requires_grad_(True)
    first, = torch.autograd.grad(L2Norm()(z).float().pow(3).sum(), z, create_graph=True)
    assert torch.autograd.grad(first.float().sum(), z)[0].shape == z.shape
    tangent = torch.func.jvp(lambda t: L2Norm()(t), (z.detach(),), (torch.ones_like(z),))[1]
    assert torch.isfinite(tangent).all()


def test_l2norm_and_gates_in_one_compiled_graph():
    x, A = torch.randn(2, 70, 64, device="cuda").to(BF), torch.randn(64, device="cuda")

    def run(x):
        gates = layer_gates(x, A, A)
        return L2Norm()(x), gates[0] if gates is not None else _reference(x.float(), None, None, A, A, False)[0]

    for got, want in zip(torch.compile(run, backend="eager", fullgraph=True)(x), run(x)):
        _close(got, want, 4)


@pytest.mark.parametrize("P,N,mode", [(1, 2, 1), (592, 2048, 0), (131, 33 * 5, 4), (40, 10, 4), (97, 256, 1)])
@pytest.mark.parametrize("dtypes", [(BF, torch.float32), (torch.float32, BF)])
def test_column_sums(P, N, mode, dtypes):
    part = torch.randn(P, N, device="cuda")
    n1 = {0: 0, 1: N // 2}.get(mode, N // 5)
    o0, o1 = (torch.full((n,), float("nan"), dtype=d, device="cuda") for n, d in zip((N - n1, n1), dtypes))
    _column_sums(part, mode, o0, o1 if n1 else None)
    want = part.double().sum(0)
    w0, w1 = (want, None) if mode == 0 else (want[:N // 2], want[N // 2:]) if mode == 1 else \
        (want.view(-1, 5)[:, :4].reshape(-1), want.view(-1, 5)[:, 4])
    _close(o0, w0, P)
    if n1:
        _close(o1, w1, P)
    if mode > 1:
        _column_sums(part, mode, o1.new_empty(N - n1))       # no bias


@pytest.mark.parametrize("B,T,D,nbs", [(1, 1, 8, 64), (2, 130, 24, 64), (1, 300, 64, 256)])
def test_block_mean_bwd_equals_the_torch_form(B, T, D, nbs):
    x = torch.randn(B, T, D, device="cuda").to(BF).requires_grad_(True)
    y = _BlockMeanFn.apply(x, nbs)
    dy = torch.randn_like(y)
    y.backward(dy)
    cnt = torch.full((y.shape[1],), float(nbs), device="cuda")
    cnt[-1] = T - (y.shape[1] - 1) * nbs
    want = (dy.float() / cnt.view(1, -1, 1)).to(BF).repeat_interleave(nbs, dim=1)[:, :T]
    assert torch.equal(x.grad, want)


@pytest.mark.parametrize("B,TN,HN,HQ,H", [(1, 1, 1, 1, 1), (2, 5, 2, 6, 4), (3, 87, 4, 4, 8)])
@pytest.mark.parametrize("dtype", [BF, torch.float32])
def test_types_grad(B, TN, HN, HQ, H, dtype):
    pa, pl = torch.randn(B, TN, HQ, device="cuda"), torch.randn(B, TN, H, device="cuda")
    types = torch.randint(0, 2, (B, TN, HN, 2), device="cuda", dtype=torch.int32)
    out = torch.empty(B, TN, HN, 2, dtype=dtype, device="cuda")
    _lib.call("natsl_types_grad", pa.data_ptr(), pl.data_ptr(), types.data_ptr(), out.data_ptr(), _lib.DT_BF16 if dtype == BF else _lib.DT_F32,
              B, TN, HN, HQ, H, torch.cuda.current_stream().cuda_stream)
    want = torch.stack([pa.double().view(B, TN, HN, -1).sum(-1) * (types[..., 0] != 0), pl.double().view(B, TN, HN, -1).sum(-1)], -1)
    _close(out, want, 4)
