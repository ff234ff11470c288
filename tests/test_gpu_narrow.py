"""Narrow projections of the layer's forward at the edges of their tiles: features that do not fill a step of 64, one and several
tiles of tokens and of columns, heads between two groups of eight; the layer against its general path, and what the kernel itself
writes (log decays, their sums within a chunk, step sizes, betas, mixing weights) against float64."""
import pytest
import torch

from tests.test_gpu_layer_forward import _make
from tests.test_gpu_layer_forward import test_fused_forward_matches_the_general_path as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rule,args,B,T", [
    ("gdn", dict(hidden=96, heads=1, head_dim=64, expand_v=1, attn_heads=1), 1, 64),
    ("gdn", dict(hidden=1056, heads=9, head_dim=64, expand_v=1, attn_heads=9), 2, 129),
    ("gdn", dict(hidden=224, heads=20, head_dim=64, expand_v=1, attn_heads=20, allow_neg_eigval=True), 1, 257),
    ("mamba", dict(hidden=160, heads=5, head_dim=128, expand_v=0.5, attn_heads=5), 3, 127),
    ("mamba", dict(hidden=96, heads=17, head_dim=128, expand_v=0.5, attn_heads=17), 1, 321),
])
def test_tiles_of_the_narrow_projections(rule, args, B, T, monkeypatch):
    _check(rule, args, B, T, True, monkeypatch)


def _own_outputs(layer, x, monkeypatch):
    """The tensors that the two calls of the kernel read and write, from the workspace of the layer's native call (whose regions start on
    256 bytes in the order of ``sizes``)."""
    from neuralattentionsearchlinear_b200 import _lib, layer_forward as lf
    seen, empty, call = {}, torch.empty, _lib.call

    def keep(*shape, **kw):
        t = empty(*shape, **kw)
        if kw.get("dtype") == torch.uint8:
            seen["ws"] = t
        return t

    def look(name, *args):
        call(name, *args)
        if name == "natsl_layer_forward":
            a = args[0]._obj
            n, mamba, up = a.B * a.T, a.rule == _lib.RULE_MAMBA, lambda b: -(-b // 256) * 256
            hk, hv = 2 * n * a.H * a.K, 2 * n * a.H * a.V
            sizes = [("q", hk), ("k", hk), ("v", hv if mamba else 0), ("qa", hk if a.qn_w or mamba and a.attn_conv else 0),
                     ("qc", hk if mamba else 0), ("g", 4 * n * a.H), ("beta", 0 if mamba else 2 * n * a.H), ("dt", 8 * n * a.H if mamba else 0)]
            at = {}
            for name_, size in sizes:
                at[name_] = sum(up(b) for _, b in sizes[:len(at)])

            def read(start, shape, dtype):
                end = start + torch.Size(shape).numel() * torch.empty((), dtype=dtype).element_size()
                return seen["ws"][start:end].view(dtype).view(shape).clone()

            assert a.workspace == seen["ws"].data_ptr()
            seen["g"] = read(at["g"], (a.B, a.T, a.H), torch.float32)
            if mamba:
                seen["dt"], seen["gcs"] = read(at["dt"], (2, a.B, a.T, a.H), torch.float32)
            else:
                seen["beta"] = read(at["beta"], (a.B, a.T, a.H), torch.bfloat16)
            seen["q"] = read(at["qc" if mamba else "q"], (a.B, a.T, a.H * a.K), torch.bfloat16)
            seen["mix"] = read(a.mix - a.workspace, (a.B, a.T, a.HQ, 2), torch.bfloat16)

    monkeypatch.setattr(torch, "empty", keep)
    monkeypatch.setattr(_lib, "call", look)
    with torch.no_grad():
        layer(x)
    monkeypatch.undo()
    assert "g" in seen, "the native call did not run"
    return seen


def _bf16(x, slack):
    """x rounded to bf16, and where x +- slack rounds to the same value."""
    up, down = (x + slack).to(torch.bfloat16), (x - slack).to(torch.bfloat16)
    return x.to(torch.bfloat16).double(), up == down


def _linear(x, w):
    # fp32 sums of exact products: at most 2^-23 of the sum of magnitudes for each doubling of the terms
    x, w = x.double(), w.detach().double()
    return _bf16(x @ w.mT, 2 ** -20 * (x.abs() @ w.abs().mT))


@pytest.mark.parametrize("rule,args,B,T", [
    ("gdn", dict(hidden=96, heads=1, head_dim=64, expand_v=1, attn_heads=1), 2, 129),
    ("gdn", dict(hidden=1056, heads=9, head_dim=64, expand_v=1, attn_heads=9), 1, 200),
    ("gdn", dict(hidden=224, heads=20, head_dim=64, expand_v=1, attn_heads=20, allow_neg_eigval=True), 2, 321),
    ("gdn", dict(hidden=416, heads=4, head_dim=64, expand_v=1, attn_heads=4), 75, 257),       # more tiles than SMs, seven steps
    ("mamba", dict(hidden=160, heads=5, head_dim=128, expand_v=0.5, attn_heads=5), 1, 127),
    ("mamba", dict(hidden=96, heads=17, head_dim=128, expand_v=0.5, attn_heads=17), 1, 321),
    ("mamba", dict(hidden=416, heads=3, head_dim=128, expand_v=0.5, attn_heads=3), 75, 257),
])
def test_outputs_against_float64(rule, args, B, T, monkeypatch):
    torch.manual_seed(T)
    layer = _make(rule, **args).cuda().bfloat16().eval()
    with torch.no_grad():
        for p in (layer.a_proj.weight, layer.nats_out_weights_layer.weight):
            p.mul_(8.0)                                      # both sides of the softplus' threshold, mixing weights near 0 and 1
    x = torch.randn(B, T, args["hidden"], generator=torch.Generator().manual_seed(B)).bfloat16().cuda() * 4
    got = _own_outputs(layer, x, monkeypatch)
    # The products are rounded to bf16 before anything else; where float64 leaves no doubt about that rounding, the rest is fp32: log1p,
    # exp and a product, a few units of 2^-24 each (step size, decay), and one rounding to bf16 (beta, weights), which is exact
    # wherever an error of 2^-20 does not reach the next value.
    z, sure = _linear(x, layer.a_proj.weight)
    dt = torch.nn.functional.softplus(z + layer.dt_bias.detach().double())
    want = -layer.A_log.detach().double().exp() * dt
    assert float(sure.double().mean()) > 0.9 and bool(((got["g"].double() - want).abs() <= 2 ** -20 * want.abs())[sure].all())
    if rule == "mamba":
        assert bool(((got["dt"].double() - dt).abs() <= 2 ** -20 * dt)[sure].all())
        pad = torch.nn.functional.pad(got["g"].double(), (0, 0, 0, -T % 64)).view(B, -1, 64, args["heads"])
        sums = pad.cumsum(2).view(B, -1, args["heads"])[:, :T]
        assert bool(((got["gcs"].double() - sums).abs() <= 2 ** -21 * sums.abs()).all())      # at most six fp32 additions deep
    else:
        z, sure = _linear(x, layer.b_proj.weight)
        beta = z.sigmoid()
        want, exact = _bf16(beta, 2 ** -20 * beta)
        assert bool((got["beta"].double() == want * (2 if args.get("allow_neg_eigval") else 1))[sure & exact].all())
    z, sure = _linear(got["q"], layer.nats_out_weights_layer.weight)
    w = z.unflatten(-1, (-1, 2)).softmax(-1)
    want, exact = _bf16(w, 2 ** -19 * w)
    both = sure.unflatten(-1, (-1, 2)).all(-1, keepdim=True) & exact
    assert float(both.double().mean()) > 0.7 and bool((got["mix"].double() == want)[both].all())


def test_infinite_mixing_logits(monkeypatch):
    """As torch's softmax: a logit of +inf gives NaN, one of -inf beside a finite one a weight of zero."""
    torch.manual_seed(1)
    layer = _make("gdn", hidden=96, heads=2, head_dim=64, expand_v=1, attn_heads=2).cuda().bfloat16().eval()
    w = layer.nats_out_weights_layer.weight
    with torch.no_grad():
        w[::2] = 0
        w[0, 5], w[2, 70] = 3e38, -3e38                      # the heads' first logits: one product each, of activations above -0.3
    got = _own_outputs(layer, torch.randn(1, 300, 96).bfloat16().cuda() * 20, monkeypatch)
    z = torch.nn.functional.linear(got["q"].double(), w.detach().double()).to(torch.bfloat16).unflatten(-1, (-1, 2))
    inf, want = z[..., 0].isinf(), z.softmax(-1)
    assert inf[..., 0].any() and (z[..., 0, 0][inf[..., 0]] > 0).all() and inf[..., 1].any() and (z[..., 1, 0][inf[..., 1]] < 0).all()
    assert want[..., 0, :][inf[..., 0]].isnan().all() and torch.equal(got["mix"][inf].nan_to_num(2.0), want[inf].nan_to_num(2.0))
