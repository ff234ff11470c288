"""GPU test (-m gpu): a tensor that both branches read gets its gradient from the linear branch's last kernel, which adds onto the
softmax branch's.  Both gradients are bf16 values and each sum is rounded once, so it is bit for bit the sum of the two gradients that
separate copies get."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rule,B,T,H,K,V,which", [
    ("gdn", 1, 1, 1, 64, 64, "qkv"), ("gdn", 2, 65, 2, 128, 64, "qkv"), ("gdn", 1, 127, 3, 64, 128, "qv"),
    ("gdn", 2, 200, 2, 128, 128, "qkv"), ("gdn", 1, 300, 2, 128, 128, "k"), ("mamba", 2, 190, 2, 128, 64, "qkv"),
    ("mamba", 1, 64, 1, 128, 64, "q")])
def test_shared_inputs_get_the_sum_of_both_gradients(rule, B, T, H, K, V, which):
    import neuralattentionsearchlinear_b200 as nat
    gen = torch.Generator().manual_seed(B * T + K + V)
    rnd = lambda *s: torch.randn(*s, generator=gen)
    one = torch.nn.functional.normalize
    base = dict(q=one(rnd(B, T, H, K), dim=-1), k=one(rnd(B, T, H, K), dim=-1), v=rnd(B, T, H, V))
    g, beta = -torch.nn.functional.softplus(rnd(B, T, H)).cuda(), rnd(B, T, H).sigmoid().bfloat16().cuda()
    types = (rnd(B, -(-T // 64), H, 2) > 0).float().cuda()
    do_l, do_a = rnd(B, T, H, V).bfloat16().cuda(), rnd(B, T, H, V).bfloat16().cuda()
    grads = []
    for shared in (True, False):
        lin = {n: x.bfloat16().cuda().requires_grad_() for n, x in base.items()}
        att = {n: lin[n] if shared and n in which else lin[n].detach().clone().requires_grad_() for n in lin}
        args = (att["q"], att["k"], att["v"], lin["q"], lin["k"], lin["v"], None, g) + ((beta,) if rule == "gdn" else ())
        op = nat.nats_mixed_attn_gdn if rule == "gdn" else nat.nats_mixed_attn_mamba
        out = op(*args, types, None, nats_block_size=64, ops_for_incomplete_chunks="all")
        torch.autograd.backward(out[:2], (do_l, do_a))
        grads.append({n: (lin[n].grad, att[n].grad) for n in lin})
    for n in "qkv":
        (one_l, one_a), (l, a) = grads[0][n], grads[1][n]
        if n in which:
            assert one_l is one_a and torch.equal(one_l, l + a), n
        else:
            assert torch.equal(one_l, l) and torch.equal(one_a, a), n


@pytest.mark.parametrize("rule,K,V", [("gdn", 64, 64), ("mamba", 128, 64)])
def test_entry_point_that_adds_nothing(rule, K, V, monkeypatch):
    """``natsl_linear_bwd_intra`` is ``natsl_linear_bwd_intra_onto`` with nothing to add to."""
    import neuralattentionsearchlinear_b200 as nat
    from neuralattentionsearchlinear_b200 import _lib
    gen, call, names = torch.Generator().manual_seed(5), _lib.call, []
    rnd = lambda *s: torch.randn(*s, generator=gen).cuda()
    base, attn = ([rnd(1, 200, 2, d).bfloat16() for d in (K, K, V)] for _ in range(2))
    g, beta = -torch.nn.functional.softplus(rnd(1, 200, 2)), rnd(1, 200, 2).sigmoid().bfloat16()
    types, do = (rnd(1, 4, 2, 2) > 0).float(), rnd(1, 200, 2, V).bfloat16()

    def other(name, *args):
        if name == "natsl_linear_bwd_intra_onto":
            assert args[-2] == 0
            names.append(name)
            return call("natsl_linear_bwd_intra", *args[:-2], args[-1])
        return call(name, *args)

    got = []
    for route in (call, other):
        monkeypatch.setattr(_lib, "call", route)
        lin = [t.clone().requires_grad_() for t in base]
        op = nat.nats_mixed_attn_gdn if rule == "gdn" else nat.nats_mixed_attn_mamba
        out = op(*attn, *lin, None, g, *((beta,) if rule == "gdn" else ()), types, None, nats_block_size=64, ops_for_incomplete_chunks="all")
        out[0].backward(do)
        got.append([t.grad for t in lin])
    assert names and all(torch.equal(a, b) for a, b in zip(*got))
