"""GPU test (-m gpu) of what the ops, the layers and the cache refuse or leave to their general paths, and of calls whose
results must not depend on the path that serves them."""
import pytest
import torch

from oracle import tables as otab
from tests.helpers import synth_gdn_inputs, synth_mamba_inputs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nat():
    import neuralattentionsearchlinear_b200 as n
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    return n


def op_inputs(rule, B, T, H, K, V, nbs, dtype=torch.bfloat16, seed=0):
    """(positional arguments up to the decays and betas, 0/1 block types with the last one forced, its own types)"""
    if rule == "gdn":
        q, k, v, g, beta, _ = (x.cuda() for x in synth_gdn_inputs(B, T, H, K, V, seed=seed, dtype=dtype))
        args = (q, k, v, q, k, v, None, g, beta)
    else:
        q, k, v, g, _ = (x.cuda() for x in synth_mamba_inputs(B, T, H, K, V, seed=seed, dtype=dtype))
        args = (q, k, v, q, k, v, None, g)
    raw = otab.synth_types(B, -(-T // nbs), H, 0.5, seed=seed, force_last=False)
    return args, otab.force_last_block(raw.clone()).cuda(), raw[:, -1].cuda()


@pytest.mark.parametrize("rule,K,V", [("gdn", 64, 64), ("mamba", 128, 64)])
@pytest.mark.parametrize("T", [100, 128])
@pytest.mark.parametrize("want", [False, True])
def test_chunk_inference_refuses_fp32(nat, rule, K, V, T, want):
    """The fp32 recurrence has no block-start state for a decoder: the op raises, with and without states asked for."""
    args, types, last = op_inputs(rule, 2, T, 2, K, V, 64, dtype=torch.float32)
    op, key = ((nat.nats_mixed_attn_gdn_chunk_inference, "output_final_state_gated_delta") if rule == "gdn" else
               (nat.nats_mixed_attn_mamba_chunk_inference, "output_final_state_mamba"))
    with pytest.raises(TypeError):
        op(*args, types, last, None, nats_block_size=64, ops_for_incomplete_chunks="all", **{key: want})


@pytest.mark.parametrize("rule", ["gdn", "mamba"])
@pytest.mark.parametrize("what", ["last types", "initial state"])
def test_host_tensors_raise(nat, rule, what):
    """Tensors in host memory never reach a kernel by address."""
    K, V = (64, 64) if rule == "gdn" else (128, 64)
    args, types, last = op_inputs(rule, 2, 128, 2, K, V, 64)
    op, key = ((nat.nats_mixed_attn_gdn_chunk_inference, "output_final_state_gated_delta") if rule == "gdn" else
               (nat.nats_mixed_attn_mamba_chunk_inference, "output_final_state_mamba"))
    if what == "last types":
        last = last.cpu()
    else:
        args = (*args[:6], torch.zeros(2, 2, K, V), *args[7:])
    with pytest.raises(ValueError):
        op(*args, types, last, None, nats_block_size=64, ops_for_incomplete_chunks="all", **{key: True})


# ------------------------------------------------------------------------------------------------ layers and their caches
def make_layer(nat, rule="gdn", **kw):
    cls = nat.NeuralAttentionSearchLinearAttnGDN if rule == "gdn" else nat.NeuralAttentionSearchLinearAttnMamba
    args = dict(hidden_size=256, expand_v=1, head_dim=64, num_heads=4, num_attn_heads=4, ops_for_incomplete_chunks="all",
                layer_idx=0, norm_eps=1e-6)
    if rule == "mamba":
        args.update(head_dim=128, expand_v=0.5)
    args.update(kw)
    torch.manual_seed(3)
    return cls(**args).cuda().bfloat16().eval()


def call(layer, x, cache=None):
    if hasattr(layer, "b_proj"):
        return layer(x, past_key_values=cache)[0]
    return layer(x, cache_params=cache)


def tokens(B, T, hidden=256, seed=0):
    return torch.randn(B, T, hidden, generator=torch.Generator().manual_seed(seed)).bfloat16().cuda()


@pytest.mark.parametrize("rule", ["gdn", "mamba"])
def test_token_of_another_width_raises(nat, rule):
    """The first token and every later one: a wrong width raises and leaves the cache as it was."""
    layer, x = make_layer(nat, rule), tokens(2, 72)
    with torch.no_grad():
        cache = nat.NAtSCache()
        call(layer, x[:, :70], cache)
        for t in (70, 71):
            state = cache[0].state.clone()
            for hidden in (128, 320):
                with pytest.raises(RuntimeError):
                    call(layer, tokens(2, 1, hidden), cache)
            assert cache[0].n_tokens == t and torch.equal(cache[0].state, state)
            call(layer, x[:, t:t + 1], cache)
    assert cache[0].n_tokens == 72


def shift(t):
    """The same values in a tensor that starts one element behind a 16-byte boundary."""
    buf = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    out = buf[1:].view(t.shape)
    out.copy_(t.detach())
    assert out.data_ptr() % 16 == t.element_size()
    return out


def prompt_and_tokens(nat, layer, x, T):
    cache = nat.NAtSCache()
    with torch.no_grad():
        ys = [call(layer, x[:, :T].contiguous(), cache)] + [call(layer, x[:, t:t + 1], cache) for t in range(T, x.shape[1])]
    return torch.cat(ys, 1)


@pytest.mark.parametrize("rule,name", [("gdn", n) for n in ("q_proj", "a_proj", "b_proj", "o_proj", "nats_out_weights_layer", "k_conv1d")]
                         + [("mamba", n) for n in ("v_proj", "g_proj", "v_conv1d")])
def test_unaligned_parameters_take_the_general_path(nat, rule, name, monkeypatch):
    """Views into a flat buffer: the fast paths decline them and the results are the general path's."""
    from neuralattentionsearchlinear_b200 import natsl_attn_gdn, natsl_attn_mamba2
    from neuralattentionsearchlinear_b200.decode_step import layer_plan
    layer, x = make_layer(nat, rule), tokens(2, 130)
    m = getattr(layer, name)
    m.weight.data = shift(m.weight)
    assert not layer_plan(layer).ok
    got = prompt_and_tokens(nat, layer, x, 126)
    for mod in (natsl_attn_gdn, natsl_attn_mamba2):
        monkeypatch.setattr(mod, "layer_forward", lambda *a: None)
        monkeypatch.setattr(mod, "decode_token", lambda *a: None)
    assert torch.equal(got, prompt_and_tokens(nat, layer, x, 126))


@pytest.mark.parametrize("rule", ["gdn", "mamba"])
def test_unaligned_inputs(nat, rule):
    """Prompt, tokens and initial state of any address give what aligned ones give."""
    layer, x = make_layer(nat, rule), tokens(1, 130)
    with torch.no_grad():
        a, b = nat.NAtSCache(), nat.NAtSCache()
        assert torch.equal(call(layer, x[:, :128], a), call(layer, shift(x[:, :128]), b))
        for t in (128, 129):
            assert torch.equal(call(layer, x[:, t:t + 1].contiguous(), a), call(layer, shift(x[:, t:t + 1]), b))
        K, V = (64, 64) if rule == "gdn" else (128, 64)
        args, types, _ = op_inputs(rule, 1, 100, 2, K, V, 64)
        h0 = torch.randn(1, 2, K, V, device="cuda")
        op = nat.nats_mixed_attn_gdn if rule == "gdn" else nat.nats_mixed_attn_mamba
        run = lambda h: op(*args[:6], h, *args[7:], types, None, nats_block_size=64, ops_for_incomplete_chunks="all")[0]
        assert torch.equal(run(h0), run(shift(h0)))


def test_entry_points_refuse_unaligned_pointers(nat):
    """The library itself: an error code before any launch."""
    import ctypes

    from neuralattentionsearchlinear_b200 import _lib
    layer, x = make_layer(nat), tokens(1, 66)
    cache = nat.NAtSCache()
    with torch.no_grad():
        call(layer, x[:, :64], cache)
        call(layer, x[:, 64:65], cache)
    st = torch.cuda.current_stream().cuda_stream
    args = cache[0]._step.args
    for field in ("x", "w_q", "w_mix", "cw_v", "state", "k_cache"):
        bad = _lib.DecodeArgs()
        ctypes.memmove(ctypes.byref(bad), ctypes.byref(args), ctypes.sizeof(bad))
        bad.pos, bad.types_new = 65, None
        setattr(bad, field, getattr(bad, field) + 2)
        with pytest.raises(_lib.NatslError, match="start on 16 bytes"):
            _lib.call("natsl_decode_step", ctypes.byref(bad), st)


# ------------------------------------------------------------------------------------------------ the current device
@pytest.mark.parametrize("what", ["gdn op", "mamba op", "fp32 op", "prompt", "token"])
def test_work_runs_with_the_tensors_device_current(nat, what, monkeypatch):
    """With another device current, the op and the layers switch to the tensors' device around their launches."""
    layer, x = make_layer(nat), tokens(1, 66)
    cache = nat.NAtSCache()
    with torch.no_grad():
        call(layer, x[:, :64], cache)
    args, types, _ = op_inputs("mamba" if what == "mamba op" else "gdn", 1, 64, 2, 128 if what == "mamba op" else 64, 64, 64,
                               dtype=torch.float32 if what == "fp32 op" else torch.bfloat16)
    op = nat.nats_mixed_attn_mamba if what == "mamba op" else nat.nats_mixed_attn_gdn
    entered = []

    class Guard:
        def __init__(self, device):
            self.index = torch.device(device).index if not isinstance(device, int) else device

        def __enter__(self):
            entered.append(self.index)

        def __exit__(self, *exc):
            pass

    from neuralattentionsearchlinear_b200 import nats_util
    monkeypatch.setattr(nats_util, "current_device", lambda: 1)
    monkeypatch.setattr(torch.cuda, "device", Guard)
    with torch.no_grad():
        if what == "prompt":
            call(layer, x[:, :64])
        elif what == "token":
            call(layer, x[:, 64:65], cache)
        else:
            op(*args, types, None, nats_block_size=64, ops_for_incomplete_chunks="all")
    assert entered and set(entered) == {0}


def test_library_refuses_memory_of_another_place(nat):
    """A host address in place of a tensor of the current device: an error code before any launch."""
    import ctypes

    from neuralattentionsearchlinear_b200 import _lib
    layer, x = make_layer(nat), tokens(1, 66)
    cache = nat.NAtSCache()
    with torch.no_grad():
        call(layer, x[:, :64], cache)
        call(layer, x[:, 64:65], cache)
    bad = _lib.DecodeArgs()
    ctypes.memmove(ctypes.byref(bad), ctypes.byref(cache[0]._step.args), ctypes.sizeof(bad))
    host = torch.zeros(256, dtype=torch.bfloat16, pin_memory=True)
    bad.pos, bad.types_new, bad.x = 65, None, host.data_ptr()
    with pytest.raises(_lib.NatslError, match="device memory"):
        _lib.call("natsl_decode_step", ctypes.byref(bad), torch.cuda.current_stream().cuda_stream)


# ------------------------------------------------------------------------------------------------ changed layers
# Both paths round the same tensors to bf16 and differ in the order of fp32 sums: 2^-8 of the largest entry for each of about
# four roundings that do not cancel (as in tests/test_gpu_decode_step.py).
TOL = 4 * 2.0 ** -8


def general_path(monkeypatch):
    from neuralattentionsearchlinear_b200 import natsl_attn_gdn, natsl_attn_mamba2
    for mod in (natsl_attn_gdn, natsl_attn_mamba2):
        monkeypatch.setattr(mod, "layer_forward", lambda *a: None)
        monkeypatch.setattr(mod, "decode_token", lambda *a: None)


def close(got, want, what):
    bound = TOL * max(float(want.float().abs().max()), 1e-3)
    err = float((got.float() - want.float()).abs().max())
    assert err <= bound, f"{what} off by {err:.3g} (bound {bound:.3g})"


def set_conv(layer, activation):
    for c in (layer.q_conv1d, layer.k_conv1d, layer.v_conv1d):
        c.activation = activation


def scaled_mix(layer):
    mix = layer.mix
    layer.mix = lambda *a: 2 * mix(*a)


CHANGES = [
    ("gdn", "block size", lambda m: setattr(m, "nats_block_size", 128)),
    ("gdn", "q/k norm eps", lambda m: [setattr(n, "eps", 3.0) for n in (m.q_norm, m.k_norm)]),
    ("gdn", "output norm eps", lambda m: setattr(m.o_norm, "eps", 3.0)),
    ("gdn", "gate activation", lambda m: setattr(m.o_norm, "activation", "sigmoid")),
    ("gdn", "convolution activation", lambda m: set_conv(m, None)),
    ("gdn", "negative eigenvalues", lambda m: setattr(m, "allow_neg_eigval", True)),
    ("gdn", "decay over skipped blocks", lambda m: setattr(m, "decay_for_non_gdn_blocks", False)),
    ("gdn", "own chunk", lambda m: setattr(m, "ops_for_incomplete_chunks", "gated_delta_net")),
    ("gdn", "another mix", scaled_mix),
    ("mamba", "l2 norm eps", lambda m: [setattr(n, "eps", 3.0) for n in (m.q_norm2, m.k_norm2)]),
    ("mamba", "decay over skipped blocks", lambda m: setattr(m, "decay_for_non_mamba_blocks", False)),
]


@pytest.mark.parametrize("rule,what,change", CHANGES, ids=[f"{r}-{w}" for r, w, _ in CHANGES])
def test_changed_attributes_take_effect(nat, rule, what, change, monkeypatch):
    """An attribute changed after the first calls counts from the next call on: prompt, and tokens of a cache in use."""
    layer, x = make_layer(nat, rule), tokens(2, 140)

    def run():
        cache = nat.NAtSCache()
        with torch.no_grad():
            y = [call(layer, x[:, :120], cache), call(layer, x[:, 120:121], cache)]
            old = {n: getattr(layer, n) for n in ("nats_block_size", "ops_for_incomplete_chunks")}
            if what == "block size":                         # of a new sequence: a cache keeps the one it was begun with
                cache = nat.NAtSCache()
                layer.nats_block_size = 128
                y += [call(layer, x[:, :130], cache)]
                t0 = 130
            else:
                undo = {m: dict(m.__dict__) for m in layer.modules()}
                change(layer)
                t0 = 121
            y += [call(layer, x[:, t:t + 1], cache) for t in range(t0, 140)] + [call(layer, x[:, :120])]
            if what == "block size":
                for n, v in old.items():
                    setattr(layer, n, v)
            else:
                for m, d in undo.items():
                    for n in ("eps", "activation", "allow_neg_eigval", "decay_for_non_gdn_blocks", "decay_for_non_mamba_blocks",
                              "ops_for_incomplete_chunks"):
                        if n in d:
                            setattr(m, n, d[n])
                layer.__dict__.pop("mix", None)
        return y

    got = run()
    general_path(monkeypatch)
    for i, (a, b) in enumerate(zip(got, run())):
        close(a, b, f"call {i}")


@pytest.mark.parametrize("rule,name", [("gdn", "b_proj"), ("gdn", "nats_out_weights_layer"), ("mamba", "nats_out_weights_layer"),
                                       ("gdn", "q_proj"), ("gdn", "nats_layer")])
@pytest.mark.parametrize("replaced", [False, True])
def test_projections_with_a_bias(nat, rule, name, replaced, monkeypatch):
    """A projection that has got a bias (another module, or the same one given a bias) takes the general path."""
    layer, x = make_layer(nat, rule), tokens(2, 140)
    got = [prompt_and_tokens(nat, layer, x, 130)]
    old = getattr(layer, name)
    m = torch.nn.Linear(old.in_features, old.out_features, bias=True).cuda().bfloat16() if replaced else old
    m.weight.data.copy_(old.weight.data)
    m.bias = torch.nn.Parameter(torch.linspace(-2, 2, old.out_features, device="cuda").bfloat16())
    setattr(layer, name, m)
    got.append(prompt_and_tokens(nat, layer, x, 130))
    general_path(monkeypatch)
    want = prompt_and_tokens(nat, layer, x, 130)
    close(got[1], want, "with the bias")
    assert float((got[0] - want).abs().max()) > TOL * float(want.abs().max()), "the bias makes no difference here"


@pytest.mark.parametrize("what", ["wider output", "narrower projection", "missing", "transposed", "other dtype"])
def test_replaced_weights(nat, what):
    """Weights of other shapes, layouts or types than the plan was made for: the fast paths see it before any launch."""
    from neuralattentionsearchlinear_b200.decode_step import layer_plan
    layer, x = make_layer(nat), tokens(2, 130)
    prompt_and_tokens(nat, layer, x, 128)
    assert layer_plan(layer).ok
    if what == "wider output":                               # the general path serves it: another width out
        layer.o_proj = torch.nn.Linear(256, 320, bias=False).cuda().bfloat16()
        want = layer.o_proj.weight
        assert not layer_plan(layer).ok
        y = prompt_and_tokens(nat, layer, x, 128)
        assert y.shape[-1] == want.shape[0] and bool(y.isfinite().all())
    elif what == "narrower projection":
        layer.k_proj.weight.data = layer.k_proj.weight.data[:192]
        assert not layer_plan(layer).ok
    elif what == "missing":
        w = layer.a_proj.weight.data
        del layer.a_proj.weight
        layer.a_proj.weight = w                              # a plain attribute in place of the parameter
        assert not layer_plan(layer).ok
        assert bool(prompt_and_tokens(nat, layer, x, 128).isfinite().all())
    elif what == "transposed":
        layer.q_proj.weight.data = layer.q_proj.weight.data.t()
        assert not layer_plan(layer).ok
    else:
        layer.v_proj.weight.data = layer.v_proj.weight.data.view(torch.float16)
        assert not layer_plan(layer).ok


# ------------------------------------------------------------------------------------------------ what a caller keeps of a cache
CACHE_STATE = ("state", "state_block_start", "g_block", "pool_sum", "conv_state", "k_attn", "v_attn", "block_types", "n_tokens")


@pytest.mark.parametrize("rule", ["gdn", "mamba"])
@pytest.mark.parametrize("T0", [70, 126])
def test_snapshot_of_a_cache_by_reference(nat, rule, T0):
    """Tensors read from a cache stay as they are while it decodes on (also over a block's end), and setting them again takes
    it back to that token."""
    layer, x = make_layer(nat, rule), tokens(2, 140)
    cache = nat.NAtSCache()
    with torch.no_grad():
        call(layer, x[:, :T0], cache)
        call(layer, x[:, T0:T0 + 1], cache)
        snap = {n: getattr(cache[0], n) for n in CACHE_STATE}
        flat = lambda: [t for n in CACHE_STATE[:-1] for t in (snap[n] if n == "conv_state" else [snap[n]])]
        values = [t.clone() for t in flat()]
        first = [call(layer, x[:, t:t + 1], cache) for t in range(T0 + 1, T0 + 5)]
        assert all(map(torch.equal, flat(), values))
        for n in CACHE_STATE:
            setattr(cache[0], n, snap[n])
        again = [call(layer, x[:, t:t + 1], cache) for t in range(T0 + 1, T0 + 5)]
        assert all(map(torch.equal, flat(), values))
    assert all(map(torch.equal, first, again))


@pytest.mark.parametrize("what", ["state storage", "types storage", "state shape", "tail shape", "key shape", "types shape"])
def test_cache_tensors_of_other_storage_or_shape(nat, what):
    """Storage exchanged behind a tensor is what the next step reads; shapes of another layer never reach the kernel."""
    layer, x = make_layer(nat), tokens(2, 140)
    with torch.no_grad():
        cache, other = nat.NAtSCache(), nat.NAtSCache()
        call(layer, x[:, :70], cache)
        call(layer, x[:, :70].flip(0).contiguous(), other)
        for c in (cache, other):
            call(layer, x[:, 70:71], c)
        c, o = cache[0], other[0]
        if what.endswith("storage"):
            if what == "state storage":
                c.state.data = o.state.data.clone()
                c.state_block_start.data = o.state_block_start.data.clone()
            else:
                c.block_types.data = 1 - c.block_types.data
            import copy
            new = nat.NAtSCache()
            new.layers = [copy.copy(c)]
            assert torch.equal(call(layer, x[:, 71:72], cache), call(layer, x[:, 71:72], new))
            return
        if what == "state shape":
            c.state = c.state[:, :, :32]
        elif what == "tail shape":
            c.conv_state = tuple(t[:, :128].contiguous() for t in c.conv_state)
        elif what == "key shape":
            c.k_attn = c.k_attn[..., :32].contiguous()
        else:
            c.block_types = c.block_types[:, :, :2].contiguous()
        from neuralattentionsearchlinear_b200.decode_step import decode_token
        assert decode_token(layer, x[:, 71:72], cache) is None


# ------------------------------------------------------------------------------------------------ transforms and traces
def op_call(nat, rule):
    op = nat.nats_mixed_attn_gdn if rule == "gdn" else nat.nats_mixed_attn_mamba
    return lambda args, types: op(*args, types, None, nats_block_size=64, ops_for_incomplete_chunks="all")[:2]


@pytest.mark.parametrize("rule", ["gdn", "mamba"])
@pytest.mark.parametrize("level", ["forward_ad", "jvp", "vmap"])
def test_op_under_a_transform_raises(nat, rule, level):
    """The ops have no forward-mode or batching rule: they raise, with and without reverse mode on, and never drop a tangent."""
    import torch.autograd.forward_ad as fwad
    run = op_call(nat, rule)
    args, types, _ = op_inputs(rule, 2, 128, 2, 64 if rule == "gdn" else 128, 64, 64)
    with_q = lambda q: run((q, *args[1:3], q, *args[4:]), types)
    for grad in (True, False):
        with torch.set_grad_enabled(grad), pytest.raises((NotImplementedError, RuntimeError)):
            if level == "forward_ad":
                with fwad.dual_level():
                    with_q(fwad.make_dual(args[0], torch.ones_like(args[0])))
            elif level == "jvp":
                torch.func.jvp(with_q, (args[0],), (torch.ones_like(args[0]),))
            else:
                torch.func.vmap(with_q)(args[0][None])
    run(args, types)


@pytest.mark.parametrize("rule", ["gdn", "mamba"])
@pytest.mark.parametrize("what", ["prompt", "token"])
def test_layer_under_forward_mode_raises(nat, rule, what):
    import torch.autograd.forward_ad as fwad
    layer, x = make_layer(nat, rule), tokens(1, 66)
    cache = nat.NAtSCache()
    with torch.no_grad():
        call(layer, x[:, :65], cache)
        with fwad.dual_level(), pytest.raises(NotImplementedError):
            piece = x[:, :64] if what == "prompt" else x[:, 65:]
            call(layer, fwad.make_dual(piece, torch.ones_like(piece)), None if what == "prompt" else cache)


@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning")
@pytest.mark.parametrize("rule", ["gdn", "mamba"])
def test_traced_op_computes_with_new_inputs(nat, rule):
    """A jit trace replays the op on other inputs: nothing of the traced call is frozen into it."""
    run, K = op_call(nat, rule), 64 if rule == "gdn" else 128
    (a, types, _), (b, _, _) = op_inputs(rule, 1, 128, 2, K, 64, 64), op_inputs(rule, 1, 128, 2, K, 64, 64, seed=1)
    fn = lambda q, k, v: run((q, k, v, q, k, v, *a[6:]), types)
    with torch.no_grad():
        traced = torch.jit.trace(fn, a[:3], check_trace=False)
        for got, want in zip(traced(*b[:3]), fn(*b[:3])):
            close(got, want, rule)


# ------------------------------------------------------------------------------------------------ threads and streams
def in_thread(fn):
    """Runs fn in a thread of its own; returns its result or raises what it raised."""
    import threading
    box = {}

    def target():
        try:
            box["result"] = fn()
        except BaseException as e:
            box["error"] = e

    t = threading.Thread(target=target)
    t.start()
    t.join(60)
    assert not t.is_alive()
    if "error" in box:
        raise box["error"]
    return box["result"]


@pytest.mark.parametrize("what", ["gdn op", "mamba op", "fp32 op", "layer"])
def test_a_capture_takes_no_work_of_another_thread(nat, what):
    """While one thread captures a call into a graph, another thread's call runs at once and stays out of it."""
    rule, K = ("mamba", 128) if what == "mamba op" else ("gdn", 64)
    if what == "layer":
        layer, a, b = make_layer(nat), tokens(1, 128), tokens(1, 128, seed=1)
        run = lambda x: call(layer, x)
    else:
        dtype = torch.float32 if what == "fp32 op" else torch.bfloat16
        (a, types, _), (b, _, _) = (op_inputs(rule, 1, 128, 2, K, 64, 64, dtype=dtype, seed=s) for s in (0, 1))
        run = lambda args: op_call(nat, rule)(args, types)[0]

    def eager(x):
        with torch.no_grad(), torch.cuda.stream(torch.cuda.Stream()):
            y = run(x)
            torch.cuda.current_stream().synchronize()
        return y

    want_a, want_b = eager(a), in_thread(lambda: eager(b))
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.no_grad(), torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        y = run(a)
        got_b = in_thread(lambda: eager(b))
        y2 = run(a)
    assert torch.equal(got_b, want_b)
    y.zero_(), y2.zero_()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want_a) and torch.equal(y2, want_a)


def test_threads_on_their_own_streams(nat):
    """Calls of four threads at once give what they give alone."""
    import concurrent.futures as cf
    inputs = [op_inputs("gdn", 2, 300, 2, 64, 64, 64, seed=s) for s in range(4)]
    run = op_call(nat, "gdn")

    def work(i):
        with torch.no_grad(), torch.cuda.stream(torch.cuda.Stream()):
            ys = [run(inputs[i][0], inputs[i][1]) for _ in range(20)]
            torch.cuda.current_stream().synchronize()
        return ys

    torch.cuda.synchronize()
    alone = [work(i)[0] for i in range(4)]
    with cf.ThreadPoolExecutor(4) as pool:
        for want, ys in zip(alone, pool.map(work, range(4))):
            for y in ys:
                assert all(map(torch.equal, y, want))


# ------------------------------------------------------------------------------------------------ switches
def kernels_of(fn):
    from torch.profiler import ProfilerActivity, profile
    fn()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    return [e.name for e in p.events()]


@pytest.mark.parametrize("what", ["op", "layer"])
def test_split_walk_switch_reaches_the_op(nat, what, monkeypatch):
    """WALK_VSPLIT runs the walk with the value dimension split, with the results of the walk it stands in for."""
    from neuralattentionsearchlinear_b200 import _ops
    monkeypatch.setattr(_ops, "WALK_MMA_MAX_HEADS", 0)
    if what == "op":
        args, types, _ = op_inputs("gdn", 2, 300, 2, 128, 128, 64)
        fn = lambda: op_call(nat, "gdn")(args, types)[0]
    else:
        layer, x = make_layer(nat, head_dim=128, num_heads=2, num_attn_heads=2), tokens(2, 300)
        fn = lambda: call(layer, x)
    with torch.no_grad():
        want = fn()
        assert not any("gdn_walk_half_kernel" in k for k in kernels_of(fn))
        monkeypatch.setattr(_ops, "WALK_VSPLIT", True)
        names = kernels_of(fn)
        assert any("gdn_walk_half_kernel" in k for k in names), names
        close(fn(), want, what)


@pytest.mark.parametrize("what", ["gdn op", "mamba op", "fp32 op", "layer"])
def test_priority_switch_moves_the_linear_branch(nat, what, monkeypatch):
    """LINEAR_BRANCH_PRIORITY: on, the linear branch leaves the caller's stream; off, the softmax branch does.  Same results."""
    from torch.profiler import ProfilerActivity, profile

    from neuralattentionsearchlinear_b200 import _ops
    if what == "layer":
        layer, x = make_layer(nat), tokens(2, 300)
        fn = lambda: call(layer, x)
    else:
        rule, K = ("mamba", 128) if what == "mamba op" else ("gdn", 64)
        args, types, _ = op_inputs(rule, 2, 300, 2, K, 64, 64, dtype=torch.float32 if what == "fp32 op" else torch.bfloat16)
        fn = lambda: op_call(nat, rule)(args, types)[0]
    mark, outs, linear = torch.zeros(256, device="cuda"), [], "linear_recurrent" if what == "fp32 op" else "walk"
    for high in (True, False):
        monkeypatch.setattr(_ops, "LINEAR_BRANCH_PRIORITY", high)
        with torch.no_grad():
            outs.append(fn())
            with profile(activities=[ProfilerActivity.CUDA]) as p:
                mark.add_(1)
                fn()
                torch.cuda.synchronize()
        stream = {k: {e.device_resource_id for e in p.events() if k in e.name} for k in (linear, "attn", "elementwise")}
        caller = min(stream["elementwise"], default=None)
        assert caller is not None and stream["attn" if high else linear] == {caller}, stream
        assert caller not in stream[linear if high else "attn"], stream
    assert torch.equal(*outs)


@pytest.mark.parametrize("what", ["gdn op", "mamba op", "fp32 op", "layer", "layer with cache", "mamba layer"])
def test_launch_accounting(nat, what):
    """kernel_launches() grows by the kernels of this library that a call runs."""
    from neuralattentionsearchlinear_b200 import _lib
    if "layer" in what:
        layer, x = make_layer(nat, "mamba" if "mamba" in what else "gdn"), tokens(2, 300)
        fn = lambda: call(layer, x, nat.NAtSCache() if "cache" in what else None)
    else:
        rule, K = ("mamba", 128) if what == "mamba op" else ("gdn", 64)
        args, types, _ = op_inputs(rule, 2, 300, 2, K, 64, 64, dtype=torch.float32 if what == "fp32 op" else torch.bfloat16)
        fn = lambda: op_call(nat, rule)(args, types)
    with torch.no_grad():
        ran = [n for n in kernels_of(fn) if "natsl::" in n]
        before = _lib.kernel_launches()
        fn()
    assert _lib.kernel_launches() - before == len(ran), ran
