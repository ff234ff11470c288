"""Timing cases of the framework: what its users have it do, through its public entry points.

Five kinds of work, each over the range of sizes that its users meet:

* ``op``       the hybrid attention ops on projected tensors (GDN and Mamba2), forward, or forward and backward;
* ``long``     the long-context Mamba2 op whose recurrence is cut into sub-segments (batch 1, one GPU);
* ``layer``    a whole NAtSL layer under eval on one prompt batch (projections, selection, both branches, mixing);
* ``request``  a layer serving one batch of requests: prefill into a cache, then token by token;
* ``train``    one training step of a decoder block or of a Mamba2 layer: forward and backward, every gradient.

Layer shapes are the configurations the repository's benchmark and tests name (16 heads of 64 or of 128; the shipped
340M shape with 6 heads of 128 / 256 and 12 softmax heads; the 760M head dims 192 / 384; Mamba2 with state dim 128 and
head dim 64).
"""
import math

import torch

import neuralattentionsearchlinear_b200 as nat
from neuralattentionsearchlinear_b200.models import (NeuralAttentionSearchLinearAttnGDNBlock,
                                                     NeuralAttentionSearchLineraAttnGDNConfig)
from neuralattentionsearchlinear_b200.sequence_parallel import nats_mixed_attn_mamba_sp

C = 64                                                    # tokens of a compute chunk

# hidden size, heads, head dim, expand_v, softmax heads
SHAPES = {
    "gdn_16x64": dict(rule="gdn", hidden=1024, heads=16, head_dim=64, expand_v=1.0, attn_heads=16),
    "gdn_16x128": dict(rule="gdn", hidden=2048, heads=16, head_dim=128, expand_v=1.0, attn_heads=16),
    "gdn_340m": dict(rule="gdn", hidden=1024, heads=6, head_dim=128, expand_v=2.0, attn_heads=12),
    "mamba_16x128": dict(rule="mamba", hidden=1024, heads=16, head_dim=128, expand_v=0.5, attn_heads=16),
    "mamba_32x128": dict(rule="mamba", hidden=2048, heads=32, head_dim=128, expand_v=0.5, attn_heads=32),
}


def listed():
    return [
        # the repository's headline benchmark: one layer's hybrid op on a prefill batch
        dict(name="op_prefill_8x4096_16x128", kind="op", rule="gdn", B=8, T=4096, H=16, HQ=16, K=128, V=128, nbs=64,
             p=0.25, dtype="bf16", train=False),
        # the same op inside a training step
        dict(name="op_train_8x4096_16x128", kind="op", rule="gdn", B=8, T=4096, H=16, HQ=16, K=128, V=128, nbs=64,
             p=0.25, dtype="bf16", train=True),
        # the op at the 760M configuration's head dims
        dict(name="op_prefill_2x2048_760m", kind="op", rule="gdn", B=2, T=2048, H=6, HQ=18, K=192, V=384, nbs=64,
             p=0.5, dtype="bf16", train=False),
        # reference-precision check runs in fp32: the smallest call
        dict(name="op_fp32_2x512_4x64", kind="op", rule="gdn", B=2, T=512, H=4, HQ=4, K=64, V=64, nbs=64, p=0.5,
             dtype="fp32", train=False),
        # a long document through one Mamba2 layer's op
        dict(name="long_mamba_65536_32x128", kind="long", rule="mamba", B=1, T=65536, H=32, HQ=32, K=128, V=64, nbs=256,
             p=0.1, dtype="bf16", train=False),
        # scoring / embedding a batch with the 24-layer 16x64 model: one of its layers
        dict(name="layer_16x4096_gdn_16x64", kind="layer", shape="gdn_16x64", B=16, T=4096, nbs=64),
        # one short document of odd length through a layer of the shipped 340M shape
        dict(name="layer_1x1501_gdn_340m", kind="layer", shape="gdn_340m", B=1, T=1501, nbs=64),
        # one chat request: prompt, then tokens one at a time
        dict(name="request_1x777_gdn_16x128", kind="request", shape="gdn_16x128", B=1, T=777, nbs=64, new=48),
        # a batch of requests with longer prompts
        dict(name="request_32x2048_gdn_16x64", kind="request", shape="gdn_16x64", B=32, T=2048, nbs=64, new=32),
        # a few requests through a Mamba2 layer with blocks of 256 tokens
        dict(name="request_4x1030_mamba_32x128", kind="request", shape="mamba_32x128", B=4, T=1030, nbs=256, new=32),
        # a block of the 1.3B model in its training step (8 sequences of 4096 per GPU)
        dict(name="train_8x4096_gdn_16x128", kind="train", shape="gdn_16x128", B=8, T=4096, nbs=64),
        # a Mamba2 layer in a training step on shorter, ragged sequences
        dict(name="train_4x1000_mamba_16x128", kind="train", shape="mamba_16x128", B=4, T=1000, nbs=64),
    ]


# ---------------------------------------------------------------------------------------------------- drawn cases
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tokens(rng, lo, hi):
    """A sequence length, spread over its logarithm: as often odd as a multiple of the chunk."""
    t = _log_int(rng, lo, hi)
    return max(lo, t // C * C) if rng.random() < 0.5 else t


def _batch(rng, most, T, tokens):
    return max(1, min(_log_int(rng, 1, most), tokens // T))


def draw(rng):
    kind = rng.choice(["op", "op", "op_train", "op_fp32", "long", "layer", "layer", "request", "request", "train"])
    if kind == "long":
        T, H = _log_int(rng, 4096, 65536), rng.choice([16, 32])
        T = T if rng.random() < 0.3 else T // 1024 * 1024
        return dict(kind="long", rule="mamba", B=1, T=T, H=H, HQ=H, K=128, V=64, nbs=rng.choice([64, 128, 256]),
                    p=round(rng.uniform(0.05, 0.1), 3), dtype="bf16", train=False)
    if kind.startswith("op"):
        train, fp32 = kind == "op_train", kind == "op_fp32"
        rule = "gdn" if rng.random() < 0.7 else "mamba"
        if fp32:
            K = V = 64
            H, T, nbs = rng.choice([2, 4, 8]), _tokens(rng, 64, 768), 64
            HQ, B = H, rng.choice([1, 2])
        elif train:
            K, V = (rng.choice([(64, 64), (128, 128)]) if rule == "gdn" else (128, 64))
            H, T, nbs = rng.choice([4, 8, 16]), _tokens(rng, 64, 4096), 64
            HQ, B = H, _batch(rng, 8, T, 32768)
        else:
            K, V, r = (rng.choice([(64, 64, 1), (128, 128, 1), (128, 256, 2), (192, 384, 3)]) if rule == "gdn" else (128, 64, 1))
            wide = K == 192
            H = 6 if r > 1 else rng.choice([4, 8, 16])
            T, nbs = _tokens(rng, 64, 2048 if wide else 4096), rng.choice([64, 64, 128, 256])
            HQ, B = H * r, _batch(rng, 8, T, 4096 if wide else 32768)
        return dict(kind="op", rule=rule, B=B, T=T, H=H, HQ=HQ, K=K, V=V, nbs=nbs, p=round(rng.uniform(0.1, 0.6), 3),
                    dtype="fp32" if fp32 else "bf16", train=train)
    if kind == "layer":
        shape, T = rng.choice(sorted(SHAPES)), _tokens(rng, 64, 4096)
        return dict(kind="layer", shape=shape, B=_batch(rng, 16, T, 32768), T=T, nbs=_blocks(rng, shape))
    if kind == "request":
        shape, T = rng.choice(sorted(SHAPES)), _tokens(rng, 64, 4096)
        return dict(kind="request", shape=shape, B=_batch(rng, 32, T, 32768), T=T, nbs=_blocks(rng, shape),
                    new=rng.randint(8, 64))
    shape, T = rng.choice(["gdn_16x64", "gdn_16x128", "mamba_16x128", "mamba_32x128"]), _tokens(rng, 128, 4096)
    return dict(kind="train", shape=shape, B=_batch(rng, 8, T, 32768), T=T, nbs=64)


def _blocks(rng, shape):
    return 64 if SHAPES[shape]["rule"] == "gdn" else rng.choice([64, 128, 256])


# ---------------------------------------------------------------------------------------------------- inputs
def _types(B, TN, HN, p, gen):
    """0/1 block types: argmax of two normal logits, shifted so that a share p takes the softmax branch; last block both."""
    logits = torch.randn(B, TN, HN, 2, generator=gen, device="cuda")
    logits[..., 0] += math.sqrt(2.0) * torch.distributions.Normal(0.0, 1.0).icdf(torch.tensor(p)).item()
    types = torch.zeros_like(logits).scatter_(-1, logits.argmax(-1, keepdim=True), 1.0)
    types[:, -1] = 1
    return types


def _prepare_op(case, gen):
    B, T, H, K, V, nbs = (case[n] for n in ("B", "T", "H", "K", "V", "nbs"))
    HQ = case["HQ"]
    dt = torch.float32 if case["dtype"] == "fp32" else torch.bfloat16
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    unit = lambda x: torch.nn.functional.normalize(x, dim=-1)
    x = dict(types=_types(B, -(-T // nbs), H, case["p"], gen))
    if case["rule"] == "gdn":
        x.update(q=unit(rnd(B, T, H, K)).to(dt), k=unit(rnd(B, T, H, K)).to(dt), v=rnd(B, T, H, V).to(dt),
                 beta=rnd(B, T, H).sigmoid().to(dt), g=-torch.nn.functional.softplus(rnd(B, T, H)))
    else:
        step = torch.nn.functional.softplus(rnd(B, T, H) - 2.0)
        A = -torch.exp(torch.rand(H, generator=gen, device="cuda") * math.log(16.0))
        x.update(q=(rnd(B, T, H, K) * K ** -0.5).to(dt), k=(rnd(B, T, H, K) * K ** -0.5).to(dt),
                 v=(rnd(B, T, H, V) * step[..., None]).to(dt), g=A * step)
    if HQ == H:                                           # the softmax branch reads the same projections
        x.update(qa=x["q"], ka=x["k"], va=x["v"])
    else:                                                 # same widths, split into more heads
        x.update(qa=rnd(B, T, HQ, H * K // HQ).to(dt), ka=rnd(B, T, HQ, H * K // HQ).to(dt), va=x["v"].view(B, T, HQ, -1))
    if case["train"]:
        names = ("q", "k", "v", "g", "types") + (("beta",) if "beta" in x else ())
        for n in names:
            x[n].requires_grad_(True)
        x.update(do_l=rnd(B, T, H, V).to(dt), do_a=rnd(B, T, HQ, H * V // HQ).to(dt), leaves=names)
    return x


def _layer(case):
    s = SHAPES[case["shape"]]
    common = dict(hidden_size=s["hidden"], expand_v=s["expand_v"], head_dim=s["head_dim"], num_heads=s["heads"],
                  num_attn_heads=s["attn_heads"], nats_block_size=case["nbs"], ops_for_incomplete_chunks="all",
                  layer_idx=0, norm_eps=1e-6)
    if s["rule"] == "mamba":
        return nat.NeuralAttentionSearchLinearAttnMamba(**common)
    return nat.NeuralAttentionSearchLinearAttnGDN(attn_qk_norm=True, attn_with_short_conv=True,
                                                  decay_for_non_gdn_blocks=True, **common)


def _block(case):
    s = SHAPES[case["shape"]]
    return NeuralAttentionSearchLinearAttnGDNBlock(NeuralAttentionSearchLineraAttnGDNConfig(
        hidden_size=s["hidden"], expand_v=s["expand_v"], head_dim=s["head_dim"], num_heads=s["heads"],
        num_attn_heads=s["attn_heads"], nats_block_size=case["nbs"], ops_for_incomplete_chunks="all",
        attn_apply_pos_encoding=False, attn_qk_norm=True, attn_with_short_conv=True, decay_for_non_gdn_blocks=True,
        norm_eps=1e-6), 0)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    state = dict(case=case)
    if case["kind"] in ("op", "long"):
        state.update(_prepare_op(case, gen))
        return state
    s = SHAPES[case["shape"]]
    torch.manual_seed(seed)
    with torch.device("cuda"):                            # a model whose weights are on the GPU, as after loading
        module = _block(case) if (case["kind"] == "train" and s["rule"] == "gdn") else _layer(case)
    module = module.bfloat16()
    n = case["T"] + case.get("new", 0)
    x = torch.randn(case["B"], n, s["hidden"], generator=gen, device="cuda").bfloat16()
    state.update(module=module, mamba=s["rule"] == "mamba")
    if case["kind"] == "train":
        module.train()
        dy = torch.randn(x.shape, generator=gen, device="cuda").bfloat16()
        state.update(x=x.requires_grad_(True), dy=dy)
    elif case["kind"] == "layer":
        module.eval()
        state.update(x=x)
    else:
        module.eval()
        T = case["T"]
        state.update(prompt=x[:, :T].contiguous(), tokens=[x[:, t:t + 1].contiguous() for t in range(T, n)])
    return state


# ---------------------------------------------------------------------------------------------------- one pass
def _op(s):
    c = s["case"]
    if c["rule"] == "gdn":
        return nat.nats_mixed_attn_gdn(s["qa"], s["ka"], s["va"], s["q"], s["k"], s["v"], None, s["g"], s["beta"],
                                       s["types"], None, nats_block_size=c["nbs"], ops_for_incomplete_chunks="all",
                                       output_final_state_gated_delta=not c["train"], decay_for_non_gdn_blocks=True)
    return nat.nats_mixed_attn_mamba(s["qa"], s["ka"], s["va"], s["q"], s["k"], s["v"], None, s["g"], s["types"], None,
                                     nats_block_size=c["nbs"], ops_for_incomplete_chunks="all",
                                     output_final_state_mamba=not c["train"], decay_for_non_mamba_blocks=True)


def _forward(s, x, cache=None):
    if s["mamba"]:
        return s["module"](x, cache_params=cache, use_cache=cache is not None)
    out = s["module"](x, past_key_values=cache, use_cache=cache is not None)
    return out[0]


def run(state):
    s, c = state, state["case"]
    if c["kind"] == "long":
        with torch.no_grad():
            return nats_mixed_attn_mamba_sp(
                s["qa"], s["ka"], s["va"], s["q"], s["k"], s["v"], s["g"], s["types"], nats_block_size=c["nbs"],
                scale_attn=c["K"] ** -0.5, decay_for_non_mamba_blocks=True)
    if c["kind"] == "op" and not c["train"]:
        with torch.no_grad():
            return _op(s)
    if c["kind"] == "op":
        for n in s["leaves"]:
            s[n].grad = None
        o_l, o_a, _ = _op(s)
        torch.autograd.backward([o_l, o_a], [s["do_l"], s["do_a"]])
        return dict(o_l=o_l.detach(), o_a=o_a.detach(), **{"d" + n: s[n].grad for n in s["leaves"]})
    if c["kind"] == "layer":
        with torch.no_grad():
            return _forward(s, s["x"])
    if c["kind"] == "request":
        with torch.no_grad():
            cache = nat.NAtSCache()
            outs = [_forward(s, s["prompt"], cache)]
            outs += [_forward(s, x, cache) for x in s["tokens"]]
            layer = cache[0]
            return dict(prompt=outs[0], tokens=torch.cat(outs[1:], 1), k=layer.k_attn, v=layer.v_attn, state=layer.state,
                        block_start=layer.state_block_start)
    module = s["module"]
    module.zero_grad(set_to_none=True)
    s["x"].grad = None
    y = _forward(s, s["x"])
    y.backward(s["dy"])
    grads = {n: p.grad for n, p in module.named_parameters() if p.grad is not None}
    return dict(y=y.detach(), dx=s["x"].grad, **grads)


# ---------------------------------------------------------------------------------------------------- floors
def _linear_flops(rule, B, T, H, K, V):
    chunks = B * -(-T // C) * H
    per = 2 * C * C * (K + V) + 2 * 2 * C * K * V                         # scores and their product, state read and write
    if rule == "gdn":
        per += 2 * C * C * (2 * K + V) + 2 * C ** 3 / 3 + 2 * C * K * V   # k k^T, its inverse applied to k and v, v'
    return chunks * per


def _attn_flops(B, T, HQ, DK, DV, nbs, p):
    own = T * (min(nbs, T) + 1) / 2
    past = p * max(0, T - nbs) * T / 2
    return B * HQ * 2 * (DK + DV) * (own + past)


def _op_work(rule, B, T, H, HQ, K, V, nbs, p, size, train, shared):
    DK, DV = H * K // HQ, H * V // HQ
    flops = _linear_flops(rule, B, T, H, K, V) + _attn_flops(B, T, HQ, DK, DV, nbs, p)
    tok = B * T * H
    reads = tok * ((2 * K + V) * size * (1 if shared else 2) + 8)
    writes = 2 * tok * V * size
    if train:                                                             # 2.5 x the products, gradients of every input
        return dict(bytes=2 * reads + 2 * writes, flops=3.5 * flops)
    return dict(bytes=reads + writes + B * H * K * V * 4, flops=flops)


def work(case):
    c = case
    if c["kind"] in ("op", "long"):
        return _op_work(c["rule"], c["B"], c["T"], c["H"], c["HQ"], c["K"], c["V"], c["nbs"], c["p"],
                        4 if c["dtype"] == "fp32" else 2, c["train"], c["HQ"] == c["H"])
    s = SHAPES[c["shape"]]
    B, T, hid, H, K = c["B"], c["T"], s["hidden"], s["heads"], s["head_dim"]
    V = int(K * s["expand_v"])
    HQ = s["attn_heads"]
    weights = hid * (2 * H * K + 3 * H * V + 4 * H) + 2 * H * K * HQ      # q, k, v, gate, output; decays, types; mixing
    if c["kind"] == "train" and s["rule"] == "gdn":
        weights += 3 * hid * 256 * (-(-int(hid * 8 / 3) // 256))
    op = _op_work(s["rule"], B, T, H, HQ, K, V, c["nbs"], 0.5, 2, c["kind"] == "train", True)
    dense = 2 * B * T * weights
    if c["kind"] == "train":
        return dict(bytes=2 * 2 * weights + 4 * B * T * hid * 2, flops=3 * dense + op["flops"])
    flops, nbytes = dense + op["flops"], 2 * weights + 2 * B * T * hid * 2
    if c["kind"] == "request":
        kv = B * T * H * (K + V) * 2
        state = B * H * K * V * 4
        per_token = 2 * weights + 0.5 * kv + 2 * state                    # each token is a call of its own
        nbytes += kv + state + c["new"] * per_token
        flops += c["new"] * B * (2 * weights + 0.5 * T * 2 * H * (K + V) + 6 * H * K * V)
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    """fp32 tensors: sums of 32-bit products through a few hundred recurrence steps.  bf16 tensors: results rounded to 8
    bits; gradients and decoded tokens pass through several tensors that are rounded so on their way."""
    if case.get("dtype") == "fp32":
        return {"rel": 2e-5, "max": 1e-3}
    if case["kind"] == "train" or case.get("train"):
        return {"rel": 2e-2}
    return {"rel": 1e-2}
