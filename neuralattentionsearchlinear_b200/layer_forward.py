"""A NAtSL layer's forward without gradients: the projections as library GEMMs, everything between them and the output
projection in one native call (``natsl_layer_forward``), for the configurations it is built for; the layers' general path
covers the rest (src/nats/layers/natsl_attn_gdn.py:411-666, src/nats/layers/natsl_attn_mamba2.py:352-599)."""
from __future__ import annotations

import ctypes

import torch
import torch.nn as nn
import torch.nn.functional as F

from . import _lib, _ops
from .decode_step import layer_plan
from .modules import hard_softmax
from .nats_util import aligned, cdiv, current_stream_ptr, device_guard, transforms_active

BF16 = torch.bfloat16


def _r256(n: int) -> int:
    return -(-n // 256) * 256


@torch.no_grad()
def layer_forward(layer, x: torch.Tensor, cache=None):
    """The layer's output [B, T, hidden] for a whole sequence, or None where the general path has to run.  ``cache``: an empty
    ``NAtSLayerCache`` that receives the state a decoder continues from."""
    if (x.dim() != 3 or x.dtype != BF16 or not x.is_cuda or x.shape[1] < 64 or layer.nats_sample_func is not hard_softmax
            or torch.is_autocast_enabled() or transforms_active()):
        return None
    plan = layer_plan(layer)
    if not plan.ok or torch.nn.modules.module._has_any_global_hook():
        return None
    B, T, D = x.shape
    d = plan.args
    sel = layer.nats_layer
    if (D != d.hidden or x.device != plan.device or not _ops.walks_with_state(d.rule, d.K, d.V, T) or B > 65535
            or type(sel) is not nn.Linear or sel.bias is not None or sel.weight.dtype != BF16 or sel._forward_hooks
            or sel._forward_pre_hooks or not sel.weight.is_cuda or tuple(sel.weight.shape) != (2 * d.HN, d.hidden)):
        return None
    with device_guard(x.device):
        return _forward(layer, plan, x, cache)


def _forward(layer, plan, x, cache):
    B, T, D = x.shape
    d, sel = plan.args, layer.nats_layer
    H, K, V, HQ, HN, nbs, rule = d.H, d.K, d.V, d.HQ, d.HN, d.nbs, d.rule
    gdn = rule == _lib.RULE_GDN
    dev = x.device
    x = aligned(x.contiguous())
    st = current_stream_ptr(dev)
    TN = cdiv(T, nbs)
    bf = dict(dtype=BF16, device=dev)
    f32 = dict(dtype=torch.float32, device=dev)
    project = lambda name: F.linear(x, layer._modules[name]._parameters["weight"])
    pooled = torch.empty(B, TN, D, **bf)
    _lib.call("natsl_block_mean", x.data_ptr(), pooled.data_ptr(), B, T, D, nbs, st)
    logits = F.linear(pooled, sel.weight)
    q_raw, k_raw, v_raw = project("q_proj"), project("k_proj"), project("v_proj")
    a = plan.layer_args
    a.B, a.T = B, T
    a.options = _ops.hybrid_options(B * H)
    DK, DV = H * K // HQ, H * V // HQ
    n, nt = B * T, B * TN * HN * 2
    tables = torch.empty(2 * nt + 3 * B * HN + B * cdiv(T, 128) * HN, dtype=torch.int32, device=dev)
    key = (B, T)
    need = plan.layer_ws.get(key)
    if need is None:
        if len(plan.layer_ws) > 256:
            plan.layer_ws.clear()
        need = plan.layer_ws[key] = _lib.load().natsl_layer_workspace_bytes(ctypes.byref(a))
    own_k, own_v = bool(d.qn_w) or a.attn_conv, a.attn_conv  # keys, values that are not the projections themselves
    # intermediates of the call, what only the mixing behind it reads, and what a cache would keep
    sizes = [_r256(need), _r256(2 * n * H * V), _r256(2 * n * H * V), _r256(4 * n * HQ), _r256(4 * n * HQ),
             _r256(2 * n * H * V) if gdn and not a.attn_conv else 0]
    if cache is None:
        sizes += [_r256(2 * n * H * K) if own_k else 0, _r256(2 * n * H * V) if own_v else 0, _r256(2 * nt)]
    ws = torch.empty(sum(sizes), dtype=torch.uint8, device=dev)
    p = ws.data_ptr()
    a.workspace, a.workspace_bytes = p, need
    a.o_lin = p + sizes[0]
    a.o_attn = a.o_lin + sizes[1]
    a.mix = a.o_attn + sizes[2]
    a.lse = a.mix + sizes[3]
    a.v_lin = a.lse + sizes[4] if sizes[5] else None
    a.x, a.logits, a.q_raw, a.k_raw, a.v_raw = x.data_ptr(), logits.data_ptr(), q_raw.data_ptr(), k_raw.data_ptr(), v_raw.data_ptr()
    a.tables = tables.data_ptr()
    if cache is None:
        kept = p + sum(sizes[:6])
        a.k_attn = kept if own_k else a.k_raw
        a.v_attn = kept + sizes[6] if own_v else a.v_raw
        a.types_raw = kept + sizes[6] + sizes[7]
        a.ht = a.hstart = a.tail_q = a.tail_k = a.tail_v = a.g_block = a.pool_sum = None
    else:
        k_attn = torch.empty(B, T, HQ, DK, **bf) if own_k else k_raw.view(B, T, HQ, DK)
        v_attn = torch.empty(B, T, HQ, DV, **bf) if own_v else v_raw.view(B, T, HQ, DV)
        types_raw = torch.empty(B, TN, HN, 2, **bf)
        ht, start = torch.empty(B, H, K, V, **f32), torch.empty(B, H, K, V, **f32)
        tails = tuple(torch.empty(B, c, 4, **bf) for c in (H * K, H * K, H * V))
        g_block, pool_sum = torch.empty(B, H, **f32), torch.empty(B, D, **f32)
        a.k_attn, a.v_attn, a.types_raw = k_attn.data_ptr(), v_attn.data_ptr(), types_raw.data_ptr()
        a.ht, a.hstart, a.g_block, a.pool_sum = ht.data_ptr(), start.data_ptr(), g_block.data_ptr(), pool_sum.data_ptr()
        a.tail_q, a.tail_k, a.tail_v = (t.data_ptr() for t in tails)
    _lib.call("natsl_layer_forward", ctypes.byref(a), st)
    gate = project("g_proj")
    y = torch.empty(B, T, H * V, **bf)
    _lib.call("natsl_norm_gate_mix", a.o_lin, a.o_attn, gate.data_ptr(), a.mix if a.w_mix else None, _lib.DT_BF16, d.w1, d.w2,
              _lib.DT_F32 if d.w12_f32 else _lib.DT_BF16, y.data_ptr(), n * HQ, DV, d.mix_eps, d.mix_sigmoid, st)
    layer.__dict__["attn_blocks"] = (tables[2 * nt:2 * nt + 2 * B * HN].view(B, HN, 2), TN)
    if cache is not None:
        r, n_done = T % nbs, T // nbs
        cache.append_kv(k_attn, v_attn)
        if n_done:
            cache.append_types(types_raw if n_done == TN else types_raw[:, :n_done].contiguous())
        cache.set_state(start.clone() if r == 0 else ht, start, g_block, pool_sum, tails)
        cache.n_tokens = T
    return F.linear(y, layer._modules["o_proj"]._parameters["weight"])
