"""Single-token decoding of a whole layer through ``natsl_decode_step`` (four launches, state updated in place) for the
configurations the kernel is built for; everything else takes the general path of ``decoding.forward_cached``
(src/nats/layers/natsl_attn_gdn.py:389-666, src/nats/layers/natsl_attn_mamba2.py:330-599 with one new token)."""
from __future__ import annotations

import ctypes
import operator
import threading
import weakref

import torch
import torch.nn as nn

from . import _lib, nats_util
from .modules import FusedMultiInputRMSNormGated, L2Norm, RMSNorm, ShortConvolution, mean_pooling
from .nats_util import aligned, current_stream_ptr, device_guard, transforms_active

BF16 = torch.bfloat16
MAX_BATCH = 64
_dtype = operator.attrgetter("dtype")
_tls = threading.local()                     # one argument block per thread: a call in flight is never rewritten


# Attributes of a layer that the plan's argument blocks or its choice of path are made from; hooks of the general path that an
# instance may have replaced (normally absent from its __dict__).
_LAYER_ATTRS = ("num_heads num_v_heads num_attn_heads num_nats_head n_ops hidden_size key_dim value_dim head_k_dim head_v_dim "
                "head_attn_k_dim head_attn_v_dim nats_block_size attn_qk_norm attn_with_short_conv use_short_conv use_gate "
                "ops_for_incomplete_chunks incomplete_block_start_with_ht usg_for_attn outputs_are_weighted outputs_are_wighted "
                "decay_for_non_gdn_blocks decay_for_non_mamba_blocks allow_neg_eigval pooling_func").split()
_LAYER_HOOKS = ("select", "project", "project_qkv", "mix", "_ops_for_cache")


class _Plan:
    """Argument blocks of one layer: shapes, options and weight pointers, valid while ``current()`` holds."""

    def __init__(self, layer):
        self.ok = False
        mods = {n: type_ for n, type_ in (
            ("q_proj", nn.Linear), ("k_proj", nn.Linear), ("v_proj", nn.Linear), ("a_proj", nn.Linear),
            ("g_proj", nn.Linear), ("o_proj", nn.Linear), ("q_conv1d", ShortConvolution), ("k_conv1d", ShortConvolution),
            ("v_conv1d", ShortConvolution), ("o_norm", FusedMultiInputRMSNormGated))}
        gdn = hasattr(layer, "b_proj")
        weighted = layer.outputs_are_weighted if gdn else layer.outputs_are_wighted
        if gdn:
            mods["b_proj"] = nn.Linear
        else:
            mods["q_norm2"] = mods["k_norm2"] = L2Norm
        if weighted:
            mods["nats_out_weights_layer"] = nn.Linear
        if layer.attn_qk_norm:
            mods["q_norm"] = mods["k_norm"] = RMSNorm
        self.mods = [(layer._modules, n, layer._modules.get(n)) for n in mods]
        self.hooks, self.params, self.device = [], [], None
        if all(type(m) is mods[n] for _, n, m in self.mods):
            self.hooks = [h for _, _, m in self.mods for h in (m._forward_hooks, m._forward_pre_hooks)]
            self.ok = self._fill(layer, gdn, weighted)
        self._hooked = any(self.hooks)
        # what current() compares, in as few passes in C as it takes (a token's host time is some 30 us)
        self._layer_dict, self._modules = layer.__dict__, layer._modules
        self._replaced = list(map(layer.__dict__.__contains__, _LAYER_HOOKS))
        self.ok = self.ok and not self._hooked and not any(self._replaced)
        self._get_mods = operator.itemgetter(*(n for n in mods if n in layer._modules))
        self._mods = self._get_mods(layer._modules)
        self._get_attrs = operator.itemgetter(*(n for n in _LAYER_ATTRS if n in layer.__dict__))
        self._attrs = self._get_attrs(layer.__dict__)
        attrs = [(m.__dict__, n) for m in self._mods for n in ("eps", "activation", "kernel_size", "hidden_size")
                 if m is not None and n in m.__dict__]
        self._att_d, self._att_n = zip(*attrs) if attrs else ((), ())
        self._att_v = list(map(dict.get, self._att_d, self._att_n))
        there = sorted(((d, n) for d, n, p in self.params if p is not None), key=lambda e: -e[0][e[1]].dim())
        self._n_mat = sum(d[n].dim() > 1 for d, n in there)   # matrices first
        self._par_d, self._par_n = zip(*there) if there else ((), ())
        absent = [(d, n) for d, n, p in self.params if p is None]
        self._abs_d, self._abs_n = zip(*absent) if absent else ((), ())
        self._nones = [None] * len(absent)
        self._par_v = self._look(map(dict.get, self._par_d, self._par_n))

    def _look(self, tensors):
        """Addresses and types, of matrices also sizes and contiguity: what a kernel takes on trust of the weights."""
        t = list(tensors)
        mats = t[:self._n_mat]
        return (list(map(torch.Tensor.data_ptr, t)), list(map(_dtype, t)), list(map(torch.Tensor.numel, mats)),
                all(map(torch.Tensor.is_contiguous, mats)))

    def _fill(self, layer, gdn: bool, weighted: bool) -> bool:
        a = self.args = _lib.DecodeArgs()

        m = layer
        self.device, index = m.q_proj.weight.device, m.q_proj.weight.get_device()
        linears = [mod for _, _, mod in self.mods if type(mod) is nn.Linear]
        self.params += [(mod._parameters, "bias", mod.bias) for mod in linears]          # the products add none
        H, HQ, K, V, DK, DV, D = (m.num_heads, m.num_attn_heads, m.head_k_dim, m.head_v_dim, m.head_attn_k_dim, m.head_attn_v_dim,
                                  m.hidden_size)

        def weight(field, owner, *shape, name="weight", any_float=None, optional=False):
            p = owner._parameters.get(name)
            self.params.append((owner._parameters, name, p))
            if p is None:
                return optional
            if type(p) not in (nn.Parameter, torch.Tensor) or p.shape != shape or p.get_device() != index:
                return False
            dtype, ptr = p.dtype, p.data_ptr()
            if any_float is not None and dtype == torch.float32:
                setattr(a, any_float, 1)
            elif dtype != BF16:
                return False
            setattr(a, field, ptr)
            # products read 16 bytes at a time, convolutions 8: a parameter that is a view into a flat buffer may start anywhere
            align = 16 if field.startswith("w_") else 8 if field.startswith("cw_") else 1
            return index >= 0 and p.is_contiguous() and ptr % align == 0

        checks = [weight("w_q", m.q_proj, H * K, D), weight("w_k", m.k_proj, H * K, D), weight("w_v", m.v_proj, H * V, D),
                  weight("w_a", m.a_proj, H, D), weight("w_g", m.g_proj, H * V, D), weight("w_o", m.o_proj, D, H * V),
                  weight("A_log", m, H, name="A_log", any_float="alog_f32"),
                  weight("dt_bias", m, H, name="dt_bias", any_float="dt_f32")]
        for n, conv, width in (("q", m.q_conv1d, H * K), ("k", m.k_conv1d, H * K), ("v", m.v_conv1d, H * V)):
            checks += [weight("cw_" + n, conv, width, 1, 4), weight("cb_" + n, conv, width, name="bias", optional=True)]
        checks += [weight(f"w{i}", m.o_norm, DV, name=f"weight{i}", any_float="w12_f32", optional=True) for i in (1, 2)]
        if gdn:
            checks.append(weight("w_b", m.b_proj, H, D))
        else:
            checks.append(m.q_norm2.eps == m.k_norm2.eps)
            a.l2_eps = m.q_norm2.eps
        if weighted:
            checks.append(weight("w_mix", m.nats_out_weights_layer, 2 * HQ, H * K))
        if m.attn_qk_norm:
            checks += [weight("qn_w", m.q_norm, DK, any_float="qn_f32"), weight("kn_w", m.k_norm, DK, any_float="kn_f32"),
                       m.q_norm.eps == m.k_norm.eps]
            a.norm_eps = m.q_norm.eps
        w1, w2 = m.o_norm.weight1, m.o_norm.weight2
        ok = bool(
            all(checks) and all(mod.bias is None for mod in linears)
            and (w1 is None) == (w2 is None) and (w1 is None or w1.dtype == w2.dtype)
            and m.num_v_heads == H and m.n_ops == 2 and m.o_norm.hidden_size == DV
            and m.key_dim == H * K == HQ * DK and m.value_dim == H * V == HQ * DV
            and all(c.kernel_size == (4,) and c.activation == m.q_conv1d.activation for c in (m.q_conv1d, m.k_conv1d, m.v_conv1d))
            and D % 32 == 0 and m.value_dim % 32 == 0 and K % 32 == 0 and K <= 256 and V % 32 == 0 and DK in (64, 128)
            and DV in (64, 128) and m.key_dim <= 10240
            and m.num_heads % m.num_nats_head == 0 and m.num_attn_heads % m.num_nats_head == 0
            and m.use_short_conv and m.use_gate and m.ops_for_incomplete_chunks != 'attn' and m.incomplete_block_start_with_ht
            and not m.usg_for_attn and m.pooling_func is mean_pooling)
        a.hidden, a.H, a.K, a.V, a.HQ, a.HN = D, H, K, V, HQ, m.num_nats_head
        self.hidden = D
        a.nbs, a.rule = m.nats_block_size, _lib.RULE_GDN if gdn else _lib.RULE_MAMBA
        a.silu = int(m.q_conv1d.activation in ("silu", "swish"))
        a.mix_sigmoid, a.mix_eps = int(m.o_norm.activation == "sigmoid"), m.o_norm.eps
        a.scale_attn, a.scale_lin = DK ** -0.5, K ** -0.5 if gdn else 1.0
        a.own_chunk, a.attn_conv = int(m.ops_for_incomplete_chunks == 'all'), int(m.attn_with_short_conv)
        a.decay = int(m.decay_for_non_gdn_blocks if gdn else m.decay_for_non_mamba_blocks)
        a.neg_eigval = int(gdn and m.allow_neg_eigval)
        self.ws_bytes = {}
        b = self.layer_args = _lib.LayerArgs()
        for n in ("hidden H K V HQ HN nbs rule attn_conv silu own_chunk decay neg_eigval qn_f32 kn_f32 alog_f32 dt_f32 norm_eps l2_eps "
                  "scale_attn scale_lin w_a w_b w_mix cw_q cw_k cw_v cb_q cb_k cb_v qn_w kn_w A_log dt_bias").split():
            setattr(b, n, getattr(a, n))
        self.layer_ws = {}
        return ok

    def current(self) -> bool:
        try:
            return (self._get_mods(self._modules) == self._mods and self._get_attrs(self._layer_dict) == self._attrs
                    and list(map(dict.get, self._att_d, self._att_n)) == self._att_v
                    and list(map(self._layer_dict.__contains__, _LAYER_HOOKS)) == self._replaced and any(self.hooks) == self._hooked
                    and list(map(dict.get, self._abs_d, self._abs_n)) == self._nones
                    and self._look(map(dict.get, self._par_d, self._par_n)) == self._par_v)
        except (KeyError, TypeError):                        # a module, attribute or weight has gone
            return False


class _Step:
    """Argument block of one layer's decoding steps on one cache: everything that stays the same from token to token."""

    def __init__(self, plan, B, dev):
        self.plan, self.cache_tensors = plan, None
        a = self.args = _lib.DecodeArgs()
        ctypes.memmove(ctypes.byref(a), ctypes.byref(plan.args), ctypes.sizeof(a))
        a.B = self.B = B
        need = plan.ws_bytes.get(B)
        if need is None:
            need = plan.ws_bytes[B] = _lib.load().natsl_decode_workspace_bytes(ctypes.byref(a))
            if need < 0:
                raise _lib.NatslError(_lib.load().natsl_last_error().decode())
        self.workspace = torch.empty(need, dtype=torch.uint8, device=dev)
        a.workspace, a.workspace_bytes = self.workspace.data_ptr(), need
        self.ref = ctypes.byref(a)

    def bind(self, cache) -> bool:
        """Takes over the cache's tensors (made contiguous where they are not); False if they are not the kernel's kind."""
        a = self.args
        B, dev, HK, HV = a.B, self.workspace.device, a.H * a.K, a.H * a.V
        state = (B, a.H, a.K, a.V)
        for name, shape in (("_state", state), ("_state_block_start", state), ("_g_block", (B, a.H)), ("_pool_sum", (B, a.hidden))):
            t = getattr(cache, name)
            if t is None or tuple(t.shape) != shape or t.device != dev:
                return False
            if t.dtype != torch.float32 or not t.is_contiguous():
                setattr(cache, name, t.float().contiguous())
        conv, rows, types = cache._conv_state, (cache._k_buf, cache._v_buf), cache.block_types
        if (conv is None or len(conv) != 3 or any(t is None or t.dtype != BF16 or t.device != dev for t in (*conv, *rows))
                or [tuple(t.shape) for t in conv] != [(B, HK, 4), (B, HK, 4), (B, HV, 4)]):
            return False
        cap = rows[0].shape[1]
        if [tuple(t.shape) for t in rows] != [(B, cap, a.HQ, HK // a.HQ), (B, cap, a.HQ, HV // a.HQ)]:
            return False
        if types is not None:
            if types.dtype not in (BF16, torch.float32) or types.device != dev or tuple(types.shape) != (B, types.shape[1], a.HN, 2):
                return False
            a.types_f32 = int(types.dtype == torch.float32)
            if not types.is_contiguous():
                types = cache.block_types = types.contiguous()
        if not all(t.is_contiguous() for t in conv):
            conv = cache._conv_state = tuple(t.contiguous() for t in conv)
        if any(t.data_ptr() % 16 for t in (cache._state, cache._state_block_start, *rows, *conv)):
            return False
        a.conv_q, a.conv_k, a.conv_v = (t.data_ptr() for t in conv)
        a.state, a.start, a.g_block = cache._state.data_ptr(), cache._state_block_start.data_ptr(), cache._g_block.data_ptr()
        a.k_cache, a.v_cache, a.cap = rows[0].data_ptr(), rows[1].data_ptr(), cap
        a.types = None if types is None else types.data_ptr()
        self.cache_tensors = (cache._state, cache._state_block_start, cache._g_block, cache._pool_sum, conv, *rows, types)
        self.pool = cache._pool_sum.data_ptr()
        return True

    def bound(self, cache) -> bool:
        """Whether these are the tensors that ``bind`` has checked.  All but the types are the cache's own (``own_state``):
        nobody else can give one of them another storage or shape."""
        t = self.cache_tensors
        return (t is not None and t[0] is cache._state and t[1] is cache._state_block_start and t[2] is cache._g_block
                and t[3] is cache._pool_sum and t[4] is cache._conv_state and t[5] is cache._k_buf and t[6] is cache._v_buf
                and t[7] is cache.block_types and (t[7] is None or t[7].data_ptr() == self.args.types))


def layer_plan(layer) -> _Plan:
    """This thread's plan of the layer, rebuilt when a module, an attribute, a parameter or its storage has changed."""
    plans = getattr(_tls, "plans", None)
    if plans is None:
        plans = _tls.plans = weakref.WeakKeyDictionary()
    p = plans.get(layer)
    if p is None or not p.current():
        p = plans[layer] = _Plan(layer)
    return p


def decode_token(layer, x: torch.Tensor, container):
    """The layer's output [B, 1, hidden] for one new token, or None where the general path has to run (which also raises
    what there is to raise).  Updates the layer's cache."""
    shape = x.shape
    if len(shape) != 3 or shape[1] != 1 or x.dtype != BF16 or not x.is_cuda or layer.layer_idx is None or not hasattr(container, "layer"):
        return None
    plan = layer_plan(layer)
    # the kernel reads and writes batch * hidden entries of x and the output: every token's width and device count
    if not plan.ok or shape[2] != plan.hidden or x.get_device() != plan.device.index:
        return None
    nbs = layer.nats_block_size
    cache = container.layer(layer.layer_idx, nbs)
    B = shape[0]
    step = cache._step
    if step is None or step.plan is not plan or step.B != B:
        if B > MAX_BATCH:
            return None
        step = _Step(plan, B, x.device)
    if torch.is_autocast_enabled() or torch.nn.modules.module._has_any_global_hook() or transforms_active():
        return None
    if nats_util.current_device() == plan.device.index:
        return _decode(layer, x, cache, step, cache.n_tokens, nbs)
    with device_guard(plan.device):
        return _decode(layer, x, cache, step, cache.n_tokens, nbs)


def _decode(layer, x, cache, step, pos: int, nbs: int):
    a = step.args
    B, D, dev = a.B, a.hidden, step.workspace.device
    if pos == 0:                                             # a prompt of one token: start from empty states
        f32 = dict(dtype=torch.float32, device=dev)
        cache.set_state(torch.zeros(B, a.H, a.K, a.V, **f32), torch.zeros(B, a.H, a.K, a.V, **f32), torch.zeros(B, a.H, **f32),
                        torch.zeros(B, D, **f32), tuple(torch.zeros(B, n, 4, dtype=BF16, device=dev)
                                                        for n in (layer.key_dim, layer.key_dim, layer.value_dim)))
        cache._k_buf = torch.empty(B, 256, a.HQ, layer.head_attn_k_dim, dtype=BF16, device=dev)
        cache._v_buf = torch.empty(B, 256, a.HQ, layer.head_attn_v_dim, dtype=BF16, device=dev)
        cache._n_kv, cache._kv_shared = 0, False
    elif cache._k_buf is None or cache._n_kv != pos:
        return None
    n_done = pos // nbs
    if n_done and (cache.block_types is None or cache.block_types.shape[1] != n_done):
        return None
    x = aligned((x.detach() if x.requires_grad else x).contiguous())
    types_new = None
    if (pos + 1) % nbs == 0:                                 # a block's type is decided once its last token is known
        with torch.no_grad():
            pooled = ((cache._pool_sum + x[:, 0].float()) / nbs).to(x.dtype)[:, None, :]
            types_new = layer.select(pooled).contiguous()
        if types_new.dtype not in (BF16, torch.float32) or (cache.block_types is not None and cache.block_types.dtype != types_new.dtype):
            return None
    cache.reserve_kv(1)
    if cache._handed_out:
        cache.own_state()
    if not step.bound(cache) and not step.bind(cache):
        return None
    cache._step = step
    out = torch.empty_like(x)
    a.pos, a.n_done = pos, n_done
    a.x, a.out = x.data_ptr(), out.data_ptr()
    if types_new is None:
        a.types_new, a.pool_sum = None, step.pool
    else:
        a.types_new, a.pool_sum, a.types_f32 = types_new.data_ptr(), None, int(types_new.dtype == torch.float32)
    _lib.call("natsl_decode_step", step.ref, current_stream_ptr(dev))
    cache._n_kv = cache.n_tokens = pos + 1
    if types_new is not None:
        cache.append_types(types_new)
        cache._pool_sum = torch.zeros_like(cache._pool_sum)
    return out
