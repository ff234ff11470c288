"""Thin launch wrappers: allocate outputs with torch, pass raw pointers to the C ABI."""
from __future__ import annotations

import ctypes
import os

import torch

from . import _lib
from .nats_util import _TYPE_CODES, SelectionTables, aligned, cdiv, current_stream_ptr, device_guard

BF16 = torch.bfloat16
USE_MAMBA_WALK = os.environ.get("NATSL_MAMBA_WALK", "1") != "0"    # natsl_mamba_walk_fused (K = 128, V = 64)
# recurrence + output in one walk: on tcgen05 (natsl_gdn_walk_fused, K = V = 128, block 64) or mma.sync (natsl_gdn_walk)
USE_FUSED_WALK = True
# (K, V) with a chunk preparation; all of them have a walk for every block size.  192 / 384 (the 760M configuration) runs the
# form that holds state and operands to fp32 precision (natsl_gdn_split_*).
GDN_HEAD_DIMS = {(64, 64), (64, 128), (128, 64), (128, 128), (128, 256), (192, 384)}
# value dimension of the fused walk split over two CTAs (natsl_gdn_walk_fused_vsplit, T <= 8192): half an SM per CTA.
# Off by default: measured alone it is no faster than the one-CTA walk (0.204 vs 0.130 ms at B=8, T=4096, H=16), and
# the kernels of the two branches do not overlap in practice (the block scheduler drains one grid before the next).
WALK_VSPLIT = os.environ.get("NATSL_WALK_VSPLIT", "0") == "1"
# chunk preparation on tcgen05 for K = V = 128 (natsl_gdn_chunk_prep_tc); "0" takes the mma.sync kernel there
PREP_TC = os.environ.get("NATSL_PREP_TC", "1") != "0"


# accepted, without effect: the softmax branch's one kernel is persistent
ATTN_PERSISTENT = os.environ.get("NATSL_ATTN_PERSISTENT", "0") == "1"

# The linear branch (chunk preparation -> walk) runs on a high-priority stream, so that its CTAs are placed ahead of the
# softmax branch's remaining ones whenever an SM frees up: the serial walk then starts earlier and the attention CTAs
# fill in around it.  Measured with the step replayed from a CUDA graph: 0.523 - 0.542 ms against 0.559 - 0.561 ms
# (three runs each); NATSL_LINEAR_PRIORITY=0 puts the branch back on the caller's stream.
LINEAR_BRANCH_PRIORITY = os.environ.get("NATSL_LINEAR_PRIORITY", "1") != "0"

# (batch, head) pairs up to which the delta rule takes the mma.sync walk also where the tcgen05 one is built (K = V = 128,
# block 64): 32 value columns per CTA make four CTAs of a pair, which fit one wave of 148 SMs up to 37 pairs, and a chunk takes
# 1.6 instead of 1.8 us.  Whole ops captured in a graph, mma.sync against tcgen05: 4 to 28 pairs 18 / 22 us at T = 256, 62 - 89 /
# 70 - 96 us at T = 2048, 111 - 172 / 124 - 179 us at T = 4096; 32 pairs 93 / 101 us at T = 2048, 201 / 190 us at T = 4096; 48
# pairs (two waves) 28 / 24, 135 / 117 and 261 / 216 us.  Between 31 and 37 the line gives way to batches of 16-head sequences:
# from two of them on a sequence's result does not depend, bit for bit, on the batch around it.  0 extends that to one sequence
# (one walk for all).
WALK_MMA_MAX_HEADS = int(os.environ.get("NATSL_WALK_MMA_MAX_HEADS", "31"))


def _attn_flags(own_chunk: bool) -> int:
    return _lib.FLAG_ATTN_OWN_CHUNK if own_chunk else 0


def prep_entry(K: int, V: int) -> str:
    """Name of the chunk-preparation entry point for these head dims (both take the arguments of ``..._prep_ex``)."""
    return "natsl_gdn_chunk_prep_tc" if (PREP_TC and K == 128 and V == 128) else "natsl_gdn_chunk_prep_ex"


def walks_with_state(rule: int, K: int, V: int, T: int) -> bool:
    """Whether ``linear_fwd`` can hand over the block-start state of these head dims without chunk intermediates."""
    if rule == _lib.RULE_GDN:
        return USE_FUSED_WALK and (K, V) in GDN_HEAD_DIMS and T <= 65536
    return USE_MAMBA_WALK and K == 128 and V == 64 and T <= 65536


def _need(cond: bool, msg: str, exc=ValueError):
    if not cond:
        raise exc(msg)


def _check_qkv(q, k, v, tables, what: str, same_heads: bool):
    """Shapes that the kernels take on trust: the same batch, key and value sequences of one length, matching head
    counts and head dims, tables built for this batch, everything on one CUDA device."""
    _need(q.dim() == 4 and k.dim() == 4 and v.dim() == 4, f"{what}: q, k, v must be [B, T, H, D]")
    _need(q.is_cuda and k.device == q.device and v.device == q.device, f"{what}: q, k, v must be on one CUDA device")
    _need(k.shape[0] == q.shape[0] and v.shape[0] == q.shape[0], f"{what}: q, k, v differ in batch size")
    _need(k.shape[3] == q.shape[3], f"{what}: q and k differ in head dim ({q.shape[3]} vs {k.shape[3]})")
    _need(v.shape[1] == k.shape[1] and v.shape[2] == k.shape[2],
          f"{what}: k {tuple(k.shape)} and v {tuple(v.shape)} differ in length or heads")
    if same_heads:
        _need(k.shape[1] == q.shape[1] and k.shape[2] == q.shape[2], f"{what}: q {tuple(q.shape)} and k {tuple(k.shape)} differ")
    else:
        _need(q.shape[2] % k.shape[2] == 0, f"{what}: {q.shape[2]} query heads over {k.shape[2]} key/value heads")
    _need(tables.types_i.shape[0] == q.shape[0] and tables.types_i.device == q.device,
          f"{what}: the selection tables were built for another batch or device")


def attn_fwd(q, k, v, tables: SelectionTables, scale: float, own_chunk: bool, mma_sync: bool = False, q_off: int = 0):
    """q [B,Tq,HQ,DK], k [B,T,HKV,DK], v [B,T,HKV,DV] bf16 -> (o [B,Tq,HQ,DV] bf16, lse [B,Tq,HQ] fp32 base-2).
    The queries are the tokens [q_off, q_off+Tq) of the T-key sequence (q_off = 0 and Tq = T normally)."""
    _need(q.dtype == BF16 and k.dtype == BF16 and v.dtype == BF16, "softmax branch needs bf16 q/k/v", TypeError)
    _check_qkv(q, k, v, tables, "softmax branch", same_heads=False)
    q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
    B, Tq, HQ, DK = q.shape
    T, HKV, DV = k.shape[1], k.shape[2], v.shape[3]
    _need(tables.T == T, f"tables were built for T={tables.T}, keys have T={T}")
    _need(0 <= q_off and q_off + Tq <= T, f"queries [{q_off}, {q_off + Tq}) do not lie inside the {T} keys")
    HN = tables.types_i.shape[2]
    o = torch.empty(B, Tq, HQ, DV, dtype=BF16, device=q.device)
    lse = torch.empty(B, Tq, HQ, dtype=torch.float32, device=q.device)
    flags = _attn_flags(own_chunk) | (_lib.FLAG_ATTN_MMA_SYNC if mma_sync else 0)
    _lib.call("natsl_attn_fwd_ex", q.data_ptr(), k.data_ptr(), v.data_ptr(), tables.types_i.data_ptr(),
              tables.indices.data_ptr(), tables.attn_n_iters.data_ptr(), o.data_ptr(), lse.data_ptr(),
              B, T, Tq, int(q_off), HQ, HKV, HN, DK, DV, tables.nats_block_size, float(scale), flags,
              current_stream_ptr(q.device))
    return o, lse


def attn_fwd_split(q, k_rem, v_rem, k, v, tables: SelectionTables, scale: float, own_chunk: bool, rem_base=None,
                   rem_slots: int = 0):
    """Softmax branch over a key sequence held in two parts: keys [0, S) gathered from other segments (shared by the
    B / B_rem local segments that sit segment-major in the batch of q, k, v) and keys [S, S+L) in k, v [B, L, HKV, .];
    the queries q [B, L, HQ, DK] are the tokens [S, S+L).  Gathered part: k_rem, v_rem [B_rem, S, HKV, .], or with
    ``rem_base`` [B_rem, G, HKV] int32 the packed selected (block, head) pairs [B_rem, tokens, .] of G segments with
    ``rem_slots`` virtual blocks per head each (S = G * rem_slots * block size).  -> o [B, L, HQ, DV] bf16."""
    for t_ in (q, k_rem, v_rem, k, v):
        _need(t_.dtype == BF16 and t_.is_contiguous(), "softmax branch needs contiguous bf16 tensors", TypeError)
    B, L, HQ, DK = q.shape
    HKV, DV = k.shape[2], v.shape[3]
    B_rem = k_rem.shape[0]
    nbs = tables.nats_block_size
    if rem_base is None:
        S, rem_tokens = k_rem.shape[1], 0
    else:
        _need(rem_base.dtype == torch.int32 and rem_base.is_contiguous() and rem_base.shape[0] == B_rem
              and rem_base.shape[2] == HKV, "rem_base must be a contiguous int32 [B_rem, G, HKV] tensor")
        S, rem_tokens = rem_base.shape[1] * int(rem_slots) * nbs, k_rem.shape[1]
    _need(tables.T == S + L, f"tables were built for T={tables.T}, keys have T={S + L}")
    o = torch.empty(B, L, HQ, DV, dtype=BF16, device=q.device)
    lse = torch.empty(B, L, HQ, dtype=torch.float32, device=q.device)
    _lib.call("natsl_attn_fwd_split", q.data_ptr(), k_rem.data_ptr(), v_rem.data_ptr(), _lib.ptr(rem_base), int(rem_slots),
              int(rem_tokens), k.data_ptr(), v.data_ptr(), tables.types_i.data_ptr(), tables.indices.data_ptr(),
              tables.attn_n_iters.data_ptr(), o.data_ptr(), lse.data_ptr(), B, B_rem, S + L, L, S, S, HQ, HKV,
              tables.types_i.shape[2], DK, DV, nbs, float(scale), _attn_flags(own_chunk), current_stream_ptr(q.device))
    return o


def attn_dense_mask(tables: SelectionTables, HQ: int, own_chunk: bool) -> torch.Tensor:
    """Debug: the dense boolean mask [B,HQ,T,T] the attention kernel realises."""
    B, TN, HN, _ = tables.types_i.shape
    T = tables.T
    mask = torch.empty(B, HQ, T, T, dtype=torch.uint8, device=tables.types_i.device)
    flags = _lib.FLAG_ATTN_OWN_CHUNK if own_chunk else 0
    _lib.call("natsl_attn_dense_mask", tables.types_i.data_ptr(), tables.indices.data_ptr(),
              tables.attn_n_iters.data_ptr(), mask.data_ptr(), B, T, HQ, HN, tables.nats_block_size, flags,
              current_stream_ptr(mask.device))
    return mask.bool()


def linear_fwd(rule: int, q, k, v, g, beta, tables: SelectionTables, scale: float, h0, decay: bool,
               use_l2norm: bool, output_final_state: bool, trailing_quirk: bool = True,
               return_intermediates: bool = False, skip_out: bool = False, own_chunk: bool = True, tables_event=None,
               want_start: bool = False, last_types=None):
    """Linear branch forward (prep -> state recurrence -> output).  Returns (o, ht, inter); with ``skip_out``
    only the recurrence runs (o is None).  ``own_chunk=False``: the output keeps only the state term (the mode
    in which the softmax branch alone covers the current chunk); ``tables`` must then be per 64-token chunk.
    ``tables_event``: CUDA event after which the tables (built on another stream) are valid; the chunk preparation
    does not read them and is launched before the wait.  ``want_start`` (head dims of ``walks_with_state``): inter is
    dict(start=...), the state a decoder rolls back to, with ``last_types`` [B,HN,2] the own types of a complete last block."""
    _need(q.dtype == BF16 and k.dtype == BF16 and v.dtype == BF16, "linear branch needs bf16 q/k/v", TypeError)
    _check_qkv(q, k, v, tables, "linear branch", same_heads=True)
    q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
    B, T, H, K = q.shape
    V = v.shape[3]
    dev = q.device
    _need(tables.T == T, f"tables were built for T={tables.T}, the sequence has T={T}")
    _need(tuple(g.shape) == (B, T, H) and g.device == dev, f"g must be [B,T,H] = {(B, T, H)} on {dev}, got {tuple(g.shape)}")
    _need(beta is None or (tuple(beta.shape) == (B, T, H) and beta.device == dev),
          f"beta must be [B,T,H] = {(B, T, H)} on {dev}")
    _need(rule != _lib.RULE_GDN or beta is not None, "the gated delta rule needs beta")
    HN = tables.types_i.shape[2]
    _need(H % HN == 0, f"{H} heads over {HN} selection heads")
    NT = cdiv(T, 64)
    nbs = tables.nats_block_size
    walk = (rule == _lib.RULE_GDN and walks_with_state(rule, K, V, T) and not return_intermediates and not skip_out and own_chunk)
    if not walk and (K not in (64, 128) or V not in (64, 128, 256)):
        # head dims the chunk kernels have no tiles for: the token recurrence with re-roll computes the same function for
        # any K in {32, 64, 96, 128, 192, 256} and V a multiple of 8 -- correct, not fast, forward only
        if return_intermediates or skip_out or not own_chunk:
            raise NotImplementedError(f"head dims K={K}, V={V} run the token recurrence, which has no chunk intermediates "
                                      "(backward pass, state-only and mode 'attn' need K in {64,128}, V in {64,128,256})")
        if tables_event is not None:
            torch.cuda.current_stream(dev).wait_event(tables_event)
        o, ht, _ = linear_recurrent(rule, q, k, v, g, beta, tables, scale, h0, decay, use_l2norm)
        return o, (ht if output_final_state else None), None
    st = current_stream_ptr(dev)
    g = g.float().contiguous()
    gcs = torch.empty(B, T, H, dtype=torch.float32, device=dev)
    fused = walk
    tc_walk = walk and K == 128 and V == 128 and nbs == 64 and B * H > WALK_MMA_MAX_HEADS
    # Mamba2 with state dim 128 and head dim 64: recurrence + output (or the recurrence alone) in one tcgen05 walk
    mamba_fused = (rule == _lib.RULE_MAMBA and K == 128 and V == 64 and NT <= 1024 and not return_intermediates
                   and own_chunk and USE_MAMBA_WALK and (not skip_out or output_final_state))
    if rule == _lib.RULE_GDN:
        beta = beta.contiguous()
        _need(beta.dtype in (BF16, torch.float32), "beta must be bf16 or fp32", TypeError)
        beta_code = _lib.DT_BF16 if beta.dtype == BF16 else _lib.DT_F32
        krstd = torch.empty(B, T, H, dtype=torch.float32, device=dev)
        qrstd = torch.empty(B, T, H, dtype=torch.float32, device=dev) if fused else None
    split = rule == _lib.RULE_GDN and K == 192
    if split:
        tp = torch.empty(B, T, H, 320, dtype=BF16, device=dev)
        egl = torch.empty(B, NT, H, dtype=torch.float32, device=dev)
        factors = (gcs, krstd, torch.empty(2, B, T, H, dtype=torch.float32, device=dev), egl)
        _lib.call("natsl_gdn_split_prep", q.data_ptr(), k.data_ptr(), g.data_ptr(), beta.data_ptr(), beta_code, tp.data_ptr(),
                  *(t.data_ptr() for t in factors), B, T, H, K, int(use_l2norm), st)
    elif rule == _lib.RULE_GDN:
        w = torch.empty(B, T, H, K, dtype=BF16, device=dev)
        u = torch.empty(B, T, H, V, dtype=BF16, device=dev)
        pmat = torch.empty(B, T, H, 64, dtype=BF16, device=dev) if fused else None
        _lib.call(prep_entry(K, V), q.data_ptr() if fused else None, k.data_ptr(), v.data_ptr(), g.data_ptr(),
                  beta.data_ptr(), beta_code, w.data_ptr(), u.data_ptr(),
                  gcs.data_ptr(), krstd.data_ptr(), _lib.ptr(qrstd), _lib.ptr(pmat), B, T, H, K, V, int(use_l2norm), st)
    else:
        w, u, krstd = None, v, None
        _lib.call("natsl_chunk_local_cumsum", g.data_ptr(), gcs.data_ptr(), B, T, H, st)
    if tables_event is not None:
        torch.cuda.current_stream(dev).wait_event(tables_event)
    ht = torch.empty(B, H, K, V, dtype=torch.float32, device=dev) if output_final_state else None
    if h0 is not None:
        h0 = aligned(h0.float().contiguous())
        _need(tuple(h0.shape) == (B, H, K, V) and h0.device == dev, f"initial state must be [B,H,K,V] on {dev}, got {tuple(h0.shape)}")
    flags = (_lib.FLAG_DECAY_SKIPPED if decay else 0) | (0 if trailing_quirk else _lib.FLAG_NO_TRAILING_QUIRK)
    start, last_code = None, _lib.DT_F32
    if want_start:
        _need(fused or mamba_fused, "the block-start state needs head dims with a fused walk", NotImplementedError)
        start = torch.empty(B, H, K, V, dtype=torch.float32, device=dev)
        if T % nbs == 0:
            _need(last_types is not None and tuple(last_types.shape) == (B, HN, 2) and last_types.device == dev,
                  f"a complete last block needs its types [B,HN,2] on {dev}")
            last_types = (last_types if last_types.dtype in (BF16, torch.float32) else last_types.float()).contiguous()
            last_code = _dt_code(last_types)
        else:
            last_types = None
    inter = dict(start=start) if want_start else None
    if fused:
        # recurrence + output in one walk; the per-chunk states are never materialised
        o = torch.empty(B, T, H, V, dtype=BF16, device=dev)
        operands = (v, tp, *factors) if split else (w, u, pmat, gcs, krstd, qrstd)
        args = (q.data_ptr(), k.data_ptr(), *(t.data_ptr() for t in operands),
                tables.types_i.data_ptr(), tables.indices.data_ptr(), tables.n_blocks.data_ptr(),
                _lib.ptr(h0), o.data_ptr(), _lib.ptr(ht))
        dims = (B, T, H, HN, K, V, nbs, float(scale), flags, st)
        if WALK_VSPLIT and tc_walk and NT <= 128 and not want_start:
            _lib.call("natsl_gdn_walk_fused_vsplit", *args, *dims)
        else:
            entry = "natsl_gdn_split_walk" if split else "natsl_gdn_walk_fused_ex" if tc_walk else "natsl_gdn_walk"
            _lib.call(entry, *args, _lib.ptr(start),
                      _lib.ptr(last_types if want_start else None), last_code, 2 * HN, *dims)
        return o, ht, inter
    if mamba_fused:
        o = None if skip_out else torch.empty(B, T, H, V, dtype=BF16, device=dev)
        _lib.call("natsl_mamba_walk_fused_ex", None if skip_out else q.data_ptr(), k.data_ptr(), v.data_ptr(), gcs.data_ptr(),
                  tables.types_i.data_ptr(), tables.indices.data_ptr(), tables.n_blocks.data_ptr(), _lib.ptr(h0),
                  _lib.ptr(o), _lib.ptr(ht), _lib.ptr(start), _lib.ptr(last_types if want_start else None), last_code,
                  2 * HN, B, T, H, HN, K, V, nbs, float(scale), flags, st)
        return o, ht, (dict(gcs=gcs) if skip_out else inter)
    state_only = skip_out and ht is not None and not return_intermediates
    h = None if state_only else torch.empty(B, NT, H, K, V, dtype=BF16, device=dev)
    carry = None if state_only else torch.empty(B, NT, H, dtype=torch.float32, device=dev)
    _lib.call("natsl_linear_fwd_h", rule, k.data_ptr(), _lib.ptr(w), u.data_ptr(), gcs.data_ptr(), _lib.ptr(krstd),
              tables.types_i.data_ptr(), tables.indices.data_ptr(), tables.n_blocks.data_ptr(), _lib.ptr(h0),
              _lib.ptr(h), _lib.ptr(carry), _lib.ptr(ht), B, T, H, HN, K, V, nbs, flags, st)
    inter = dict(w=w, u=u, gcs=gcs, k_rstd=krstd, h=h, carry=carry) if return_intermediates else None
    if skip_out:
        return None, ht, (inter or dict(gcs=gcs))
    o = torch.empty(B, T, H, V, dtype=BF16, device=dev)
    _lib.call("natsl_linear_fwd_o", rule, q.data_ptr(), k.data_ptr(), _lib.ptr(w), u.data_ptr(), gcs.data_ptr(),
              _lib.ptr(krstd), h.data_ptr(), carry.data_ptr(), o.data_ptr(), B, T, H, K, V, float(scale),
              int(use_l2norm and rule == _lib.RULE_GDN) | (0 if own_chunk else 2), st)
    return o, ht, inter


def tables_from_flat(flat, B: int, TN: int, HN: int, T: int, nbs: int) -> SelectionTables:
    """Views of the tables ``hybrid_fwd`` built into one buffer (without the compact chunk list and its offsets)."""
    NT, NTq = cdiv(T, 64), cdiv(T, _lib.ATTN_BT)
    sizes = [B * TN * HN * 2, B * TN * HN * 2, B * HN * 2, B * HN, B * NT * HN, B * NTq * HN]
    ti, ix, nb, nc, sh, an = torch.split(flat, sizes)
    return SelectionTables(types_i=ti.view(B, TN, HN, 2), indices=ix.view(B, TN, HN, 2), n_blocks=nb.view(B, HN, 2), n_chunks_lin=nc,
                           offsets=None, chunk_indices=None, starting_h_idx=sh.view(B, NT, HN), attn_n_iters=an.view(B, NTq, HN),
                           T=T, nats_block_size=nbs)


def hybrid_options(pairs: int) -> int:
    """``options`` of the native op and layer calls for this many (batch, head) pairs of the linear branch."""
    return ((0 if PREP_TC else _lib.HYBRID_PREP_MMA) | (_lib.HYBRID_WALK_MMA if pairs <= WALK_MMA_MAX_HEADS else 0)
            | (_lib.HYBRID_WALK_VSPLIT if WALK_VSPLIT else 0) | (0 if LINEAR_BRANCH_PRIORITY else _lib.HYBRID_PLAIN_PRIORITY))


_hybrid_ws: dict = {}


def hybrid_fwd(rule: int, q_attn, k_attn, v_attn, q, k, v, g, beta, types, nbs: int, scale_attn: float, scale_lin: float, h0,
               own_attn: bool, decay: bool, use_l2norm: bool, want_ht: bool, want_start: bool = False, last_types=None):
    """Tables and both branches in one native call (bf16 tensors with head dims of ``walks_with_state``, or fp32 tensors;
    own-block linear attention).  -> (o_lin, o_attn, lse, ht, start, flat tables for ``tables_from_flat``)."""
    for t_ in (q_attn, k_attn, v_attn, q, k, v):
        _need(t_.dim() == 4, "q, k, v must be [B, T, H, D]")
        _need(t_.is_cuda and t_.device == q.device, "q, k, v of both branches must be on one CUDA device")
    _need(q.dtype == k.dtype == v.dtype and q_attn.dtype == k_attn.dtype == v_attn.dtype, "q, k, v must share a dtype", TypeError)
    fp32 = q.dtype == torch.float32
    _need(q_attn.dtype == q.dtype or (fp32 and q_attn.dtype == BF16), f"softmax branch in {q_attn.dtype} beside a linear branch "
          f"in {q.dtype}", TypeError)
    _need(fp32 or q.dtype == BF16, f"unsupported dtype {q.dtype} (fp32 or bf16)", TypeError)
    _need(not (fp32 and want_start), "the block-start state needs bf16 tensors", TypeError)
    q_attn, k_attn, v_attn, q, k, v = (t_.contiguous() for t_ in (q_attn, k_attn, v_attn, q, k, v))
    B, T, H, K = map(int, q.shape)                           # a trace gives sizes as tensors
    V, HQ, DK, HKV, DV = map(int, (v.shape[3], q_attn.shape[2], q_attn.shape[3], k_attn.shape[2], v_attn.shape[3]))
    dev = q.device
    TN, HN = map(int, types.shape[1:3])
    _need(tuple(k.shape) == (B, T, H, K), f"linear branch: q {tuple(q.shape)} and k {tuple(k.shape)} differ")
    _need(tuple(v.shape) == (B, T, H, V), f"linear branch: k {tuple(k.shape)} and v {tuple(v.shape)} differ in length or heads")
    _need(tuple(q_attn.shape) == (B, T, HQ, DK) and tuple(k_attn.shape) == (B, T, HKV, DK) and tuple(v_attn.shape) == (B, T, HKV, DV),
          f"softmax branch: q {tuple(q_attn.shape)}, k {tuple(k_attn.shape)}, v {tuple(v_attn.shape)} do not match")
    _need(HQ % HKV == 0, f"softmax branch: {HQ} query heads over {HKV} key/value heads")
    _need(tuple(g.shape) == (B, T, H) and g.device == dev, f"g must be [B,T,H] = {(B, T, H)} on {dev}, got {tuple(g.shape)}")
    if not types.is_cuda:
        raise ValueError("nats_block_types must be a CUDA tensor (there is no CPU path)")
    if types.dtype not in _TYPE_CODES:
        raise TypeError(f"unsupported nats_block_types dtype {types.dtype}")
    if types.shape[3] != 2:
        raise NotImplementedError("selection tables are specified for n_ops == 2")
    _need(types.shape[0] == B and types.device == dev, "the block types were made for another batch or device")
    _need(TN == cdiv(T, nbs), f"{TN} blocks of {nbs} tokens do not cover T={T}")
    _need(H % HN == 0 and HQ % HN == 0, f"{H} / {HQ} heads over {HN} selection heads")
    g = g.float().contiguous()
    types = types.contiguous()
    a = _lib.HybridArgs()
    if rule == _lib.RULE_GDN:
        _need(beta is not None, "the gated delta rule needs beta")
        _need(tuple(beta.shape) == (B, T, H) and beta.device == dev, f"beta must be [B,T,H] = {(B, T, H)} on {dev}")
        beta = beta.float().contiguous() if fp32 else beta.contiguous()
        _need(beta.dtype in (BF16, torch.float32), "beta must be bf16 or fp32", TypeError)
        a.beta, a.beta_dtype = beta.data_ptr(), _dt_code(beta)
    if h0 is not None:
        h0 = aligned(h0.float().contiguous())
        _need(tuple(h0.shape) == (B, H, K, V) and h0.device == dev, f"initial state must be [B,H,K,V] on {dev}, got {tuple(h0.shape)}")
        a.h0 = h0.data_ptr()
    o_lin = torch.empty(B, T, H, V, dtype=q.dtype, device=dev)
    o_attn = torch.empty(B, T, HQ, DV, dtype=q_attn.dtype, device=dev)
    lse = torch.empty(B, T, HQ, dtype=torch.float32, device=dev)
    ht = torch.empty(B, H, K, V, dtype=torch.float32, device=dev) if want_ht else None
    start = torch.empty(B, H, K, V, dtype=torch.float32, device=dev) if want_start else None
    if want_start and T % nbs == 0:
        _need(last_types is not None and tuple(last_types.shape) == (B, HN, 2) and last_types.device == dev,
              f"a complete last block needs its types [B,HN,2] on {dev}")
        last_types = (last_types if last_types.dtype in (BF16, torch.float32) else last_types.float()).contiguous()
        a.last_types, a.last_dtype, a.last_stride = last_types.data_ptr(), _dt_code(last_types), 2 * HN
    NT, NTq = cdiv(T, 64), cdiv(T, _lib.ATTN_BT)
    nt = B * TN * HN * 2
    flat = torch.empty(2 * nt + 3 * B * HN + B * (NT + NTq) * HN, dtype=torch.int32, device=dev)
    p = flat.data_ptr()
    a.types_i, a.indices, a.n_blocks = p, p + 4 * nt, p + 8 * nt
    a.n_chunks_lin = a.n_blocks + 8 * B * HN
    a.starting_h_idx = a.n_chunks_lin + 4 * B * HN
    a.attn_n_iters = a.starting_h_idx + 4 * B * NT * HN
    a.B, a.T, a.H, a.HN, a.K, a.V, a.HQ, a.HKV, a.DK, a.DV, a.nbs, a.rule = B, T, H, HN, K, V, HQ, HKV, DK, DV, nbs, rule
    a.types_dtype = _TYPE_CODES[types.dtype]
    a.own_attn, a.decay, a.use_l2norm = int(own_attn), int(decay), int(use_l2norm)
    a.options = hybrid_options(B * H)
    a.scale_attn, a.scale_lin = float(scale_attn), float(scale_lin)
    a.q_attn, a.k_attn, a.v_attn, a.q, a.k, a.v = (t_.data_ptr() for t_ in (q_attn, k_attn, v_attn, q, k, v))
    a.g, a.types, a.o_attn, a.lse, a.o_lin = g.data_ptr(), types.data_ptr(), o_attn.data_ptr(), lse.data_ptr(), o_lin.data_ptr()
    a.ht, a.hstart = _lib.ptr(ht), _lib.ptr(start)
    if fp32:
        a.options |= _lib.HYBRID_FP32 | (_lib.HYBRID_ATTN_BF16 if q_attn.dtype == BF16 else 0)
        with device_guard(dev):
            _lib.call("natsl_hybrid_forward", ctypes.byref(a), current_stream_ptr(dev))
        return o_lin, o_attn, lse, ht, start, flat
    key = (rule, B, T, H, K, V)
    need = _hybrid_ws.get(key)
    if need is None:
        if len(_hybrid_ws) > 1024:
            _hybrid_ws.clear()
        need = _hybrid_ws[key] = _lib.load().natsl_hybrid_workspace_bytes(ctypes.byref(a))
    ws = torch.empty(need, dtype=torch.uint8, device=dev)
    a.workspace, a.workspace_bytes = ws.data_ptr(), need
    with device_guard(dev):
        _lib.call("natsl_hybrid_forward", ctypes.byref(a), current_stream_ptr(dev))
    return o_lin, o_attn, lse, ht, start, flat


def _dt_code(t):
    if t.dtype == torch.float32:
        return _lib.DT_F32
    if t.dtype == BF16:
        return _lib.DT_BF16
    raise TypeError(f"unsupported dtype {t.dtype} (fp32 or bf16)")


def linear_recurrent(rule: int, q, k, v, g, beta, tables: SelectionTables, scale: float, h0, decay: bool,
                     use_l2norm: bool):
    """Reference-precision linear branch: token recurrence with re-roll (fp32 math; fp32 or bf16 tensors).
    Returns (o, ht, hstart): output, state after the last selected block, block-start state at the end."""
    _need(q.dtype == k.dtype == v.dtype, "q, k, v must share a dtype", TypeError)
    code = _dt_code(q)
    _check_qkv(q, k, v, tables, "linear branch (recurrent form)", same_heads=True)
    q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
    B, T, H, K = q.shape
    V = v.shape[3]
    dev = q.device
    _need(tables.T == T, f"tables were built for T={tables.T}, the sequence has T={T}")
    _need(tuple(g.shape) == (B, T, H), f"g must be [B,T,H] = {(B, T, H)}, got {tuple(g.shape)}")
    _need(beta is None or tuple(beta.shape) == (B, T, H), f"beta must be [B,T,H] = {(B, T, H)}")
    g = g.float().contiguous()
    if beta is not None:
        beta = beta.to(q.dtype).contiguous()
    if h0 is not None:
        h0 = h0.float().contiguous()
    o = torch.empty(B, T, H, V, dtype=q.dtype, device=dev)
    ht = torch.empty(B, H, K, V, dtype=torch.float32, device=dev)
    hstart = torch.empty_like(ht)
    _lib.call("natsl_linear_recurrent_fwd", rule, code, q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(),
              _lib.ptr(beta), tables.types_i.data_ptr(), _lib.ptr(h0), o.data_ptr(), ht.data_ptr(), hstart.data_ptr(),
              B, T, H, tables.types_i.shape[2], K, V, tables.nats_block_size, float(scale),
              _lib.FLAG_DECAY_SKIPPED if decay else 0, int(use_l2norm), current_stream_ptr(dev))
    return o, ht, hstart


def linear_recurrent_step(rule: int, q, k, v, g, beta, block_types, state, state_block_start, g_block, t_off: int, nbs: int,
                          scale: float, decay: bool, use_l2norm: bool):
    """Decoding step of the linear branch: the T new tokens continue a block that already holds ``t_off`` tokens.
    ``block_types`` [B, cdiv(t_off + T, nbs), HN, 2] (0/1 floats or ints) are read only where a block ends inside the
    call.  -> (o [B,T,H,V], new current state, new block-start state), states fp32 [B,H,K,V]."""
    code = _dt_code(q)
    q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
    B, T, H, K = q.shape
    V = v.shape[3]
    dev = q.device
    g = g.float().contiguous()
    if beta is not None:
        beta = beta.to(q.dtype).contiguous()
    types_i = torch.round(block_types.float()).to(torch.int32).contiguous()
    _need(types_i.shape[1] == cdiv(t_off + T, nbs) and types_i.shape[3] == 2, "block_types must cover the blocks the step touches")
    state = state.float().contiguous()
    start = state_block_start.float().contiguous()
    g_block = g_block.float().contiguous()
    _need(tuple(state.shape) == (B, H, K, V) and tuple(start.shape) == (B, H, K, V) and tuple(g_block.shape) == (B, H),
          "states must be [B,H,K,V] and the block decay [B,H]")
    o = torch.empty(B, T, H, V, dtype=q.dtype, device=dev)
    new_state, new_start = torch.empty_like(state), torch.empty_like(start)
    _lib.call("natsl_linear_recurrent_step", rule, code, q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr(), _lib.ptr(beta),
              types_i.data_ptr(), state.data_ptr(), start.data_ptr(), g_block.data_ptr(), int(t_off), o.data_ptr(),
              new_state.data_ptr(), new_start.data_ptr(), B, T, H, types_i.shape[2], K, V, int(nbs), float(scale),
              _lib.FLAG_DECAY_SKIPPED if decay else 0, int(use_l2norm), current_stream_ptr(dev))
    return o, new_state, new_start


# ------------------------------------------------------------------------------------------------ backward
class StageTimer:
    """Optional per-stage device timing of the backward pass: CUDA events on the launching stream around every C-ABI
    call; ``result()`` synchronises and returns {stage: milliseconds} (summed over repeated calls)."""

    def __init__(self):
        self.events = []

    def call(self, stage: str, name: str, *args):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        _lib.call(name, *args)
        e1.record()
        self.events.append((stage, e0, e1))

    def result(self) -> dict:
        torch.cuda.synchronize()
        out = {}
        for stage, e0, e1 in self.events:
            out[stage] = out.get(stage, 0.0) + e0.elapsed_time(e1)
        return out


def _call(timer, stage, name, *args):
    if timer is None:
        _lib.call(name, *args)
    else:
        timer.call(stage, name, *args)


def attn_bwd(q, k, v, o, lse, do, tables: SelectionTables, scale: float, own_chunk: bool, reference_compat: bool = False,
             timer: StageTimer | None = None, per_tile: bool = False):
    """Backward of the softmax branch.  -> (dq, dk, dv bf16, dnats_attn [B,TN,HN] fp32): ``dnats_attn`` is the sum of the
    score gradients of the keys of a softmax-selected block over the queries of later blocks, summed over the heads
    of a selection group and zero for the other blocks (src/nats/ops/attns/attns.py:922, 975-978, 1625-1629, 1749-1755).
    ``reference_compat``: leave out every own-block term like the reference's default backward.  ``per_tile``: the sums of the
    key tiles [B,NT,HQ], whatever their blocks' types, in the place of ``dnats_attn``."""
    for t_ in (q, k, v, o, do):
        _need(t_.dtype == BF16, "softmax-branch backward needs bf16 tensors", TypeError)
    _check_qkv(q, k, v, tables, "softmax branch (backward)", same_heads=False)
    q, k, v, o, do, lse = (t_.contiguous() for t_ in (q, k, v, o, do, lse))
    B, T, HQ, DK = q.shape
    HKV, DV = k.shape[2], v.shape[3]
    _need(k.shape[1] == T and tables.T == T, "q, k and the tables must cover the same sequence")
    _need(tuple(do.shape) == (B, T, HQ, DV) and tuple(o.shape) == (B, T, HQ, DV), "o and do must be [B,T,HQ,DV]")
    TN, HN = tables.types_i.shape[1], tables.types_i.shape[2]
    nbs = tables.nats_block_size
    NT = cdiv(T, 64)
    dev = q.device
    dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)
    delta = torch.empty(B, T, HQ, dtype=torch.float32, device=dev)
    part = torch.empty(B, NT, HQ, dtype=torch.float32, device=dev)
    flags = (_lib.FLAG_ATTN_OWN_CHUNK if own_chunk else 0) | (_lib.FLAG_BWD_REFERENCE_COMPAT if reference_compat else 0)
    _call(timer, "attn_bwd", "natsl_attn_bwd", q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), do.data_ptr(), lse.data_ptr(),
              tables.types_i.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), delta.data_ptr(), part.data_ptr(),
              B, T, HQ, HKV, HN, DK, DV, nbs, float(scale), flags, current_stream_ptr(dev))
    if per_tile:
        return dq, dk, dv, part
    cpb = nbs // 64
    if NT != TN * cpb:                                        # ragged last block: pad the tile axis
        part = torch.nn.functional.pad(part, (0, 0, 0, TN * cpb - NT))
    per_block = part.view(B, TN, cpb, HN, HQ // HN).sum((2, 4))
    dnats = per_block * (tables.types_i[..., 0] != 0)
    return dq, dk, dv, dnats


def linear_bwd(rule: int, q, k, v, g, beta, tables: SelectionTables, scale: float, h0, decay: bool, use_l2norm: bool,
               do, dht=None, invalid_dnats: bool = True, trailing_quirk: bool = True, return_intermediates: bool = False,
               timer: StageTimer | None = None, per_tile: bool = False, onto=None):
    """Backward of the linear branch (block size 64).  Recomputes the forward's preparation and recurrence, then runs the
    five backward stages.  -> dict(dq, dk, dv bf16; dg fp32; dbeta fp32 or None; dh0 fp32 or None; dnats [B,NT,HN] fp32
    = the reference's dnats column for the linear branch, src/nats/ops/common/chunk_o.py:440-443, 459-492, 1568-1575; with
    ``per_tile`` [B,NT,H], per head).  ``onto``: gradients of q, k and (delta rule) v (or None) to add to, in place; a separate sum of two
    [8,4096,16,128] tensors is a pass of 59 us."""
    gdn = rule == _lib.RULE_GDN
    for t_ in (q, k, v, do):
        _need(t_.dtype == BF16, "linear-branch backward needs bf16 tensors", TypeError)
    _check_qkv(q, k, v, tables, "linear branch (backward)", same_heads=True)
    _need(tables.nats_block_size == 64, "the backward pass is built for nats_block_size = 64", NotImplementedError)
    q, k, v, do = q.contiguous(), k.contiguous(), v.contiguous(), do.contiguous()
    B, T, H, K = q.shape
    V = v.shape[3]
    _need(K in (64, 128) and V in (64, 128), f"backward head dims K={K} V={V}: 64 or 128 each", NotImplementedError)
    _need(tables.T == T, f"tables were built for T={tables.T}, the sequence has T={T}")
    dev = q.device
    HN = tables.types_i.shape[2]
    NT = cdiv(T, 64)
    st = current_stream_ptr(dev)
    g = g.float().contiguous()
    bf = dict(dtype=BF16, device=dev)
    f32 = dict(dtype=torch.float32, device=dev)
    gcs = torch.empty(B, T, H, **f32)
    # ---- forward recompute: w, u, gcs; the state and the carried decay every chunk reads
    if gdn:
        beta = beta.contiguous()
        _need(beta.dtype in (BF16, torch.float32), "beta must be bf16 or fp32", TypeError)
        w, u = torch.empty(B, T, H, K, **bf), torch.empty(B, T, H, V, **bf)
        krs0 = torch.empty(B, T, H, **f32)
        _call(timer, "recompute_prep", prep_entry(K, V), None, k.data_ptr(), v.data_ptr(), g.data_ptr(), beta.data_ptr(),
                  _lib.DT_BF16 if beta.dtype == BF16 else _lib.DT_F32, w.data_ptr(), u.data_ptr(), gcs.data_ptr(),
                  krs0.data_ptr(), None, None, B, T, H, K, V, int(use_l2norm), st)
    else:
        w, u, krs0 = None, v, None
        _call(timer, "recompute_prep", "natsl_chunk_local_cumsum", g.data_ptr(), gcs.data_ptr(), B, T, H, st)
    if h0 is not None:
        h0 = h0.float().contiguous()
    flags = (_lib.FLAG_DECAY_SKIPPED if decay else 0) | (0 if trailing_quirk else _lib.FLAG_NO_TRAILING_QUIRK)
    h = torch.empty(B, NT, H, K, V, **bf)
    carry = torch.empty(B, NT, H, **f32)
    _call(timer, "recompute_scan", "natsl_linear_fwd_h", rule, k.data_ptr(), _lib.ptr(w), u.data_ptr(), gcs.data_ptr(), _lib.ptr(krs0),
              tables.types_i.data_ptr(), tables.indices.data_ptr(), tables.n_blocks.data_ptr(), _lib.ptr(h0),
              h.data_ptr(), carry.data_ptr(), None, B, T, H, HN, K, V, 64, flags, st)
    # ---- 1: normalised q, k and the chunk-local part of dv'
    l2 = bool(use_l2norm and gdn)
    if l2:
        qn, kn = torch.empty_like(q), torch.empty_like(k)
        qrs, krs = torch.empty(B, T, H, **f32), torch.empty(B, T, H, **f32)
    else:
        qn, kn, qrs, krs = q, k, None, None
    dvl = torch.empty(B, T, H, V, **bf)
    _call(timer, "bwd_pre", "natsl_linear_bwd_pre", q.data_ptr(), k.data_ptr(), do.data_ptr(), gcs.data_ptr(), _lib.ptr(qn if l2 else None),
              _lib.ptr(kn if l2 else None), _lib.ptr(qrs), _lib.ptr(krs), dvl.data_ptr(), B, T, H, K, V, float(scale), int(l2), st)
    # ---- 2: reverse walk
    dS_all = torch.empty(B, NT, H, K, V, **bf)
    dvp = torch.empty(B, T, H, V, **bf)
    dh0 = torch.empty(B, H, K, V, **f32) if h0 is not None else None
    if dht is not None:
        dht = dht.float().contiguous()
    _call(timer, "bwd_dh", "natsl_linear_bwd_dh", rule, qn.data_ptr(), kn.data_ptr(), _lib.ptr(w), do.data_ptr(), dvl.data_ptr(),
              gcs.data_ptr(), carry.data_ptr(), tables.types_i.data_ptr(), tables.indices.data_ptr(),
              tables.n_blocks.data_ptr(), _lib.ptr(dht), dS_all.data_ptr(), dvp.data_ptr(), _lib.ptr(dh0), B, T, H, HN, K, V,
              float(scale), st)
    # ---- 3: everything that contracts with the state or its gradient
    vp = torch.empty(B, T, H, V, **bf) if gdn else v
    dw = torch.empty(B, T, H, K, **bf) if gdn else None
    dq1, dk1 = torch.empty(B, T, H, K, **bf), torch.empty(B, T, H, K, **bf)
    dkd = torch.empty(B, T, H, **f32)
    scal = torch.empty(B, NT, H, 4, **f32)
    dn_lin = torch.empty(B, NT, H, **f32)
    _call(timer, "bwd_state", "natsl_linear_bwd_state", rule, kn.data_ptr(), _lib.ptr(v if gdn else None), _lib.ptr(w), u.data_ptr(),
              do.data_ptr(), dvp.data_ptr(), gcs.data_ptr(), h.data_ptr(), carry.data_ptr(), dS_all.data_ptr(),
              tables.types_i.data_ptr(), tables.indices.data_ptr(), tables.n_blocks.data_ptr(),
              tables.starting_h_idx.data_ptr(), _lib.ptr(vp if gdn else None), _lib.ptr(dw), dq1.data_ptr(), dk1.data_ptr(),
              dkd.data_ptr(), scal.data_ptr(), dn_lin.data_ptr(), B, T, H, HN, K, V, float(scale), int(invalid_dnats), st)
    # ---- 4: the 64 x 64 part, the WY transform and the l2 norm
    bits = 0
    if onto is None:
        dq, dk, dv = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v) if gdn else dvp
    else:
        _need(gdn or onto[2] is None, "Mamba2's dv is not added to another gradient", NotImplementedError)
        for i, (d, x) in enumerate(zip(onto, (q, k, v))):
            _need(d is None or (d.shape == x.shape and d.dtype == BF16 and d.is_contiguous()), "a gradient to add to has another form")
            bits |= 0 if d is None else 1 << i
        dq, dk, dv = (torch.empty_like(x) if d is None else d for d, x in zip(onto, (q, k, v)))
        if not gdn:
            dv = dvp
    dbeta = torch.empty(B, T, H, **f32) if gdn else None
    dg_tok = torch.empty(B, T, H, **f32)
    _call(timer, "bwd_intra", "natsl_linear_bwd_intra_onto", rule, qn.data_ptr(), kn.data_ptr(), _lib.ptr(v if gdn else None), _lib.ptr(w),
              _lib.ptr(u if gdn else None), vp.data_ptr(), _lib.ptr(dvp if gdn else None), _lib.ptr(dw), do.data_ptr(),
              dq1.data_ptr(), dk1.data_ptr(), gcs.data_ptr(), _lib.ptr(beta if gdn else None),
              _lib.DT_BF16 if (gdn and beta.dtype == BF16) else _lib.DT_F32, _lib.ptr(qrs), _lib.ptr(krs), dkd.data_ptr(),
              tables.types_i.data_ptr(), dq.data_ptr(), dk.data_ptr(), _lib.ptr(dv if gdn else None), _lib.ptr(dbeta),
              dg_tok.data_ptr(), scal.data_ptr(), B, T, H, HN, K, V, float(scale), int(l2), bits, st)
    # ---- 5: decay gradients
    dg = torch.empty(B, T, H, **f32)
    _call(timer, "bwd_dg", "natsl_linear_bwd_dg", dg_tok.data_ptr(), scal.data_ptr(), tables.types_i.data_ptr(), tables.indices.data_ptr(),
              tables.n_blocks.data_ptr(), dg.data_ptr(), B, T, H, HN, flags, st)
    dnats = dn_lin if per_tile else dn_lin.view(B, NT, HN, H // HN).sum(-1)
    out = dict(dq=dq, dk=dk, dv=dv, dg=dg, dbeta=dbeta, dh0=dh0, dnats=dnats)
    if return_intermediates:
        out.update(dS=dS_all, dvp=dvp, dw=dw, vp=vp, h=h, carry=carry, gcs=gcs, w=w, u=u)
    return out
