"""Decoding state of the NAtSL layers: what a layer keeps between a prefill and the following single-token steps.

The reference's ``NAtSLayerCache`` / ``NAtSCache`` (src/nats/models/utils.py:34-670, 671-853) hold, per layer, the softmax
branch's keys and values, the linear state and the state at the start of the current block, the convolution tails and
the running sum of the layer input over the current block (the selection of a block is decided when its last token has
arrived).  This is a compact restatement of the same bookkeeping for batches without padding:

* keys / values of every token are kept together with the 0/1 types of the finished blocks; visibility of a key for a
  query is evaluated from the types (``generate_msk``), the same object the reference's ``generate_msk`` (:209-287) builds.
  (The reference additionally drops the keys of unselected blocks to save memory; outputs do not depend on that.)
  The rows live in buffers that grow by a quarter at a time, so that a decoding token writes its own row only.
* ``state`` / ``state_block_start`` / ``g_block``: the current recurrent state, the state the current block started from
  and the log decay accumulated in the current block (re-roll at the block end needs all three).

Single-token steps update these tensors in place, but never one that a caller has seen: reading or setting ``state`` and the
like hands the tensor out, and the next step works on copies.  ``copy.copy`` of a layer cache gives an independent
continuation (one prompt, several completions): the small tensors are cloned, the key/value rows are shared until either
side appends.
"""
from __future__ import annotations

from typing import List, Optional

import torch

from . import _lib
from .nats_util import current_stream_ptr, device_guard, transforms_active


_IN_PLACE = ("_state", "_state_block_start", "_g_block", "_pool_sum", "_conv_state")


def _seen(name: str, doc: str) -> property:
    """Attribute whose tensor belongs to the caller as well once it has been read or set."""
    def get(self):
        self._handed_out = True
        return getattr(self, name)

    def put(self, value):
        self._handed_out = True
        setattr(self, name, value)

    return property(get, put, doc=doc)


def _copy(t):
    return None if t is None else tuple(map(_copy, t)) if isinstance(t, tuple) else t.clone()


def _copy_rows(dst: torch.Tensor, src: torch.Tensor, n: int) -> None:
    """dst[:, :n] = src[:, :n] of two [B, rows, ...] tensors, as one kernel where both are plain device memory and nothing
    (a transform, a trace, a compiler) has to see the copy."""
    if (src.is_cuda and not torch.compiler.is_compiling() and not transforms_active() and n > 0 and src.numel()
            and not (src.requires_grad and torch.is_grad_enabled()) and src.is_contiguous() and dst.is_contiguous()
            and dst.dtype == src.dtype and dst.device == src.device):
        B = src.shape[0]
        from_pitch, to_pitch = src.numel() // B * src.element_size(), dst.numel() // B * dst.element_size()
        size, to, at = from_pitch // src.shape[1] * n, dst.data_ptr(), src.data_ptr()
        if B <= 65535 and (size | from_pitch | to_pitch | to | at) % 16 == 0:
            with device_guard(src.device):
                _lib.call("natsl_copy_batches", to, at, B, size, to_pitch, from_pitch, current_stream_ptr(src.device))
            return
    dst[:, :n].copy_(src[:, :n])


class NAtSLayerCache:
    state = _seen("_state", "[B, H, K, V] fp32: current state")
    state_block_start = _seen("_state_block_start", "[B, H, K, V] fp32: state the current block started from")
    g_block = _seen("_g_block", "[B, H] fp32: log decay accumulated in the current block")
    pool_sum = _seen("_pool_sum", "[B, D] fp32: sum of the layer input over the current block")
    conv_state = _seen("_conv_state", "(q, k, v) tails of the short convolutions")

    def __init__(self, nats_block_size: int = 64):
        self.nats_block_size = nats_block_size
        self.n_tokens = 0                               # tokens seen so far
        self._k_buf: Optional[torch.Tensor] = None      # [B, capacity, HKV, DK]
        self._v_buf: Optional[torch.Tensor] = None      # [B, capacity, HKV, DV]
        self._n_kv = 0                                  # rows of the buffers in use
        self._kv_shared = False                         # another cache reads the same buffers
        self._step = None                               # argument block and workspace of the single-token steps
        self.block_types: Optional[torch.Tensor] = None  # [B, finished blocks, HN, 2] sampled types
        for name in _IN_PLACE:
            setattr(self, name, None)
        self._handed_out = False                         # a caller may hold one of these tensors

    def __copy__(self):
        new = type(self).__new__(type(self))
        new.__dict__.update(self.__dict__)
        new._handed_out = True
        new.own_state()
        new._step = None
        self._kv_shared = new._kv_shared = True
        return new

    def __getstate__(self):
        return dict(self.__dict__, _step=None)             # holds addresses: not for another process

    def __setstate__(self, saved):
        self.__init__(saved["nats_block_size"])
        for name, value in saved.items():                  # also those of caches saved with plain k_attn, state, ... attributes
            setattr(self, name, value)

    def own_state(self) -> None:
        """Makes the tensors that a step updates in place this cache's own: copies them if they have been handed out."""
        if self._handed_out:
            for name in _IN_PLACE:
                setattr(self, name, _copy(getattr(self, name)))
            self._handed_out = False

    def set_state(self, state, state_block_start, g_block, pool_sum, conv_state) -> None:
        """Takes over tensors that nobody else holds."""
        self._state, self._state_block_start, self._g_block, self._pool_sum, self._conv_state = (state, state_block_start, g_block,
                                                                                                pool_sum, conv_state)
        self._handed_out = False

    @property
    def k_attn(self) -> Optional[torch.Tensor]:
        """Keys of every token so far [B, n_tokens, HKV, DK]."""
        return None if self._k_buf is None else self._k_buf[:, :self._n_kv]

    @k_attn.setter
    def k_attn(self, k: Optional[torch.Tensor]) -> None:
        self._k_buf, self._n_kv = k, 0 if k is None else k.shape[1]

    @property
    def v_attn(self) -> Optional[torch.Tensor]:
        """Values of every token so far [B, n_tokens, HKV, DV]."""
        return None if self._v_buf is None else self._v_buf[:, :self._n_kv]

    @v_attn.setter
    def v_attn(self, v: Optional[torch.Tensor]) -> None:
        self._v_buf, self._n_kv = v, 0 if v is None else v.shape[1]

    @property
    def n_tokens_in_nats_block(self) -> int:
        return self.n_tokens % self.nats_block_size

    @property
    def n_finished_blocks(self) -> int:
        return self.n_tokens // self.nats_block_size

    def reserve_kv(self, n: int) -> None:
        """Makes room for ``n`` more key/value rows that nobody else reads."""
        cap = self._k_buf.shape[1]
        if (self._n_kv + n <= cap and cap == self._v_buf.shape[1] and not self._kv_shared and self._k_buf.is_contiguous()
                and self._v_buf.is_contiguous()):
            return
        need = self._n_kv + n
        cap = -(-(need + max(256, need // 4)) // 64) * 64
        for name in ("_k_buf", "_v_buf"):
            old = getattr(self, name)
            buf = old.new_empty((old.shape[0], cap) + tuple(old.shape[2:]))
            _copy_rows(buf, old, self._n_kv)
            setattr(self, name, buf)
        self._kv_shared = False

    def append_kv(self, k: torch.Tensor, v: torch.Tensor) -> None:
        if self._k_buf is None:
            self._k_buf, self._v_buf, self._n_kv = k, v, k.shape[1]
            return
        n = k.shape[1]
        self.reserve_kv(n)
        self._k_buf[:, self._n_kv:self._n_kv + n].copy_(k)
        self._v_buf[:, self._n_kv:self._n_kv + n].copy_(v)
        self._n_kv += n

    def append_types(self, types: torch.Tensor) -> None:
        self.block_types = types if self.block_types is None else torch.cat([self.block_types, types], 1)

    def generate_msk(self, n_data: int, HQ: int, own_chunk: bool = True) -> torch.Tensor:
        """Boolean mask [B, HQ, n_data, n_keys] for the last ``n_data`` tokens as queries over all cached keys (the new
        tokens' keys already appended): a key is visible when its block is finished, softmax-selected and lies before
        the query's block, or when both are in the same block and the key is not later than the query."""
        nbs = self.nats_block_size
        n_keys = self.k_attn.shape[1]
        dev = self.k_attn.device
        B = self.k_attn.shape[0]
        t = torch.arange(n_keys - n_data, n_keys, device=dev)
        s = torch.arange(n_keys, device=dev)
        blk_t, blk_s = t // nbs, s // nbs
        n_done = 0 if self.block_types is None else self.block_types.shape[1]
        if n_done:
            HN = self.block_types.shape[2]
            sel = (self.block_types[..., 0] > 0.5).repeat_interleave(HQ // HN, dim=2).permute(0, 2, 1)     # [B,HQ,n_done]
            col_sel = torch.zeros(B, HQ, n_keys, dtype=torch.bool, device=dev)
            inside = blk_s < n_done
            col_sel[:, :, inside] = sel[:, :, blk_s[inside]]
        else:
            col_sel = torch.zeros(B, HQ, n_keys, dtype=torch.bool, device=dev)
        past = blk_s[None, :] < blk_t[:, None]
        m = col_sel[:, :, None, :] & past[None, None]
        if own_chunk:
            own = (blk_s[None, :] == blk_t[:, None]) & (s[None, :] <= t[:, None])
            m = m | own[None, None]
        return m


class NAtSCache:
    """One ``NAtSLayerCache`` per layer, indexed by ``layer_idx`` (created on first use)."""

    def __init__(self):
        self.layers: List[NAtSLayerCache] = []

    def __len__(self) -> int:
        return len(self.layers)

    def __getitem__(self, layer_idx: int) -> NAtSLayerCache:
        return self.layers[layer_idx]

    def layer(self, layer_idx: int, nats_block_size: int) -> NAtSLayerCache:
        while len(self.layers) <= layer_idx:
            self.layers.append(NAtSLayerCache(nats_block_size))
        return self.layers[layer_idx]

    def get_seq_length(self, layer_idx: int = 0) -> int:
        return self.layers[layer_idx].n_tokens if len(self.layers) > layer_idx else 0
