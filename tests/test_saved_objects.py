"""Caches and layers that were pickled with plain attributes load, and today's round-trip."""
import copy
import pickle

import pytest
import torch

import neuralattentionsearchlinear_b200 as nat
from neuralattentionsearchlinear_b200.cache import NAtSLayerCache


def test_cache_saved_with_plain_attributes():
    tensors = dict(k_attn=torch.randn(2, 70, 4, 8), v_attn=torch.randn(2, 70, 4, 8), block_types=torch.ones(2, 1, 4, 2),
                   state=torch.randn(2, 4, 8, 8), state_block_start=torch.randn(2, 4, 8, 8), g_block=torch.randn(2, 4),
                   pool_sum=torch.randn(2, 16))
    cache = NAtSLayerCache.__new__(NAtSLayerCache)
    cache.__setstate__(dict(nats_block_size=64, n_tokens=70, conv_state=(torch.ones(1),) * 3, **tensors))
    for copied in (cache, pickle.loads(pickle.dumps(cache)), copy.deepcopy(cache), copy.copy(cache)):
        assert copied.n_tokens == 70 and copied.n_tokens_in_nats_block == 6 and len(copied.conv_state) == 3
        for name, t in tensors.items():
            assert torch.equal(getattr(copied, name), t), name
    cache.append_kv(torch.ones(2, 1, 4, 8), torch.ones(2, 1, 4, 8))
    assert cache.k_attn.shape[1] == 71 and torch.equal(cache.k_attn[:, :70], tensors["k_attn"])


@pytest.mark.parametrize("cls", ["NeuralAttentionSearchLinearAttnGDN", "NeuralAttentionSearchLinearAttnMamba"])
def test_layer_saved_with_plain_attributes(cls):
    layer = getattr(nat, cls)(hidden_size=64, expand_v=1, head_dim=64, num_heads=1, num_attn_heads=1, layer_idx=0)
    saved = dict(layer.__dict__)
    saved["attn_fraction"] = saved.pop("_attn_fraction") + 0.25
    old = type(layer).__new__(type(layer))
    old.__setstate__(saved)
    assert float(old.attn_fraction) == 0.25 and old.attn_blocks is None
    layer.attn_blocks = (torch.tensor([[[1, 2]]]), 4)
    assert float(copy.deepcopy(layer).attn_fraction) == 0.25
    assert float(layer.attn_fraction) == 0.25
    layer.attn_blocks[0].mul_(2)                             # what a graph's replay does to the counts
    assert float(layer.attn_fraction) == 0.5
