"""Narrow projections of the layer's forward at the edges of their tiles: features that do not fill a step of 64, one and several
tiles of tokens and of columns, heads between two groups of eight; against the layers' general path."""
import pytest

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
