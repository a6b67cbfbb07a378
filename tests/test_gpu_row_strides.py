"""GPU: token rows that lie apart in memory (``h[:, -1]`` of a batch of prompts) give the bits of the same rows side by side,
whichever kernels the token count takes."""

import pytest
import torch

from zmlx_b200 import _lib, synthetic
from zmlx_b200 import nn as znn
from zmlx_b200.layer import MoELayer
from zmlx_b200.patch import patch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SHAPES = {"c1": {}, "c2": {}, "c3": {}, "c5": dict(n_experts=64)}  # c5: as wide as it is, with fewer experts
TOKENS = [1, 4, 9, 12, 16, 32, 64]
_PARAMS: dict = {}


def _params(name):
    if name not in _PARAMS:
        _PARAMS.clear()
        cfg = synthetic.CONFIGS[name].scaled(**SHAPES[name])
        _PARAMS[name] = (cfg, synthetic.make_layer(cfg, device=DEV))
    return _PARAMS[name]


def _views(cfg, T):
    h = synthetic.make_tokens(cfg, 3 * T, device=DEV).view(T, 3, cfg.d_model)
    return h[:, -1], h[:, -1:, :]  # (T, d) with rows 3 d apart, and the (T, 1, d) a decoder passes on


@pytest.mark.parametrize("T", TOKENS)
@pytest.mark.parametrize("name", list(SHAPES))
def test_layer_and_patched_block(name, T):
    cfg, params = _params(name)
    rows, deep = _views(cfg, T)
    dense = rows.contiguous()
    for fused in (True, False):
        layer = MoELayer(cfg, params, max_tokens=64, fused=fused)
        want, idx = layer(dense).clone(), layer.indices[:T].clone()
        assert torch.equal(layer(rows), want) and torch.equal(layer.indices[:T], idx), f"fused={fused}"
    block = znn.block_from_params(cfg, params)
    patch(torch.nn.ModuleList([block]), patterns=["moe_mlp"])
    want = block(dense)
    assert torch.equal(block(rows), want)
    assert torch.equal(block(deep).view(T, -1), want)


@pytest.mark.parametrize("T", [2, 16])
def test_overlapping_rows_stay_refused(T):
    cfg, params = _params("c1")
    layer = MoELayer(cfg, params, max_tokens=16, fused=False)
    row = synthetic.make_tokens(cfg, 1, device=DEV)
    with pytest.raises(_lib.ZmoeError):
        layer(row.expand(T, -1))


@pytest.mark.parametrize("T", [4, 16])
def test_patched_block_on_a_transposed_input(T):
    """The columns of a (d, T) matrix: the result has rows of its own, not the strides of its input."""
    cfg, params = _params("c1")
    block = znn.block_from_params(cfg, params)
    patch(torch.nn.ModuleList([block]), patterns=["moe_mlp"])
    dense = synthetic.make_tokens(cfg, T, device=DEV)
    across = dense.T.contiguous().T
    assert across.stride() == (1, T)
    assert torch.equal(block(across), block(dense))
