"""GPU: the one-launch block for mxfp4 banks (zmoe_layer_decode_mxfp4) against the oracle and the separate kernels."""

import pytest
import torch

from tests.helpers import assert_close_rel, oracle_layer, t2n
from zmlx_b200 import _lib, synthetic
from zmlx_b200.layer import MoELayer

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# d_ff = 1536 (c3) ends inside a weight stage; 256 and 768 leave warps of a team without work
SHAPES = {"c3": {}, "narrow": dict(d_model=256, d_ff=256, n_experts=16), "ragged": dict(d_model=1280, d_ff=768, n_shared=0),
          "softmax": dict(d_model=512, d_ff=1024, family="qwen3", n_experts=32, top_k=8, n_shared=0)}


@pytest.mark.parametrize("shape", list(SHAPES))
@pytest.mark.parametrize("T", [1, 2, 3, 4, 7, 8])
def test_block_matches_the_oracle(shape, T):
    cfg = synthetic.CONFIGS["c3"].scaled(**SHAPES[shape])
    params = synthetic.make_layer(cfg, device=DEV)
    # block scales far apart inside a row: 20 binades, beyond what a plain fp16 scale would hold beside the largest
    g = torch.Generator().manual_seed(T)
    s = params["gate_s"]
    params["gate_s"] = (s.int() - torch.randint(0, 21, s.shape, generator=g).to(DEV)).clamp(1, 254).to(torch.uint8)
    layer = MoELayer(cfg, params, max_tokens=8)
    assert layer._one_launch_bytes(T) > 0 and layer.fused_workspace_bytes(T) == 0
    x = synthetic.make_tokens(cfg, T, device="cpu").to(DEV)
    out = layer(x).clone()
    layer.check_status()
    ref, _ = oracle_layer(cfg, params, x, layer.router_logits(T), layer.indices[:T])
    assert_close_rel(t2n(out), ref, 2e-2, f"{shape} T={T}")  # the bound of the affine block's test
    sep = MoELayer(cfg, params, max_tokens=8, fused=False)
    assert_close_rel(t2n(out), t2n(sep(x)), 2e-2, f"{shape} T={T} against the separate kernels")
    assert torch.equal(layer.indices[:T], sep.indices[:T]) and torch.equal(layer.weights[:T], sep.weights[:T])
    for _ in range(3):
        assert torch.equal(layer(x), out)


def test_the_affine_entry_keeps_refusing_mxfp4_banks():
    import ctypes

    cfg = synthetic.CONFIGS["c3"].scaled(**SHAPES["narrow"])
    layer = MoELayer(cfg, synthetic.make_layer(cfg, device=DEV), max_tokens=8)
    x = synthetic.make_tokens(cfg, 1, device=DEV)
    ws = torch.zeros(1 << 20, dtype=torch.uint8, device=DEV)
    lib = _lib.load()
    rc = lib.zmoe_layer_decode(ctypes.byref(layer._desc), x.data_ptr(), x.stride(0), 1, ws.data_ptr(), ws.numel(), None, None,
                               layer.out.data_ptr(), None)
    assert rc == _lib.ERR_UNSUPPORTED
    affine = synthetic.CONFIGS["c1"]
    other = MoELayer(affine, synthetic.make_layer(affine, device=DEV), max_tokens=8)
    assert lib.zmoe_layer_decode_mxfp4_workspace_bytes(ctypes.byref(other._desc), 1) == 0


def test_capture_without_a_warm_up_pass():
    """The first call of a block may happen inside a capture: it is then recorded on the separate kernels."""
    cfg = synthetic.CONFIGS["c3"].scaled(**SHAPES["narrow"])
    params = synthetic.make_layer(cfg, device=DEV)
    x = synthetic.make_tokens(cfg, 2, device=DEV)
    want = MoELayer(cfg, params, max_tokens=8, fused=False)(x).clone()
    layer, out = MoELayer(cfg, params, max_tokens=8), torch.empty_like(want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        layer(x, out)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


@pytest.mark.parametrize("T", [1, 8])
def test_blocks_far_below_their_neighbours_keep_their_bits(T):
    """Half of gate's and up's blocks are 2^-30 of the others, which the token rows meet with zeros: the result is the one of
    the same blocks without neighbours, times a power of two, and follows the oracle."""
    cfg = synthetic.CONFIGS["c3"].scaled(**SHAPES["narrow"], n_shared=0)
    params = synthetic.make_layer(cfg, device=DEV)
    x = synthetic.make_tokens(cfg, T, device=DEV)
    x.view(T, -1, 32)[:, ::2] = 0
    low = {}
    for k in ("gate_s", "up_s"):
        s = params[k].clone()
        s[..., 1::2] = 120
        low[k] = s.clone()
        s[..., ::2] = 150  # met by zeros only
        params[k] = s
    layer = MoELayer(cfg, params, max_tokens=8)
    out = layer(x).clone()
    layer.check_status()
    alone = MoELayer(cfg, dict(params, **low), max_tokens=8)
    assert layer.passes(T) and torch.equal(out, alone(x))


@pytest.mark.parametrize("T", [1, 8, 12])
def test_weights_on_eight_byte_boundaries_take_the_separate_kernels(T):
    """A tensor that starts eight bytes into its storage, as slices of a mapped file do, was always served."""
    cfg = synthetic.CONFIGS["c3"].scaled(**SHAPES["narrow"])
    params = synthetic.make_layer(cfg, device=DEV)
    x = synthetic.make_tokens(cfg, T, device=DEV)
    want = MoELayer(cfg, params, max_tokens=16, fused=False)(x).clone()

    def shifted(w):
        buf = torch.empty(w.numel() + 2, dtype=torch.int32, device=DEV)
        buf[2:] = w.view(torch.int32).reshape(-1)
        return buf[2:].view(w.shape).view(w.dtype)

    moved = dict(params, **{f"{k}_w": shifted(params[f"{k}_w"]) for k in ("gate", "up", "down")},
                 gate_b=torch.zeros(3, dtype=torch.uint8, device=DEV)[1:])
    assert moved["gate_w"].data_ptr() % 16 == 8
    layer = MoELayer(cfg, moved, max_tokens=16)
    assert_close_rel(t2n(layer(x)), t2n(want), 2e-2, f"T={T}")
    assert not layer.passes(T)
