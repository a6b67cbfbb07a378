"""GPU: q/k normalisation and rotation at the edges of the form that takes four heads at a time."""

import pytest
import torch

from zmlx_b200 import ops
from zmlx_b200.model import apply_rope, rms_norm, rope_tables

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("hq,hk,hd", [(5, 1, 128), (2, 1, 4), (3, 3, 132), (4, 1, 126), (1, 1, 124), (9, 3, 256)])
@pytest.mark.parametrize("odd", [False, True])  # rows on 4-byte boundaries, or 2 bytes off
@pytest.mark.parametrize("units", [9600, 9601])  # either side of 9600 (token, head) pairs
def test_qkv_post_head_shapes(hq, hk, hd, odd, units):
    heads_all = hq + 2 * hk
    B, S, pos = 1, units // heads_all + (units == 9601), 3
    g = torch.Generator(device=DEV).manual_seed(hd)

    def rows(n, width):
        t = torch.randn(n * width + 1, generator=g, device=DEV).to(torch.bfloat16)
        return t[odd:odd + n * width].view(n, width)

    max_seq = pos + S + 1
    cos, sin = rope_tables(hd, max_seq, 1e6, DEV)
    q, k = rows(B * S, hq * hd), rows(B * S, hk * hd)
    v = torch.randn((B * S, hk * hd), generator=g, device=DEV).to(torch.bfloat16)
    qn, kn = rows(1, hd)[0], rows(1, hd)[0]
    kc = torch.zeros((B, hk, max_seq, hd), dtype=torch.bfloat16, device=DEV)
    vc = kc.clone()
    out = ops.qkv_post(q, k, v, qn, kn, cos, sin, 1e-6, B, S, pos, kc, vc)

    def heads(t):
        return t.view(B, S, -1, hd).transpose(1, 2)

    c, s = cos[pos:pos + S], sin[pos:pos + S]
    assert torch.equal(vc[:, :, pos:pos + S], heads(v))
    for got, want in ((out, apply_rope(rms_norm(heads(q), qn, 1e-6), c, s)),
                      (kc[:, :, pos:pos + S], apply_rope(rms_norm(heads(k), kn, 1e-6), c, s))):
        # the mean is summed in another order: a normalised value may round to its neighbour (2^-7 of it) before the rotation
        # mixes it with its partner, and the result may round to the neighbour in turn
        near = want.float().abs().amax(-1, keepdim=True)
        assert bool(((got.float() - want.float()).abs() <= 3 * 2.0 ** -7 * near).all())
        assert float((got != want).float().mean()) < 0.02
    assert bool((kc[:, :, :pos] == 0).all()) and bool((kc[:, :, pos + S:] == 0).all())
