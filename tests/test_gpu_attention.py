"""GPU: the attention side of the stacked decoder (csrc/attn.cu) against float64."""

import math

import pytest
import torch

from zmlx_b200 import ops
from zmlx_b200.model import apply_rope, rms_norm, rope_tables

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _randn(g, *shape, std=1.0):
    return (torch.randn(shape, generator=g, device=DEV) * std).to(torch.bfloat16)


@pytest.mark.parametrize("rows,d", [(1, 8), (3, 2048), (5, 2056), (2, 16384), (300, 256)])
@pytest.mark.parametrize("with_delta", [False, True])
def test_add_rms_norm(rows, d, with_delta):
    g = torch.Generator(device=DEV).manual_seed(rows + d)
    h, w = _randn(g, rows, d, std=3.0), _randn(g, d)
    delta = _randn(g, rows, d) if with_delta else None
    sum_ = h + delta if with_delta else h.clone()
    x = ops.add_rms_norm(h, delta, w, 1e-6)
    assert torch.equal(h, sum_)  # the residual add rounds once, as torch does
    hd = sum_.double()
    ref = hd * torch.rsqrt(hd.pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    # one bfloat16 rounding (half an ulp: 2^-8) and a float32 sum of d squares and three roundings, far below it
    assert bool(((x.double() - ref).abs() <= (2.0 ** -8 + 2.0 ** -17) * ref.abs() + 1e-30).all())


@pytest.mark.parametrize("B,S,hq,hk,hd,pos", [(1, 1, 4, 2, 64, 0), (3, 1, 32, 4, 128, 77), (2, 9, 8, 8, 128, 5),
                                              (1, 130, 8, 1, 64, 0), (2, 1, 6, 2, 48, 3)])
@pytest.mark.parametrize("on_device", [False, True])
def test_qkv_post_matches_the_torch_form(B, S, hq, hk, hd, pos, on_device):
    g = torch.Generator(device=DEV).manual_seed(B * 100 + S)
    max_seq = pos + S + 3
    cos, sin = rope_tables(hd, max_seq, 1e6, DEV)
    q, k, v = _randn(g, B * S, hq * hd, std=2.0), _randn(g, B * S, hk * hd, std=2.0), _randn(g, B * S, hk * hd)
    qn, kn = _randn(g, hd), _randn(g, hd)
    kc = torch.full((B + 1, hk, max_seq, hd), 7.0, dtype=torch.bfloat16, device=DEV)
    vc = kc.clone()
    at = torch.tensor([pos], dtype=torch.int64, device=DEV) if on_device else pos
    out = ops.qkv_post(q, k, v, qn, kn, cos, sin, 1e-6, B, S, at, kc, vc)

    def heads(t):
        return t.view(B, S, -1, hd).transpose(1, 2)

    c, s = cos[pos:pos + S], sin[pos:pos + S]
    want_q = apply_rope(rms_norm(heads(q), qn, 1e-6), c, s)
    want_k = apply_rope(rms_norm(heads(k), kn, 1e-6), c, s)
    assert torch.equal(vc[:B, :, pos:pos + S], heads(v))
    for got, want in ((out, want_q), (kc[:B, :, pos:pos + S], want_k)):
        # the mean is summed in another order: a normalised value may round to its neighbour (2^-7 of it) before the
        # rotation mixes it with its partner, and the result may round to the neighbour in turn
        near = want.float().abs().amax(-1, keepdim=True)
        assert bool(((got.float() - want.float()).abs() <= 3 * 2.0 ** -7 * near).all())
        assert float((got != want).float().mean()) < 0.01
    untouched = torch.ones(max_seq, dtype=torch.bool, device=DEV)
    untouched[pos:pos + S] = False
    assert bool((kc[:, :, untouched] == 7.0).all()) and bool((vc[:, :, untouched] == 7.0).all())
    assert bool((kc[B] == 7.0).all()) and bool((vc[B] == 7.0).all())  # sequences beyond the batch


@pytest.mark.parametrize("hq,hk,hd", [(4, 4, 64), (4, 2, 64), (8, 2, 128), (32, 4, 128), (8, 1, 64)])
@pytest.mark.parametrize("B,npos", [(1, 1), (2, 63), (3, 64), (1, 65), (2, 300), (1, 4097)])
def test_decode_attention(hq, hk, hd, B, npos):
    g = torch.Generator(device=DEV).manual_seed(npos)
    max_seq = npos + 5
    q = _randn(g, B, hq, 1, hd, std=2.0)
    kc, vc = _randn(g, B + 1, hk, max_seq, hd, std=2.0), _randn(g, B + 1, hk, max_seq, hd)
    kc[:, :, npos:], vc[:, :, npos:] = float("nan"), float("nan")  # never read
    rep = hq // hk
    kd, vd = (t[:B, :, :npos].double().repeat_interleave(rep, 1) for t in (kc, vc))
    pr = torch.softmax((q.double() @ kd.transpose(-1, -2)) / math.sqrt(hd), dim=-1)
    ref, mass = (pr @ vd)[:, :, 0].reshape(B, -1), (pr @ vd.abs())[:, :, 0].reshape(B, -1)
    pos = torch.tensor([npos - 1], dtype=torch.int64, device=DEV)
    for kw in ({"npos": npos}, {"pos": pos}):
        got = ops.decode_attention(q, kc, vc, **kw).double()
        # the result's rounding (2^-8), and float32 throughout: a score of some tens is off by about 2^-20, so is its exponential
        assert bool(((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -15 * mass).all()), kw


def test_head_shapes_without_a_kernel_are_left_to_torch():
    for hq, hk, hd in ((6, 2, 64), (16, 1, 128), (4, 2, 96)):
        q = torch.zeros((1, hq, 1, hd), dtype=torch.bfloat16, device=DEV)
        c = torch.zeros((1, hk, 8, hd), dtype=torch.bfloat16, device=DEV)
        assert ops.decode_attention(q, c, c, npos=3) is None


@pytest.mark.parametrize("hq,hk,hd", [(4, 2, 64), (8, 1, 128)])
def test_decode_attention_with_infinite_keys(hq, hk, hd):
    """Positions whose score is -inf weigh nothing, also where a whole block or slice of the cache holds only such; a row
    without any other score, or with one of +inf, is NaN, as softmax has it."""
    g = torch.Generator(device=DEV).manual_seed(5)
    npos, n = 700, 64
    q = _randn(g, 4, hq, 1, hd).abs() + 0.125
    kc, vc = _randn(g, 4, hk, npos, hd), _randn(g, 4, hk, npos, hd)
    dead = torch.zeros((4, npos), dtype=torch.bool, device=DEV)
    dead[0, :3 * n], dead[1, n + 5:-1], dead[2] = True, True, True
    kd, vd = (t.double().repeat_interleave(hq // hk, 1) for t in (kc, vc))
    sc = ((q.double() @ kd.transpose(-1, -2)) / math.sqrt(hd))[:, :, 0].masked_fill(dead[:, None], -math.inf)
    pr = torch.softmax(sc, dim=-1)[:, :, None]
    ref, mass = (pr @ vd)[:, :, 0], (pr @ vd.abs())[:, :, 0]
    kc[:, :, :, 7] = torch.where(dead[:, None], -math.inf, kc[:, :, :, 7].float()).to(torch.bfloat16)
    kc[3, :, 100, 7] = math.inf
    got = ops.decode_attention(q, kc, vc, npos=npos).view(4, hq, hd).double()
    for b in (0, 1):
        assert bool(((got[b] - ref[b]).abs() <= 2.0 ** -8 * ref[b].abs() + 2.0 ** -15 * mass[b]).all()), b
    assert bool(got[2].isnan().all()) and bool(got[3].isnan().all())


def test_tensors_the_kernels_cannot_read_are_refused():
    """Another dtype, a transposed or a short tensor: an error, not other values read through the pointer."""
    h, w = torch.zeros((4, 64), dtype=torch.bfloat16, device=DEV), torch.ones(64, dtype=torch.bfloat16, device=DEV)
    for delta in (h.float(), torch.zeros((64, 4), dtype=torch.bfloat16, device=DEV).T, h[:2]):
        with pytest.raises(ValueError):
            ops.add_rms_norm(h, delta, w, 1e-6)
    c = torch.zeros((2, 2, 8, 64), dtype=torch.bfloat16, device=DEV)
    q = torch.zeros((2, 64, 1, 2), dtype=torch.bfloat16, device=DEV).transpose(1, 3)
    with pytest.raises(ValueError):
        ops.decode_attention(q, c, c, npos=3)
    cos = torch.zeros((8, 32), device=DEV)
    rows = torch.zeros((2, 128), dtype=torch.bfloat16, device=DEV)
    with pytest.raises(ValueError):
        ops.qkv_post(rows, rows.float(), rows, w, w, cos, cos, 1e-6, 2, 1, 0, c, c)


@pytest.mark.parametrize("pairs,npos", [(32, 200), (33, 200), (64, 70), (65, 300), (128, 130), (129, 130),  # 8, 4, 2, 1 CTAs
                                        (2, 8192), (40, 4096), (40, 4097), (130, 1024), (130, 1025), (3, 18000)])
def test_decode_attention_work_sharing(pairs, npos):
    """Either side of every cluster size, and of the lengths that several clusters share."""
    g = torch.Generator(device=DEV).manual_seed(npos)
    q, kc, vc = _randn(g, pairs, 2, 1, 64, std=2.0), _randn(g, pairs, 1, npos, 64, std=2.0), _randn(g, pairs, 1, npos, 64)
    kd, vd = kc.double().expand(-1, 2, -1, -1), vc.double().expand(-1, 2, -1, -1)
    pr = torch.softmax((q.double() @ kd.transpose(-1, -2)) / math.sqrt(64), dim=-1)
    ref, mass = (pr @ vd)[:, :, 0].reshape(pairs, -1), (pr @ vd.abs())[:, :, 0].reshape(pairs, -1)
    for _ in range(3):
        got = ops.decode_attention(q, kc, vc, npos=npos).double()
        assert bool(((got - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -15 * mass).all())
