"""GPU: the tensor-memory matmul's work sharing -- sets of expanders and finishers that take turns at chunks and items -- and the
line between its two expansions."""

import pytest
import torch

from zmlx_b200 import ops

from test_gpu_qmm_tma import DEV, _bank, _call, _weights, _within

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["affine", "mxfp4"])
@pytest.mark.parametrize("K", [256, 768, 2304])  # 1, 3 and 9 chunks of an item: every phase of the sets against the items
@pytest.mark.parametrize("per", [3, 33, 70])     # token rows of an expert: 16, 48 and 96 columns
def test_several_items_per_cta(per, K, mode):
    """Four to five items per CTA: 36 experts x 18 row tiles on 148 SMs."""
    E, N = 36, 18 * 128
    g = torch.Generator(device=DEV).manual_seed(K + per)
    a, A = _bank(g, E, N, K, mode, False)
    rows = E * per
    x = torch.randn((rows, K), generator=g, device=DEV).to(torch.bfloat16)
    ids = torch.arange(rows, device=DEV) // per
    plan = ops.build_plan(ids, E)
    ws = ops.qmm_workspace(rows, E, K, rows_hint=max(per, 9), mode=mode, device=DEV)
    for _ in range(3):
        got = _call(x, rows, K, [a], E, N, mode, plan, rows, max(per, 9), 1, ws)
        for e in range(0, E, 5):
            xe = x[e * per:(e + 1) * per].double()
            _within(got[e * per:(e + 1) * per], xe @ A[e].T, xe.abs() @ A[e].abs().T, K)


@pytest.mark.parametrize("rows", [9, 60])
@pytest.mark.parametrize("down", [0, 7, 8, 9, 13])
@pytest.mark.parametrize("of", ["scale", "offset"])
def test_values_around_the_narrow_expansions_reach(of, down, rows):
    """One group's scale (or offset) is 2^-down of the largest scale: on either side of the 8 binades, and at the older line of
    12, its weights keep all their bits.  The activations are large where the value is small."""
    E, N, K = 1, 64, 512
    g = torch.Generator(device=DEV).manual_seed(down)
    word = torch.randint(-2 ** 31, 2 ** 31, (E, N, K // 8), generator=g, device=DEV).to(torch.int32)
    s = (torch.rand((E, N, K // 64), generator=g, device=DEV) + 1.0) / 2
    b = -8.0 * s
    lift = torch.zeros(K // 64, device=DEV)
    if of == "scale":
        s[..., 2::4] *= 2.0 ** -down
        b[..., 2::4] *= 2.0 ** -down
        lift[2::4] = down
    else:
        b[..., 1::4] = s[..., 1::4] * 2.0 ** -down
        b[..., 3::4] = 0.0
    s, b = s.to(torch.bfloat16), b.to(torch.bfloat16)
    x = torch.randn((rows, K // 64, 64), generator=g, device=DEV) * torch.exp2(lift)[None, :, None]
    x = x.reshape(rows, K).to(torch.bfloat16)
    A = _weights(word, s, b)[0]
    ws = ops.qmm_workspace(rows, E, K, rows_hint=rows, mode="affine", device=DEV)
    plan = ops.build_plan(torch.zeros(rows, dtype=torch.int32, device=DEV), E)
    got = _call(x, rows, K, [(word, s, b)], E, N, "affine", plan, rows, rows, 1, ws)
    _within(got, x.double() @ A.T, x.double().abs() @ A.abs().T, K)


@pytest.mark.parametrize("mode", ["affine", "mxfp4"])
@pytest.mark.parametrize("counts", [[9] * 24, [10] * 24, [1, 40, 3, 17, 16, 0, 33, 8] * 3, [2] * 23 + [170]])
def test_items_of_16_rows_with_larger_tasks(counts, mode):
    """Averages of 7 to 10 rows: items of 16 up to 9.6, which larger tasks are cut into."""
    E, N, K = len(counts), 160, 768
    g = torch.Generator(device=DEV).manual_seed(len(set(counts)))
    a, A = _bank(g, E, N, K, mode, False)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))
    ids = ids[torch.randperm(len(ids), generator=torch.Generator().manual_seed(1))].to(DEV)
    rows = len(ids)
    x = torch.randn((rows, K), generator=g, device=DEV).to(torch.bfloat16)
    ws = ops.qmm_workspace(rows, E, K, rows_hint=rows, mode=mode, device=DEV)
    got = _call(x, rows, K, [a], E, N, mode, ops.build_plan(ids, E), rows, rows, 1, ws)
    for e in range(E):
        m = ids == e
        _within(got[m], x[m].double() @ A[e].T, x[m].double().abs() @ A[e].abs().T, K)
