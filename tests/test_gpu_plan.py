"""GPU: the expert plan, from one pair to more than one CTA takes, against a sort on the host."""

import numpy as np
import pytest
import torch

from zmlx_b200 import ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("E", [1, 3, 128, 4096])
@pytest.mark.parametrize("P", [1, 4095, 4096, 4097, 32768 + 5])  # 4096 pairs: the last count that one CTA takes
@pytest.mark.parametrize("M,with_lhs,bad", [(1, False, False), (3, True, False), (1, False, True)])
def test_plan_groups_the_pairs(E, P, M, with_lhs, bad):
    g = torch.Generator().manual_seed(E + P)
    rhs = torch.randint(0, E, (P,), generator=g, dtype=torch.int32)
    rhs[torch.rand(P, generator=g) < 0.3] = E // 2  # one crowded expert
    if bad:
        rhs[P // 2] = E
        rhs[P - 1] = -1
    lhs = torch.randint(0, 50, (P,), generator=g, dtype=torch.int32) if with_lhs else None
    plan = ops.build_plan(rhs.to(DEV), E, M=M, lhs=None if lhs is None else lhs.to(DEV), lhs_div=8).cpu().numpy()
    r = rhs.numpy()
    ok = (r >= 0) & (r < E)
    counts = np.bincount(r[ok], minlength=E) * M
    assert list(plan[:4]) == [int((counts > 0).sum()), P * M, int(bad), E]
    n = int(plan[0])
    tasks = plan[4:4 + 4 * E].reshape(E, 4)
    offset = plan[4 + 4 * E:4 + 4 * E + E + 1]
    owners = np.nonzero(counts)[0]
    assert np.array_equal(offset, np.concatenate([[0], np.cumsum(counts)]))
    assert np.array_equal(tasks[:n], np.stack([owners, offset[owners], counts[owners], 0 * owners], 1))
    assert not tasks[n:].any()
    at = 4 + 4 * E + E + 1
    assert np.array_equal(plan[at:at + n], owners)
    src, dst = plan[at + E:at + E + P * M], plan[at + E + P * M:at + E + 2 * P * M]
    total = int(offset[-1])
    pair, m = dst[:total] // M, dst[:total] % M
    assert np.array_equal(np.sort(dst[:total]), np.sort((np.nonzero(ok)[0][:, None] * M + np.arange(M)).reshape(-1)))
    assert np.array_equal(r[pair], np.repeat(owners, counts[owners]))
    first = lhs.numpy()[pair] if with_lhs else pair // 8
    assert np.array_equal(src[:total], first * M + m)
