"""GPU: gather_qmm_swiglu's default rows, for every way in which the activations broadcast against the expert indices."""

import pytest
import torch

from zmlx_b200 import quant
from zmlx_b200.kernels.fused_moe import _pairs_per_row, gather_qmm_swiglu

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("xshape,ishape,div", [((5, 1), (5, 4), 4), ((5, 4), (5, 4), 1), ((1, 4), (5, 4), 0), ((), (5, 4), 20),
                                               ((1,), (5, 4), 20), ((2, 3, 1), (2, 3, 4), 4), ((2, 1, 1), (2, 3, 4), 12),
                                               ((2, 1, 4), (2, 3, 4), 0), ((6, 1), (4,), 4), ((6, 1), (1, 4), 4), ((3,), (1,), 1),
                                               ((4,), (5, 1), 0)])
@pytest.mark.parametrize("dtype", [torch.uint32, torch.int64])
def test_default_rows_are_the_broadcast_arange(xshape, ishape, div, dtype):
    E, N, K, M = 6, 64, 256, 2
    g = torch.Generator(device=DEV).manual_seed(len(xshape))
    bank = [quant.quantize_affine(torch.randn((E, N, K), generator=g, device=DEV) * 0.02, 64) for _ in range(2)]
    x = torch.randn((*xshape, M, K), generator=g, device=DEV).to(torch.bfloat16)
    idx = torch.randint(0, E, ishape, generator=g, device=DEV)
    batch = torch.broadcast_shapes(xshape, ishape)
    assert _pairs_per_row(xshape, tuple(batch)) == div
    rows = torch.arange(max(1, x[..., 0, 0].numel()), device=DEV).reshape(xshape)
    idx_in = idx.to(torch.int32).view(torch.uint32) if dtype == torch.uint32 else idx
    args = (*bank[0], *bank[1])
    got = gather_qmm_swiglu(x, *args, rhs_indices=idx_in)
    want = gather_qmm_swiglu(x, *args, lhs_indices=rows.expand(batch), rhs_indices=idx.expand(batch))
    assert got.shape == (*batch, M, N) and torch.equal(got, want)
