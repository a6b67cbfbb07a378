"""GPU: the combine's 16-byte form against its scalar form (which an address off a 16-byte boundary takes), bit for bit."""

import pytest
import torch

from zmlx_b200 import _lib, ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("mode", sorted(_lib.COMBINE_MODES.values()))
@pytest.mark.parametrize("T,K,D", [(1, 1, 8), (3, 8, 24), (2, 9, 1032), (5, 11, 2048), (2, 16, 16)])
@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("flags", [0, 1, 3])
def test_wide_combine_equals_the_scalar_one(mode, T, K, D, residual, flags):
    fp32 = mode in (_lib.COMBINE_MODES["fp32"], _lib.COMBINE_MODES["fp32_no_fma"]) and not flags & 1
    if residual and fp32:
        pytest.skip("a residual needs an output in T")
    g = torch.Generator(device=DEV).manual_seed(mode * 7 + D)
    y = torch.randn((T * K * D + 8,), generator=g, device=DEV).to(torch.bfloat16)
    y[3] = float("inf")
    y[D + 1 if T * K > 1 else 1] = float("nan")
    w = torch.rand((T, K), generator=g, device=DEV)
    res = torch.randn((T, D), generator=g, device=DEV).to(torch.bfloat16) if residual else None
    lib, p = _lib.load(), ops._ptr

    def call(rows):
        out = torch.empty((T, D), dtype=torch.float32 if fp32 else torch.bfloat16, device=DEV)
        _lib.check(lib.zmoe_moe_combine(rows.data_ptr(), _lib.BF16, p(w), _lib.F32, T, K, D, mode, p(out), flags, p(res),
                                        ops._stream()))
        return out

    shifted = torch.empty_like(y)
    shifted[2:2 + T * K * D] = y[:T * K * D]
    a, b = call(y), call(shifted[2:])
    bits = torch.int32 if fp32 else torch.int16
    same = (a.view(bits) == b.view(bits)) | (a.isnan() & b.isnan())
    assert bool(same.all())
