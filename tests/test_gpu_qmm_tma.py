"""GPU: the grouped matmul that is fed through tensor memory (csrc/qmm_tma.cu) against float64, and against the register-fed
kernels that serve the same call without a workspace.

Sizes sit at the edges of its tiles: one to several token blocks per expert with ragged ends, output rows that do not
fill a tile of 128 (64 for gate and up), the smallest K, one expert and many, experts without rows.
"""

import pytest
import torch

from zmlx_b200 import _lib, ops, quant

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _bank(g, E, N, K, mode, spread):
    w = torch.randn((E, N, K), generator=g, device=DEV) * 0.02
    if spread:  # scales over 12 binades inside a row
        s = torch.exp2(torch.randint(-6, 7, (E, N, K // 64, 1), generator=g, device=DEV).float())
        w = (w.view(E, N, K // 64, 64) * s).view(E, N, K)
    if mode == "affine":
        p, s, b = quant.quantize_affine(w, 64)
        return (p, s, b), quant.dequantize_affine(p, s, b, 64).double()
    p, s = quant.quantize_mxfp4(w)
    return (p, s, None), quant.dequantize_mxfp4(p, s).double()


def _call(x, T, K, banks, E, N, mode, plan, rows, hint, by_dst, ws):
    lib, p, st = _lib.load(), ops._ptr, ops._stream()
    gs, qm = (64 if mode == "affine" else 32), ops.qmode_code(mode)
    out = torch.full((rows, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    w = ops._ws_args(ws)
    if len(banks) == 1:
        (a,) = banks
        _lib.check(lib.zmoe_gather_qmm_ws(p(x), T, K, p(a[0]), p(a[1]), p(a[2]), E, N, K, gs, qm, p(plan), rows, hint,
                                          by_dst, p(out), *w, st))
    else:
        a, u = banks
        _lib.check(lib.zmoe_gather_qmm_swiglu_ws(p(x), T, K, p(a[0]), p(a[1]), p(a[2]), p(u[0]), p(u[1]), p(u[2]), E, N,
                                                 K, gs, qm, p(plan), rows, hint, p(out), _lib.SWIGLU_CPU, *w, st))
    torch.cuda.synchronize()
    assert int(plan[2]) == 0
    return out


def _within(got, ref, mass, K):
    """The result's bfloat16 rounding (half an ulp: 2^-8 relative) plus fp32 sums: a chunk adds 272 products, then the
    chunks are added, each step within 2^-23 of the partial sums, which the sum of magnitudes `mass` bounds."""
    bound = 2.0 ** -8 * ref.abs() + (272 + K // 256) * 2.0 ** -23 * mass
    bad = (got.double() - ref).abs() > bound
    assert not bool(bad.any()), f"{int(bad.sum())} of {bad.numel()} outside"


CASES = [
    # E, N, K, rows of each expert
    (1, 64, 256, [9]), (1, 200, 768, [16]), (2, 128, 512, [17, 15]), (3, 72, 1024, [96, 97, 0]),
    (4, 136, 2048, [1, 193, 33, 64]), (8, 256, 256, [12, 0, 3, 48, 49, 1, 0, 25]), (2, 192, 7168, [95, 289]),
    (40, 128, 768, [i % 5 for i in range(40)]), (300, 64, 256, [2] * 300),
]


@pytest.mark.parametrize("mode", ["affine", "mxfp4"])
@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("case", range(len(CASES)))
def test_matches_float64_and_the_register_fed_kernels(case, spread, mode):
    E, N, K, counts = CASES[case]
    g = torch.Generator(device=DEV).manual_seed(100 + case)
    rows = sum(counts)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))
    ids = ids[torch.randperm(rows, generator=torch.Generator().manual_seed(case))].to(DEV)
    plan = ops.build_plan(ids, E)
    x = torch.randn((rows, K), generator=g, device=DEV)
    x *= torch.exp2(torch.randint(-20, 12, (rows, 1), generator=g, device=DEV).float())  # rows of very different size
    x = x.to(torch.bfloat16)
    a, A = _bank(g, E, N, K, mode, spread)
    u, U = _bank(g, E, N, K, mode, spread)
    ws = ops.qmm_workspace(rows, E, K, rows_hint=rows, mode=mode, device=DEV)
    assert ws is not None
    ref = torch.empty((rows, N), dtype=torch.float64, device=DEV)
    up, mass, up_mass = torch.empty_like(ref), torch.empty_like(ref), torch.empty_like(ref)
    for e in range(E):
        m = ids == e
        xe = x[m].double()
        ref[m], up[m], mass[m], up_mass[m] = xe @ A[e].T, xe @ U[e].T, xe.abs() @ A[e].abs().T, xe.abs() @ U[e].abs().T
    got = _call(x, rows, K, [a], E, N, mode, plan, rows, rows, case & 1, ws)
    _within(got, ref, mass, K)
    assert torch.equal(got, _call(x, rows, K, [a], E, N, mode, plan, rows, rows, case & 1, ws))
    h = _call(x, rows, K, [a, u], E, N, mode, plan, rows, rows, 0, ws)
    old = _call(x, rows, K, [a, u], E, N, mode, plan, rows, rows, 0, None)
    assert torch.equal(h, _call(x, rows, K, [a, u], E, N, mode, plan, rows, rows, 0, ws))
    if not spread:  # gate and up round to bfloat16 first: at most a few of them fall to the other side of a boundary
        differ = (h != old) & ~(h.isnan() & old.isnan())
        # rows far below 2^-14 lose bits in the fp16 staging of the older kernels: compare the ordinary ones
        ordinary = (x.float().abs().amax(1) > 2.0 ** -6)[:, None]
        assert float((differ & ordinary).float().mean()) < 0.01
        gv, uv = ref.to(torch.bfloat16).double(), up.to(torch.bfloat16).double()
        want = gv * torch.sigmoid(gv) * uv
        err = (h.double() - want).abs()
        # gate and up may round to the neighbour (2^-7 of them; |silu'| <= 1.1), their fp32 sums are off as in _within,
        # and the result rounds once (2^-8)
        sums = (272 + K // 256) * 2.0 ** -23
        bound = 1.1 * (2.0 ** -7 * gv.abs() + sums * mass) * uv.abs() + (2.0 ** -7 + 2.0 ** -8) * want.abs() + \
            (gv * torch.sigmoid(gv)).abs() * sums * up_mass + 1e-30
        assert bool((err <= 1.01 * bound).all())


@pytest.mark.parametrize("tokens", [96 * 3 + 5, 1400])
def test_repeated_calls_give_the_same_bits_under_load(tokens):
    """Many items per CTA, full token tiles: a hand-over between the kernel's roles that is not ordered shows as a
    rare difference between runs."""
    E, N, K, top = 16, 768, 2048, 4
    g = torch.Generator(device=DEV).manual_seed(7)
    a, _ = _bank(g, E, N, K, "affine", False)
    u, _ = _bank(g, E, N, K, "affine", False)
    x = torch.randn((tokens, K), generator=g, device=DEV).to(torch.bfloat16)
    ids = torch.rand((tokens, E), generator=g, device=DEV).topk(top, dim=-1).indices.to(torch.int32)
    plan = ops.build_plan(ids.reshape(-1), E, lhs_div=top)
    ws = ops.qmm_workspace(tokens * top, E, K, rows_hint=tokens, mode="affine", device=DEV)
    first = _call(x, tokens, K, [a, u], E, N, "affine", plan, tokens * top, tokens, 0, ws)
    for _ in range(20):
        assert torch.equal(first, _call(x, tokens, K, [a, u], E, N, "affine", plan, tokens * top, tokens, 0, ws))


@pytest.mark.parametrize("K", [768, 2048])
@pytest.mark.parametrize("per", [40, 256])
def test_long_sums_keep_their_precision(K, per):
    """How often the result is not the float64 result's rounding.  A relative error of e before the rounding moves about
    2^8 e of the results over a boundary, so 1.4e-4 of them says e = 9 x 2^-24: the few float32 roundings of chunk sums and
    folds that the path states.  Sums over whole chunks of 256 codes in the tensor core give 1.7e-4 at 49 and more rows."""
    N, E = 4096, 1024 // per
    g = torch.Generator(device=DEV).manual_seed(3)
    a, A = _bank(g, E, N, K, "affine", False)
    rows = E * per
    x = torch.randn((rows, K), generator=g, device=DEV).to(torch.bfloat16)
    ids = torch.arange(rows, device=DEV) // per
    ws = ops.qmm_workspace(rows, E, K, rows_hint=rows, mode="affine", device=DEV)
    got = _call(x, rows, K, [a], E, N, "affine", ops.build_plan(ids, E), rows, rows, 1, ws)
    ref = torch.cat([x[e * per:(e + 1) * per].double() @ A[e].T for e in range(E)])
    assert float((got != ref.to(torch.bfloat16)).float().mean()) < 1.4e-4


def _one_row(codes, scales, biases, x, rows):
    """`rows` equal token rows against an expert whose 64 weight rows hold the same codes: the results, all equal."""
    K, N = x.numel(), 64
    c = codes.to(torch.int64).view(K // 8, 8)
    word = (c << (4 * torch.arange(8))).sum(1)
    word = torch.where(word >= 2 ** 31, word - 2 ** 32, word).to(torch.int32)
    a = tuple(t.expand(1, N, -1).contiguous().to(DEV)
              for t in (word, scales.to(torch.bfloat16), biases.to(torch.bfloat16)))
    X = x.to(torch.bfloat16).expand(rows, K).contiguous().to(DEV)
    plan = ops.build_plan(torch.zeros(rows, dtype=torch.int32, device=DEV), 1)
    ws = ops.qmm_workspace(rows, 1, K, rows_hint=rows, mode="affine", device=DEV)
    got = _call(X, rows, K, [a], 1, N, "affine", plan, rows, rows, 1, ws)
    assert bool((got == got[0, 0]).all())
    return float(got[0, 0])


@pytest.mark.parametrize("rows", [9, 96])
def test_group_sums_and_offsets_keep_24_bits(rows):
    """Results that only the last bits of a group's sum, or of b + 8 s, decide; everything else is exact."""
    K = 256
    # w = q - 7 = 0 everywhere, formed as -x + X; the sum 64 + 2^-5 + 2^-17 has 24 bits
    x = torch.zeros(K)
    x[:64] = 1.0
    x[0], x[1], x[2] = 3.0, 2.0 ** -5, 2.0 ** -17
    assert _one_row(torch.full((K,), 7), torch.ones(K // 64), torch.full((K // 64,), -7.0), x, rows) == 0.0
    # codes of 8: the groups' results are their offsets, 1 + 2^-7 + 8 s and -(1 + 2^-7); what is left is 8 s, 2^-16 of it
    x = torch.zeros(K)
    x[5] = x[64 + 9] = 1.0
    s8 = 2.0 ** -16 * (1 + 2.0 ** -7)
    got = _one_row(torch.full((K,), 8), torch.tensor([s8 / 8, 0, 0, 0]), torch.tensor([1 + 2.0 ** -7, -(1 + 2.0 ** -7), 0, 0]),
                   x, rows)
    assert got == s8


@pytest.mark.parametrize("rows", [9, 100])
@pytest.mark.parametrize("steps", [(0, 7, 14, 20), (20, 0, 1, 13)])
def test_scales_far_apart_in_one_chunk(steps, rows):
    """A group's scale is 2^-d of the largest and its activations 2^d larger: every group weighs the same in the result,
    and none of the small scales' bits may go."""
    E, N, K = 2, 100, 512
    g = torch.Generator(device=DEV).manual_seed(rows)
    d = torch.tensor(steps, device=DEV).repeat(K // 256)
    s = (torch.rand((E, N, K // 64), generator=g, device=DEV) + 1.0) * torch.exp2(-d.float())
    b = -s * (4.0 + 8.0 * torch.rand((E, N, K // 64), generator=g, device=DEV))
    s, b = s.to(torch.bfloat16), b.to(torch.bfloat16)
    word = torch.randint(-2 ** 31, 2 ** 31, (E, N, K // 8), generator=g, device=DEV).to(torch.int32)
    A = _weights(word, s, b)
    x = torch.randn((2 * rows, K), generator=g, device=DEV).view(2 * rows, K // 64, 64) * torch.exp2(d.float())[None, :, None]
    x = x.reshape(2 * rows, K).to(torch.bfloat16)
    ids = torch.arange(2 * rows, device=DEV) % E
    ws = ops.qmm_workspace(2 * rows, E, K, rows_hint=2 * rows, mode="affine", device=DEV)
    got = _call(x, 2 * rows, K, [(word, s, b)], E, N, "affine", ops.build_plan(ids, E), 2 * rows, 2 * rows, 1, ws)
    ref = torch.stack([x[r].double() @ A[ids[r]].T for r in range(2 * rows)])
    mass = torch.stack([x[r].double().abs() @ A[ids[r]].abs().T for r in range(2 * rows)])
    _within(got, ref, mass, K)


def _weights(word, s, b):
    code = (word.unsqueeze(-1) >> torch.arange(0, 32, 4, device=word.device, dtype=torch.int32)) & 15
    code = code.reshape(*word.shape[:-1], -1).double()
    return (code.view(*s.shape, 64) * s.double()[..., None] + b.double()[..., None]).reshape(code.shape)


@pytest.mark.parametrize("rows", [9, 100])
@pytest.mark.parametrize("mode,depth", [("affine", 24), ("mxfp4", 29)])
def test_token_values_far_below_the_rows_largest(mode, depth, rows):
    """The row's largest value meets a weight of zero; values of 2^-depth of it decide the result, with all their bits."""
    E, N, K = 1, 100, 256
    g = torch.Generator(device=DEV).manual_seed(depth)
    word = torch.randint(-2 ** 31, 2 ** 31, (E, N, K // 8), generator=g, device=DEV).to(torch.int32)
    if mode == "affine":
        s = (torch.rand((E, N, K // 64), generator=g, device=DEV) + 1.0).to(torch.bfloat16)
        s[..., 0] = 0.0
        a = (word, s, -8.0 * s)
        A = _weights(*a)
    else:
        word[..., :8] = 0
        s = torch.full((E, N, K // 32), 120, dtype=torch.uint8, device=DEV)
        a, A = (word, s, None), quant.dequantize_mxfp4(word, s).double()
    # two binades of values that need all eight bits of a bfloat16
    x = (torch.rand((rows, K), generator=g, device=DEV) + 1.0) * torch.exp2(-torch.rand((rows, K), generator=g, device=DEV))
    x = x.to(torch.bfloat16).float() * 2.0 ** -depth
    x[:, :64] = 0.0
    x[:, 3] = 1.0
    x = x.to(torch.bfloat16)
    plan = ops.build_plan(torch.zeros(rows, dtype=torch.int32, device=DEV), E)
    ws = ops.qmm_workspace(rows, E, K, rows_hint=rows, mode=mode, device=DEV)
    got = _call(x, rows, K, [a], E, N, mode, plan, rows, rows, 1, ws)
    _within(got, x.double() @ A[0].T, x.double().abs() @ A[0].abs().T, K)


@pytest.mark.parametrize("rows", [9, 100])
def test_block_exponents_far_apart_in_one_chunk(rows):
    """mxfp4: the blocks far down carry the row's largest activations, the others small enough ones not to drown them: what
    a block 30 binades down adds is far above the result's float32 error, and must be there."""
    E, N, K = 2, 100, 512
    g = torch.Generator(device=DEV).manual_seed(rows)
    d = torch.tensor([0, 14, 27, 6, 34, 30, 21, 3], device=DEV).repeat(K // 256)
    s = (150 - d).expand(E, N, K // 32).to(torch.uint8).contiguous()
    word = torch.randint(-2 ** 31, 2 ** 31, (E, N, K // 8), generator=g, device=DEV).to(torch.int32)
    A = quant.dequantize_mxfp4(word, s).double()
    lift = torch.where(d >= 27, 0, -28)
    x = torch.randn((2 * rows, K), generator=g, device=DEV).view(2 * rows, K // 32, 32) * torch.exp2(lift.float())[None, :, None]
    x = x.reshape(2 * rows, K).to(torch.bfloat16)
    ids = torch.arange(2 * rows, device=DEV) % E
    ws = ops.qmm_workspace(2 * rows, E, K, rows_hint=2 * rows, mode="mxfp4", device=DEV)
    got = _call(x, 2 * rows, K, [(word, s, None)], E, N, "mxfp4", ops.build_plan(ids, E), 2 * rows, 2 * rows, 1, ws)
    ref = torch.stack([x[r].double() @ A[ids[r]].T for r in range(2 * rows)])
    mass = torch.stack([x[r].double().abs() @ A[ids[r]].abs().T for r in range(2 * rows)])
    # what is not exact is stated: a token value below 2^-31 of its row's largest is off by at most 2^-39 of that
    slack = 2.0 ** -39 * x.double().abs().amax(1)[:, None] * torch.stack([A[ids[r]].abs().sum(1) for r in range(2 * rows)])
    bound = 2.0 ** -8 * ref.abs() + (256 + K // 256) * 2.0 ** -23 * mass + slack
    assert bool(((got.double() - ref).abs() <= bound).all())


@pytest.mark.parametrize("rows", [9, 60])
@pytest.mark.parametrize("mode", ["affine", "mxfp4"])
def test_a_row_that_is_not_finite_stays_alone(mode, rows):
    """An infinity or a NaN makes its own row's results non-finite and leaves its neighbours' bits as they are."""
    E, N, K = 2, 200, 512
    g = torch.Generator(device=DEV).manual_seed(4)
    a, _ = _bank(g, E, N, K, mode, False)
    x = torch.randn((E * rows, K), generator=g, device=DEV).to(torch.bfloat16)
    plan = ops.build_plan(torch.arange(E * rows, device=DEV) // rows, E)
    ws = ops.qmm_workspace(E * rows, E, K, rows_hint=E * rows, mode=mode, device=DEV)
    clean = _call(x, E * rows, K, [a], E, N, mode, plan, E * rows, E * rows, 1, ws)
    x[3, 7], x[rows + 2, 300] = float("inf"), float("nan")
    got = _call(x, E * rows, K, [a], E, N, mode, plan, E * rows, E * rows, 1, ws)
    bad = torch.zeros(E * rows, dtype=torch.bool, device=DEV)
    bad[3] = bad[rows + 2] = True
    assert torch.equal(got[~bad], clean[~bad]) and not bool(got[bad].isfinite().any())


def test_more_items_than_a_cta_keeps_in_its_list():
    """400 experts x 128 row tiles over the SMs: 346 items per CTA on 148 of them, 256 of which are kept in shared memory."""
    E, N, K = 400, 16384, 256
    g = torch.Generator(device=DEV).manual_seed(6)
    word = torch.randint(-2 ** 31, 2 ** 31, (E, N, K // 8), generator=g, device=DEV, dtype=torch.int64).to(torch.int32)
    s = (torch.rand((E, N, K // 64), generator=g, device=DEV) + 0.5).to(torch.bfloat16)
    b = (-8.0 * torch.rand((E, N, K // 64), generator=g, device=DEV)).to(torch.bfloat16)
    rows = E + 20
    ids = torch.cat([torch.arange(E, device=DEV), torch.full((20,), E - 1, device=DEV)])
    x = torch.randn((rows, K), generator=g, device=DEV).to(torch.bfloat16)
    ws = ops.qmm_workspace(rows, E, K, rows_hint=21, mode="affine", device=DEV)
    got = _call(x, rows, K, [(word, s, b)], E, N, "affine", ops.build_plan(ids, E), rows, 21, 1, ws)
    for e in range(E):
        m = ids == e
        A, xe = _weights(word[e], s[e], b[e]), x[m].double()
        _within(got[m], xe @ A.T, xe.abs() @ A.abs().T, K)
