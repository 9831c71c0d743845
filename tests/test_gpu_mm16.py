"""The GEMM on 16-bit running sums (gemm16_kernel.cuh) against the CPU oracle, bit for bit: every format pair it takes, at
the edges of its tiles and groups, and at the rounding thresholds of each format."""
import numpy as np
import pytest
import torch

from conftest import mismatch_report, same_bits
from test_gpu_mm import cpu_mm, gpu_mm

pytestmark = pytest.mark.gpu

# (add, mul) as (exp, man); the fused form uses the add format alone
PAIRS = [((5, 10), (5, 2)), ((5, 10), (4, 3)), ((5, 10), (5, 10)), ((8, 7), (5, 2)), ((8, 7), (4, 3)), ((8, 7), (8, 7)),
         ((5, 2), (5, 2)), ((4, 3), (4, 3))]


@pytest.fixture(scope="module")
def be():
    from mptorch_b200 import backend

    return backend


def check(be, oracle, a, b, what, **kw):
    got, want = gpu_mm(be, a, b, **kw), cpu_mm(oracle, a, b, **kw)
    assert same_bits(got, want), f"{what} {kw}: " + mismatch_report(got, want)


# (batch, M, K, N): single elements, one short of and one past a group of 8, a slab of 32 and the tiles' edges.  The rule sends
# the plain and fused forms of all of them to tiles of 8 rows and compensated sums to tiles of 64; the other tile heights
# are further down.
SHAPES = [(1, 1, 1, 1), (1, 15, 7, 63), (1, 17, 9, 65), (1, 16, 32, 64), (1, 33, 33, 4), (160, 3, 31, 5), (160, 5, 8, 66), (2, 129, 64, 68)]


@pytest.mark.parametrize("fmts", PAIRS)
@pytest.mark.parametrize("form", ["plain", "fma", "comp", "fma comp"])
@pytest.mark.parametrize("sub", [True, False])
def test_shapes_and_scales(be, oracle, fmts, form, sub):
    """Scales that keep the products in range, below the smallest normal value, and past the range of the formats (the
    per-group and per-entry fallbacks)."""
    fadd, fmul = fmts
    rng = np.random.default_rng(1000 * fadd[1] + 10 * fmul[1] + sub)
    for B, M, K, N in SHAPES:
        a = rng.standard_normal((B, M, K)).astype(np.float32)
        b = rng.standard_normal((B, K, N)).astype(np.float32)
        for scale in (1.0, 2.0 ** -6, 2.0 ** -13, 24.0):
            for order in (("cuda",) if "comp" in form else ("cuda", "seq")):
                check(be, oracle, a * np.float32(scale), b, (B, M, K, N, scale), fadd=fadd, fmul=fmul, sub=sub,
                      fma="fma" in form, comp="comp" in form, order=order)


@pytest.mark.parametrize("fmts", PAIRS)
@pytest.mark.parametrize("fma", [False, True])
@pytest.mark.parametrize("sub", [True, False])
def test_rounding_thresholds(be, oracle, fmts, fma, sub):
    """Products by 1 and sums of two values: every tie of the formats near and below the smallest normal value with its
    fp32 neighbours, and random patterns over the whole range the kernel takes."""
    fadd, fmul = fmts
    rng = np.random.default_rng(7)
    vals = []
    for e, m in (fadd, fmul):
        lo = 2 - (1 << (e - 1))
        if e == 8:
            lo = -30                                     # denormal proof: stay well above 2^-126
        for k in range(-m - 3, 7):
            vals.append(np.ldexp(1.0 + np.arange(2 ** min(m + 2, 8)) / 2.0 ** min(m + 2, 8), lo + k))
    x = np.concatenate(vals).astype(np.float32)
    x = np.concatenate([x, np.nextafter(x, np.float32(0)), np.nextafter(x, np.float32(np.inf))])
    r = np.ldexp(1 + rng.random(1 << 15), rng.integers(-26, 6, 1 << 15)).astype(np.float32)
    x = np.concatenate([x, r])
    x = x[np.abs(x) < 100]
    x = np.concatenate([x, -x, np.zeros(3, np.float32)])
    y = rng.permutation(x)
    for order in ("cuda", "seq"):
        one = np.ones((1, 1), np.float32)
        check(be, oracle, x[:, None], one, "products", fadd=fadd, fmul=fmul, fma=fma, sub=sub, order=order)
        check(be, oracle, np.stack([x, y], 1), np.ones((2, 1), np.float32), "sums", fadd=fadd, fmul=fmul, fma=fma, sub=sub, order=order)
        # the second operand lands in the next group of eight: the fold of the CUDA order
        a = np.zeros((x.size, 9), np.float32)
        a[:, 0], a[:, 8] = x, y
        check(be, oracle, a, np.ones((9, 1), np.float32), "folds", fadd=fadd, fmul=fmul, fma=fma, sub=sub, order=order)


@pytest.mark.parametrize("fmts", PAIRS)
def test_continuing_from_sums_outside_the_format(be, oracle, fmts):
    """A piece that continues from what C holds, where C is not a rounded sum: the first group starts from its 32 bits.
    Oracle: the same product with C as the products' first step (times 1, in a multiply format that keeps it) is not
    expressible, so the 32-bit kernel (MPT_MM_SCALAR cannot be switched in process) is stood in for by the definition."""
    fadd, fmul = fmts
    rng = np.random.default_rng(3)
    a = rng.standard_normal((20, 8)).astype(np.float32)
    b = rng.standard_normal((8, 12)).astype(np.float32)
    c0 = rng.standard_normal((20, 12)).astype(np.float32)
    c0[0, 0] = -0.0
    c = torch.from_numpy(c0.copy()).cuda()
    be.float_mm_nearest_piece(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), c, fadd[1], fadd[0], fmul[1], fmul[0], True, False,
                              False, be.MM_PIECE_FROM_C, order="cuda")
    inner = cpu_mm(oracle, a, b, fadd, fmul)             # one group of eight from zero, folded into +0
    want = oracle.float_quantize((c0 + inner).astype(np.float32), fadd[1], fadd[0], "nearest", True, False)
    assert same_bits(c.cpu().numpy(), want), mismatch_report(c.cpu().numpy(), want)


# ---- every tile height ------------------------------------------------------------------------------------------------
# Results that the rule sends to tiles of 8, 64 and 128 rows on a GPU of 148 SMs (`tile` is asked of the library, so that a rule
# that moves is noticed), each ragged in both directions and with K short of and past whole groups and slabs.
BATCHED = {8: (40, 21, 41, 37), 64: (140, 63, 41, 61), 128: (140, 113, 41, 50)}
# compensated sums have no tiles of 8 rows
COMPENSATED = {64: (40, 61, 21, 63), 128: (140, 113, 21, 50)}
# tiles inside the matrix beside ragged ones, with 16-byte copies (K and N multiples of 4) and without; three slabs of 32, two of 64
LARGE = {8: [(252, 72, 100), (67, 73, 99)], 64: [(700, 72, 700), (707, 73, 701)], 128: [(700, 72, 1028), (701, 73, 1027)]}


def tile(be, M, N, batch=1, comp=False):
    return be.mm16_tile_rows(M, N, batch, comp)


def scaled_batch(rng, B, M, K, N):
    """Batch entries in turn: in range, below the smallest normal value, sums that flush, past the formats' range, with
    infinities and NaN, zeros of both signs with a plan and (an infinity among them) without, exact cancellations without."""
    a = rng.standard_normal((B, M, K)).astype(np.float32)
    b = rng.standard_normal((B, K, N)).astype(np.float32)
    for i, scale in enumerate((1.0, 2.0 ** -6, 2.0 ** -13, 24.0)):
        a[i::8] *= np.float32(scale)
    a[4::8][rng.random(a[4::8].shape) < 0.01] = np.inf
    b[4::8][rng.random(b[4::8].shape) < 0.01] = np.nan
    for i in (5, 6):
        a[i::8] = np.where(rng.random(a[i::8].shape) < 0.9, np.float32(-0.0), a[i::8])
    a[7::8, :, 1::2], b[7::8, 1::2] = -a[7::8, :, :K - 1:2], b[7::8, :K - 1:2]
    a[6::8, M // 2, K // 2] = a[7::8, M // 3, K // 2] = np.inf
    a[2::8, 0, 0], b[2::8, 0, 0] = 2.0 ** -80, 2.0 ** -60      # 8-bit exponents: a product that is an fp32 denormal
    return a, b


@pytest.mark.parametrize("rows", [8, 64, 128])
@pytest.mark.parametrize("sub", [True, False])
@pytest.mark.parametrize("fmts", PAIRS)
def test_each_tile_height(be, oracle, fmts, sub, rows):
    fadd, fmul = fmts
    rng = np.random.default_rng(100 * fadd[1] + fmul[1] + rows)
    B, M, K, N = BATCHED[rows]
    assert tile(be, M, N, B) == rows
    a, b = scaled_batch(rng, B, M, K, N)
    for order in ("cuda", "seq"):
        for fma in (False, True):
            check(be, oracle, a, b, BATCHED[rows], fadd=fadd, fmul=fmul, sub=sub, fma=fma, order=order)
    check(be, oracle, a, b, BATCHED[rows], fadd=fadd, fmul=fmul, sub=sub, sat=True)
    if rows in COMPENSATED:
        B, M, K, N = COMPENSATED[rows]
        assert tile(be, M, N, B, True) == rows
        a, b = scaled_batch(rng, B, M, K, N)
        for fma in (False, True):
            check(be, oracle, a, b, COMPENSATED[rows], fadd=fadd, fmul=fmul, sub=sub, fma=fma, comp=True)


@pytest.mark.parametrize("rows", [8, 64, 128])
@pytest.mark.parametrize("sub", [True, False])
@pytest.mark.parametrize("fmts", PAIRS)
def test_tiles_inside_the_matrix(be, oracle, fmts, sub, rows):
    fadd, fmul = fmts
    rng = np.random.default_rng(10 * fadd[1] + fmul[1] + rows)
    for M, K, N in LARGE[rows]:
        assert tile(be, M, N) == rows
        # rows of every size of sum: in range, flushing, and (e4m3, e5m2) past the limit of the range check in the long run
        a = rng.standard_normal((M, K)).astype(np.float32) * np.float32(2.0) ** rng.integers(-9, 1, (M, 1)).astype(np.float32)
        b = rng.standard_normal((K, N)).astype(np.float32)
        for order in ("cuda", "seq"):
            check(be, oracle, a, b, (M, K, N), fadd=fadd, fmul=fmul, sub=sub, order=order)
        check(be, oracle, a, b, (M, K, N), fadd=fadd, fmul=fmul, sub=sub, fma=True)


def continued(oracle, a, b, c, fadd, fmul, sub, order):
    """The definition of a last piece: the product's steps from what C holds, one rounded operation at a time."""
    def q(x, fmt):
        return oracle.float_quantize(np.ascontiguousarray(x, np.float32), fmt[1], fmt[0], "nearest", sub, False)

    K = a.shape[1]
    steps = [q(a[:, k, None] * b[None, k, :], fmul) for k in range(K)]
    acc = c.copy()
    if order == "seq":
        for p in steps:
            acc = q(acc + p, fadd)
        return acc
    for k0 in range(0, K + 8 - K % 8, 8):                 # the order's last group is of zeros where K is a multiple of eight
        inner = np.zeros_like(c)
        for p in steps[k0:k0 + 8]:
            inner = q(inner + p, fadd)
        for _ in range(max(k0 + 8 - max(K, k0), 0)):
            inner = q(inner + np.float32(0.0), fadd)
        acc = q(acc + inner, fadd)
    return acc


@pytest.mark.parametrize("rows", [8, 64, 128])
@pytest.mark.parametrize("order", ["cuda", "seq"])
@pytest.mark.parametrize("sub,planned", [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize("fmts", PAIRS)
def test_continuing_on_each_tile_height(be, oracle, fmts, sub, planned, order, rows):
    """Pieces that continue from sums outside the format (32-bit values, zeros of both signs, infinities, NaN) and from rounded
    ones; with operands that pass the range check (where the formats let them) and with an infinity, which never does."""
    fadd, fmul = fmts
    M, K, N = LARGE[rows][0]
    K = K if rows == 8 else 40                            # two slabs of either kernel
    rng = np.random.default_rng(17 + rows)
    a = rng.standard_normal((M, K)).astype(np.float32)
    b = rng.standard_normal((K, N)).astype(np.float32)
    a[1] = -0.0
    if not planned:
        a[M // 2, K - 2] = np.inf
    c0 = rng.standard_normal((M, N)).astype(np.float32)
    c0[rng.random(c0.shape) < 0.05] = -0.0
    c0[rng.random(c0.shape) < 0.001] = np.inf
    c0[rng.random(c0.shape) < 0.001] = np.nan
    c0[: M // 2] = oracle.float_quantize(c0[: M // 2], fadd[1], fadd[0], "nearest", sub, False)
    c0[1] = -0.0
    c = torch.from_numpy(c0.copy()).cuda()
    be.float_mm_nearest_piece(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), c, fadd[1], fadd[0], fmul[1], fmul[0], sub, False,
                              False, be.MM_PIECE_FROM_C, order=order)
    with np.errstate(all="ignore"):
        want = continued(oracle, a, b, c0, fadd, fmul, sub, order)
    assert same_bits(c.cpu().numpy(), want), mismatch_report(c.cpu().numpy(), want)
