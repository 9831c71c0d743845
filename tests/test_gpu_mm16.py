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


# (batch, M, K, N): single elements, one short of and one past a group of 8, a slab of 32 and both tile heights; 160 batch
# entries are more tiles than SMs, which selects the 128-row tiles
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
