"""Column chains on 16-bit sums (colsum16.cu) against the CPU oracle, bit for bit: run and tile edges in rows, sector edges in
columns, and values that send a run back to the exact caster."""
import numpy as np
import pytest
import torch

from conftest import mismatch_report, same_bits

pytestmark = pytest.mark.gpu

FORMATS = [(5, 10), (8, 7)]                      # (exp, man); the general chain covers the others
ROWS = [1, 31, 32, 33, 191, 192, 193, 700]       # around loads of 32 and a tile of 192 rows, more tiles than stages
COLS = [1, 7, 8, 9, 33]                          # around a CTA's eight columns


def dev(x):
    return torch.from_numpy(np.ascontiguousarray(x, dtype=np.float32)).cuda()


def value_sets(rng, shape):
    x = rng.standard_normal(shape).astype(np.float32)
    yield "ordinary", x
    yield "binary16 subnormal sums", x * np.float32(2.0 ** -20)
    yield "sums that flush", x * np.float32(2.0 ** -13)
    yield "overflow", x * np.float32(9000.0)
    yield "overflow past 2^127", x * np.float32(1e38)
    yield "fp32 denormal sums", x * np.float32(2.0 ** -127)
    y = x.copy()
    y[rng.random(shape) < 0.02] = np.inf
    y[rng.random(shape) < 0.01] = np.nan
    yield "infinities and NaN", y
    z = np.where(rng.random(shape) < 0.5, np.float32(-0.0), np.float32(0.0)).astype(np.float32)
    yield "zeros of both signs", z
    yield "negative zeros", np.full(shape, -0.0, np.float32)
    yield "ties", (rng.integers(-4096, 4097, shape) * 0.5).astype(np.float32)


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("sub", [True, False])
@pytest.mark.parametrize("sat", [True, False])
def test_qsum_rows(oracle, fmt, sub, sat):
    import mptorch_b200.quant as q

    e, m = fmt
    rng = np.random.default_rng(e)
    for rows in ROWS:
        for cols in COLS:
            for name, x in value_sets(rng, (rows, cols)):
                got = q.qsum_rows(dev(x), e, m, sub, sat).cpu().numpy()
                want = oracle.qsum_rows(x, m, e, sub, sat)
                assert same_bits(got, want), f"{rows}x{cols} {name}: " + mismatch_report(got, want)


@pytest.mark.parametrize("fmt", FORMATS + [(4, 3), (5, 2)])
@pytest.mark.parametrize("rows", [1, 7, 8, 19])
def test_qsum_of_few_rows_and_many_columns(oracle, fmt, rows):
    import mptorch_b200.quant as q

    e, m = fmt
    for name, x in value_sets(np.random.default_rng(rows), (rows, 32768 + 5)):
        got, want = q.qsum_rows(dev(x), e, m, True, False).cpu().numpy(), oracle.qsum_rows(x, m, e, True, False)
        assert same_bits(got, want), f"{name}: " + mismatch_report(got, want)


@pytest.mark.parametrize("rows,cols", [(40, 8192), (40, 8193), (31, 8200), (32, 8200), (255, 8200), (256, 8200), (128, 32768), (129, 32768),
                                       (129, 65535), (129, 65536)])
@pytest.mark.parametrize("sub", [True, False])
@pytest.mark.parametrize("fmt", FORMATS + [(4, 3), (8, 23)])
def test_qsum_on_both_sides_of_each_rule(oracle, fmt, sub, rows, cols):
    """The kernel changes with the columns, the rows and the format; the sums do not."""
    import mptorch_b200.quant as q

    e, m = fmt
    x = np.random.default_rng(rows).standard_normal((rows, cols)).astype(np.float32)
    x[:, ::7] *= np.float32(2.0 ** -13)
    x[:, 1::7] *= np.float32(9000.0)
    x[rows // 2, 2::7] = np.inf
    got, want = q.qsum_rows(dev(x), e, m, sub, False).cpu().numpy(), oracle.qsum_rows(x, m, e, sub, False)
    assert same_bits(got, want), mismatch_report(got, want)


@pytest.mark.parametrize("acc,mul", [((5, 10), (5, 10)), ((8, 7), (8, 7)), ((5, 10), (4, 3)), ((8, 7), (5, 10))])
@pytest.mark.parametrize("sub", [True, False])
@pytest.mark.parametrize("sat", [True, False])
def test_layernorm_parameter_gradients(oracle, acc, mul, sub, sat):
    """Both chains and the producers' roundings; mean and reciprocal deviation given, so that only this kernel is at work."""
    import mptorch_b200.quant as q

    (ea, ma), (em, mm) = acc, mul
    rng = np.random.default_rng(11)
    for rows, cols in [(1, 5), (16, 8), (193, 33), (800, 16)]:
        mean = rng.standard_normal(rows).astype(np.float32)
        rstd = (0.5 + rng.random(rows)).astype(np.float32)
        w = rng.standard_normal(cols).astype(np.float32)
        for name, x in value_sets(rng, (rows, cols)):
            g = rng.standard_normal((rows, cols)).astype(np.float32)
            for xx, gg in ((x, g), (g, x)):
                _, gw, gb = q.float_layernorm_backward(dev(xx), dev(gg), dev(w), dev(w), dev(mean), dev(rstd), [-1], ma, ea, mm, em, ma, ea,
                                                       "nearest", sub, sat)
                _, wg, wb = oracle.layernorm_backward(xx, gg, w, mean, rstd, [-1], ma, ea, mm, em, ma, ea, sub, sat, "tree64")
                assert same_bits(gw.cpu().numpy(), wg), f"gamma {rows}x{cols} {name}: " + mismatch_report(gw.cpu().numpy(), wg)
                assert same_bits(gb.cpu().numpy(), wb), f"beta {rows}x{cols} {name}: " + mismatch_report(gb.cpu().numpy(), wb)
