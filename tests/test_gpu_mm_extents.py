"""Products whose extents pass what a 32-bit byte count holds."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one format pair of the 16-bit kernels and one of the FP32 kernel
@pytest.mark.parametrize("add,mul", [((10, 5), (3, 4)), ((9, 6), (3, 4))])
@pytest.mark.parametrize("order", ["cuda", "seq"])
def test_more_than_2_to_29_columns(add, mul, order):
    """Four bytes a column: the first 8192 columns have at least 2^31 bytes to the right of them."""
    import mptorch_b200.quant as q

    g = torch.Generator(device="cuda").manual_seed(1)
    n, head = (1 << 29) + 8192, 16384
    a = torch.randn(1, 4, device="cuda", generator=g)
    b = torch.zeros(4, n, device="cuda")
    b[:, :head] = torch.randn(4, head, device="cuda", generator=g)
    kw = dict(man_add=add[0], exp_add=add[1], man_mul=mul[0], exp_mul=mul[1], rounding="nearest", fma=False, subnormals=True,
              saturate=False)
    with q.orders(accum=order):
        want = q.float_mm(a, b[:, :head].contiguous(), **kw)
        got = q.float_mm(a, b, **kw)
    assert want.any() and torch.equal(got[:, :head], want)
    assert not got[:, head:].any()
