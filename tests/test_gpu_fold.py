"""The fold kernel against torch's fold, bit for bit: fp32 sums from zero in ascending output position."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# n, channels, H, W, kernel, stride, padding, dilation: single pixels, ragged tiles, strides that skip pixels, dilation, kernels
# larger than the stride and padding past the image, channel counts around a CTA's, tiles in both directions
CASES = [(1, 1, 1, 1, (1, 1), (1, 1), (0, 0), (1, 1)), (2, 3, 9, 7, (3, 3), (1, 1), (1, 1), (1, 1)),
         (3, 17, 15, 70, (3, 5), (1, 2), (2, 1), (1, 1)), (2, 5, 13, 13, (3, 3), (2, 2), (0, 0), (1, 1)),
         (1, 8, 20, 20, (3, 3), (1, 1), (2, 2), (2, 2)), (2, 4, 12, 11, (2, 2), (3, 3), (1, 1), (1, 1)),
         (1, 2, 40, 130, (7, 7), (1, 1), (3, 3), (1, 1)), (1, 3, 30, 30, (11, 11), (4, 4), (2, 2), (1, 1)),
         (2, 64, 56, 56, (3, 3), (1, 1), (1, 1), (1, 1)), (1, 2, 33, 9, (1, 9), (1, 1), (0, 4), (1, 1)),
         (1, 1, 24, 24, (12, 12), (1, 1), (0, 0), (1, 1)), (2, 6, 16, 16, (1, 1), (2, 2), (0, 0), (1, 1))]


@pytest.mark.parametrize("case", CASES)
def test_fold_equals_torch(case):
    from mptorch_b200 import backend as be

    n, c, h, w, k, s, p, d = case
    oh = (h + 2 * p[0] - d[0] * (k[0] - 1) - 1) // s[0] + 1
    ow = (w + 2 * p[1] - d[1] * (k[1] - 1) - 1) // s[1] + 1
    cols = torch.randn(n * oh * ow, c * k[0] * k[1], device="cuda", generator=torch.Generator(device="cuda").manual_seed(h))
    cols[cols.abs() < 0.1] = -0.0
    out = torch.full((n, c + 2, h, w), float("nan"), device="cuda")
    assert be.fold_into(cols, out, 1, c, k, s, p, d)
    want = torch.nn.functional.fold(cols.view(n, oh * ow, -1).transpose(1, 2), (h, w), k, dilation=d, padding=p, stride=s)
    assert torch.equal(out[:, 1:1 + c].contiguous().view(torch.int32), want.view(torch.int32))
    assert out[:, 0].isnan().all() and out[:, 1 + c].isnan().all()      # nothing written beside the channels asked for


def test_shapes_left_to_torch():
    from mptorch_b200 import backend as be

    out = torch.empty(1, 1, 13, 13, device="cuda")
    assert not be.fold_into(torch.empty(1, 169, device="cuda"), out, 0, 1, (13, 13), (1, 1), (0, 0), (1, 1))
    assert not be.fold_into(torch.empty(169, 1, device="cuda").double(), out, 0, 1, (1, 1), (1, 1), (0, 0), (1, 1))


def test_threads_folding_different_shapes():
    """Several host threads, each on a stream of its own, with shapes that take the same kernel and 5 KB or 81 KB of shared
    memory: no thread's launch depends on what another one has set."""
    import threading

    from mptorch_b200 import backend as be

    failures = []

    def work(c, size, k, pad):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                cols = torch.randn(size * size, c * k * k, device="cuda")
                out = torch.empty(1, c, size, size, device="cuda")
                for _ in range(3000):
                    assert be.fold_into(cols, out, 0, c, (k, k), (1, 1), (pad, pad), (1, 1))
                want = torch.nn.functional.fold(cols.view(1, size * size, -1).transpose(1, 2), (size, size), (k, k), padding=pad)
                assert torch.equal(out, want)
        except Exception as e:
            failures.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=a) for a in ((16, 14, 3, 1), (16, 8, 1, 0)) * 3]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[0]
