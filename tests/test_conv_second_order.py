"""Second derivatives and batched gradients of QConv2d where the backward pass is plain torch arithmetic (formats for the forward
multiply-accumulates only), and the fold kernel in an ordinary backward pass."""
import pytest
import torch

CASES = [(2, 4, 6, 3, 1, 1), (2, 4, 6, 3, 1, 2), (1, 3, 5, 2, 2, 1)]        # batch, channels in and out, kernel, stride, groups


def make(case, device):
    import mptorch_b200.quant as q
    from mptorch_b200 import FloatingPoint

    n, cin, cout, k, stride, groups = case
    torch.manual_seed(5)
    f = q.QAffineFormats(fwd_mac=(FloatingPoint(5, 10, True, False), FloatingPoint(4, 3, True, False)))
    conv = q.QConv2d(cin, cout, k, f, stride=stride, padding=k // 2, groups=groups).to(device)
    x = torch.randn(n, cin, 7, 8, device=device, requires_grad=True)
    return conv, x


def first_and_second(conv, x):
    """First gradients of the output against a fixed direction, and the gradients of their squared norm with respect to that
    direction, the input and the weight."""
    y = conv(x)
    g = torch.randn(y.shape, device=y.device, generator=torch.Generator(y.device).manual_seed(9)).requires_grad_()
    first = torch.autograd.grad(y, [x, conv.weight, conv.bias], g, create_graph=True)
    assert all(t.requires_grad for t in first)
    return list(first) + list(torch.autograd.grad(sum(t.square().sum() for t in first), [g, x, conv.weight]))


def plain_forward(x, wt, out, groups, kernel_size, stride, padding, dilation, *a, **k):
    """Stands in for the implicit GEMM where there is no GPU; the backward pass is what is looked at."""
    w = wt.transpose(1, 2).reshape(out.shape[1], -1, *kernel_size)
    out.copy_(torch.nn.functional.conv2d(x, w, None, stride, padding, dilation, groups))


def test_batched_gradients_of_a_grouped_convolution(monkeypatch):
    import mptorch_b200.backend as be
    from mptorch_b200.quant.functional import qconv2d

    monkeypatch.setattr(be, "float_conv2d_nearest", plain_forward)
    conv, x = make((2, 4, 6, 3, 1, 2), "cpu")
    y = qconv2d(x, conv.weight, conv.bias, conv.formats, (1, 1), (1, 1), (1, 1), 2)
    many = torch.randn(3, *y.shape)
    got = torch.autograd.grad(y, [x, conv.weight, conv.bias], many, is_grads_batched=True, retain_graph=True)
    for i in range(3):
        for a, b in zip(got, torch.autograd.grad(y, [x, conv.weight, conv.bias], many[i], retain_graph=True)):
            torch.testing.assert_close(a[i], b, rtol=1e-5, atol=1e-5)


def test_raw_memory_is_not_used_under_a_graph_or_vmap():
    from mptorch_b200.quant.functional import _by_pointer

    t = torch.randn(3, 4, requires_grad=True)
    assert not _by_pointer(t) and not _by_pointer(t * 2)
    with torch.no_grad():
        assert _by_pointer(t * 2)
    seen = []
    torch.vmap(lambda v: (seen.append(_by_pointer(v)), v * 2)[1])(t.detach())
    x = torch.randn(3, requires_grad=True)
    y = x * 2
    y.register_hook(lambda g: (seen.append(_by_pointer(g)), g)[1])
    torch.autograd.grad(y, x, torch.eye(3), is_grads_batched=True)
    assert seen == [False, False]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_second_derivatives_match_the_composition(case, monkeypatch):
    import mptorch_b200.quant.modules as modules

    conv, x = make(case, "cuda")
    taken = []
    real = modules.qconv2d
    monkeypatch.setattr(modules, "qconv2d", lambda *a, **k: (taken.append(1), real(*a, **k))[1])
    got = first_and_second(conv, x)
    assert taken
    monkeypatch.setattr(modules, "implicit_conv_eligible", lambda f, t: False)
    want = first_and_second(conv, x)
    # fp32 sums of at most a few hundred terms in another order, squared and summed again: 2^-24 times a few hundred
    for a, b in zip(got, want):
        assert (a - b).norm() <= 1e-4 * b.norm()


@pytest.mark.gpu
def test_batched_gradients_on_the_gpu():
    conv, x = make((2, 4, 6, 3, 1, 2), "cuda")
    y = conv(x)
    many = torch.randn(3, *y.shape, device="cuda")
    got = torch.autograd.grad(y, [x, conv.weight, conv.bias], many, is_grads_batched=True, retain_graph=True)
    for i in range(3):
        for a, b in zip(got, torch.autograd.grad(y, [x, conv.weight, conv.bias], many[i], retain_graph=True)):
            assert (a[i] - b).norm() <= 1e-5 * b.norm()


@pytest.mark.gpu
@pytest.mark.parametrize("size,low,kernel", [(7, False, False), (7, True, True), (64, False, True)])
def test_ordinary_backward_takes_the_fold_kernel(monkeypatch, size, low, kernel):
    """Where the backward pass has its own formats, and in the default one from the size on that repays the call."""
    import mptorch_b200.backend as be
    import mptorch_b200.quant as q
    from mptorch_b200 import FloatingPoint

    took = []
    real = be.fold_into
    monkeypatch.setattr(be, "fold_into", lambda *a: (took.append(real(*a)), took[-1])[1])
    mac = (FloatingPoint(5, 10, True, False), FloatingPoint(4, 3, True, False))
    conv = q.QConv2d(16, 6, 3, q.QAffineFormats(fwd_mac=mac, **({"bwd_mac": mac} if low else {})), padding=1, groups=2).cuda()
    x = torch.randn(2, 16, size, size, device="cuda", requires_grad=True)
    y = conv(x)
    g = torch.randn_like(y)
    y.backward(g)
    assert took == ([True, True] if kernel else [])
    if not low:
        want = torch.nn.grad.conv2d_input(x.shape, conv.weight, g, padding=1, groups=2)
        assert (x.grad - want).norm() <= 1e-5 * want.norm()
