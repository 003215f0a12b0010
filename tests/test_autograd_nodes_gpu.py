"""The operators' native autograd nodes under what looks at autograd Functions from outside: torch.jit traces, forward-mode
differentiation, torch.func transforms, saved-tensor hooks."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operators():
    """name -> (differentiable function of one tensor, input)"""
    from spherical_distortion import functional as F
    from spherical_distortion.nn import InterpolationType
    g = torch.Generator().manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    it = InterpolationType.BILINEAR
    m = (torch.rand(6, 9, 9, 2, generator=g) * torch.tensor([13.0, 7.0])).cuda()
    w, b, wt, bt, m1 = r(5, 4, 9), r(5), r(4, 5, 9), r(5), m[:, :, 0].contiguous()
    return {"convolution": (lambda x: F.mapped_convolution(x, w, b, m, 9, it), r(2, 4, 8, 14)),
            "convolution_relu": (lambda x: F.mapped_convolution(x, w, b, m, 9, it, activation="relu"), r(2, 4, 8, 14)),
            "transposed": (lambda x: F.mapped_transposed_convolution(x, wt, bt, m, 8, 14, 9, it), r(2, 4, 6, 9)),
            "max_pool": (lambda x: F.mapped_max_pool(x, m, 9, it)[0], r(2, 4, 8, 14)),
            "resample": (lambda x: F.resample(x, m1, (8, 14), it), r(2, 4, 6, 9)),
            "unresample": (lambda x: F.unresample(x, m1, it), r(2, 4, 8, 14))}


NAMES = ["convolution", "convolution_relu", "transposed", "max_pool", "resample", "unresample"]


def _gradient(f, x):
    x = x.clone().requires_grad_(True)
    out = f(x)
    out.backward(torch.arange(out.numel(), device="cuda", dtype=out.dtype).view_as(out))
    return out.detach(), x.grad


@pytest.mark.parametrize("name", NAMES)
def test_traced(name):
    f, x = _operators()[name]
    traced = torch.jit.trace(f, x)
    other = torch.randn(x.shape, generator=torch.Generator().manual_seed(2)).cuda()
    for a, b in zip(_gradient(traced, other), _gradient(f, other)):
        assert torch.equal(a, b)
    with torch.no_grad():
        assert torch.equal(traced(other), f(other))


@pytest.mark.parametrize("name", NAMES)
def test_forward_mode_is_refused(name):
    import torch.autograd.forward_ad as fw
    f, x = _operators()[name]
    with fw.dual_level():
        with pytest.raises(RuntimeError):
            f(fw.make_dual(x, torch.ones_like(x)))


@pytest.mark.parametrize("name", NAMES)
def test_function_transforms_are_refused(name):
    f, x = _operators()[name]
    with pytest.raises(RuntimeError):
        torch.func.vmap(f)(x[None])
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: f(t).sum())(x)


@pytest.mark.parametrize("name", NAMES)
def test_saved_tensor_hooks(name):
    f, x = _operators()[name]
    want = _gradient(f, x)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t) or t.cpu(), lambda t: t.cuda()):
        got = _gradient(f, x)
    assert packed and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("name", NAMES)
def test_undefined_output_gradient_gives_zeros(name):
    class Blocks(torch.autograd.Function):
        forward = staticmethod(lambda ctx, x: x.clone())
        backward = staticmethod(lambda ctx, g: None)

    f, x = _operators()[name]
    x.requires_grad_(True)
    Blocks.apply(f(x)).sum().backward()
    assert x.grad is not None and not x.grad.any()


@pytest.mark.parametrize("weighted", [False, True])
def test_maps_that_require_gradients(weighted):
    """They get none, but the result requires one and backward runs, whatever else takes part."""
    from spherical_distortion import functional as F
    from spherical_distortion.nn import InterpolationType
    it = InterpolationType.NEAREST
    g = torch.Generator().manual_seed(3)
    r = lambda *s: torch.rand(*s, generator=g).cuda()  # noqa: E731
    x, m = r(1, 3, 8, 9), r(8, 9, 4, 2, 2) * 7 if weighted else r(8, 9, 4, 2) * 7
    iw = r(8, 9, 4, 2) if weighted else None
    w, b = r(2, 3, 4), r(2)
    wanting = iw if weighted else m
    m1, iw1 = m[:, :, 0].contiguous(), iw[:, :, 0].contiguous() if weighted else None
    for t in (wanting, iw1 if weighted else m1):
        t.requires_grad_(True)
    for out, t in ((F.mapped_convolution(x, w, b, m, 4, it, iw), wanting),
                   (F.mapped_transposed_convolution(x, w.transpose(0, 1).contiguous(), b, m, 8, 9, 4, it, iw), wanting),
                   (F.mapped_max_pool(x, m, 4, it, iw)[0], wanting),
                   (F.resample(x, m1, (8, 9), it, iw1), iw1 if weighted else m1), (F.unresample(x, m1, it, iw1), iw1 if weighted else m1)):
        assert out.requires_grad
        out.sum().backward()
        assert t.grad is None
    x.requires_grad_(True)
    F.mapped_convolution(x, w, b, m, 4, it, iw).sum().backward()
    assert x.grad.any() and wanting.grad is None
