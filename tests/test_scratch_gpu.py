"""Operators whose scratch is optional, where the memory for it is not to be had: they run with the smaller scratch."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _short_of_memory(fn, spare):
    """fn() with the allocator held to `spare` bytes beyond what it has."""
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + spare) / total)
    try:
        return fn()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)


def _case(cin, cout, h, w, oh, ow, K):
    g = torch.Generator().manual_seed(cin)
    r = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    m = (torch.rand(oh, ow, K, 2, generator=g) * torch.tensor([w - 1.0, h - 1.0])).cuda()
    return r, m


@pytest.mark.parametrize("op", ["convolution", "relu", "transposed"])
def test_convolutions(op):
    """64 channels of 4 x 128 x 256: every tensor takes 34 MB; results and plan fit, a channels-last copy does not."""
    import _spherical_distortion_ext._C as C
    r, m = _case(64, 64, 128, 256, 128, 256, 4)
    x, w, b, go = r(4, 64, 128, 256), r(64, 64, 4), r(64), r(4, 64, 128, 256)
    it = C.InterpolationType.BILINEAR

    def run():
        if op == "convolution":
            return [C.mapped_conv_forward(x, m, w, b, 4, it)], lambda: C.mapped_conv_backward(go, m, x, w, b, 4, it)
        if op == "relu":
            out = C.mapped_conv_relu_forward(x, m, None, w, b, 4, it)
            return [out], lambda: C.mapped_conv_relu_backward(go, out, m, None, x, w, b, 4, it)
        return [C.mapped_transposed_conv_forward(x, m, w, b, 128, 256, 4, it)], lambda: C.mapped_transposed_conv_backward(go, m, x, w, b, 4, it)

    forward, backward = run()
    want = [t.cpu() for t in forward + list(backward())]
    forward, backward = _short_of_memory(run, 60 << 20)   # (34 MB, and 22 in the allocator's steps for small ones)
    more = 60 << 20 if op != "relu" else 110 << 20       # (the masked gradient is a tensor more)
    got = [t.cpu() for t in forward + list(_short_of_memory(backward, more))]
    for a, b_ in zip(got, want):
        assert ((a - b_).norm() / b_.norm()).item() < 5e-6


@pytest.mark.parametrize("op", ["max_pool", "avg_pool", "unpool", "gather", "scatter"])
def test_plane_groups(op):
    """64 planes of 256 x 512 (34 MB) or their results: the transposed copies do not fit, the bits are the same."""
    import _spherical_distortion_ext._C as C
    it = C.InterpolationType.BILINEAR
    if op == "gather":
        r, m = _case(1, 1, 256, 512, 1024, 512, 1)
        x, m = r(1, 64, 256, 512), m[:, :, 0].contiguous()
        run, spare = lambda: [C.resample_from_map(x, m, it)], 140 << 20
    elif op == "scatter":
        r, m = _case(1, 1, 128, 256, 256, 512, 1)
        x, m = r(1, 64, 256, 512), m[:, :, 0].contiguous()
        run, spare = lambda: [C.resample_to_map(x, m, 128, 256, it)], 24 << 20
    else:
        r, m = _case(1, 1, 256, 512, 128, 256, 9)
        x, g = r(1, 64, 256, 512), r(1, 64, 128, 256)
        idx = C.mapped_max_pool(x, m, 9, it)[1]
        run, spare = {"max_pool": (lambda: C.mapped_max_pool(x, m, 9, it), 46 << 20),
                      "avg_pool": (lambda: [C.mapped_avg_pool(x, m, 9, it)], 24 << 20),
                      "unpool": (lambda: [C.mapped_max_unpool(g, idx, m, 256, 512, 9, it)], 38 << 20)}[op]
    want = run()
    for a, b in zip(_short_of_memory(run, spare), want):
        assert torch.equal(a, b)
