"""Channels-last copies of activations (bf16 precision) are found again only where they hold what the tensor holds: not by the
replays of a CUDA graph, on another stream, or for tensors whose modifications nothing counts."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _bf16():
    import _spherical_distortion_ext as ext
    ext.set_precision("bf16")
    yield
    ext.set_precision("fp32")


def _layers():
    from spherical_distortion.nn import InterpolationType, MappedConvolution
    from spherical_distortion.util import inverse_gnomonic_projection_map
    torch.manual_seed(0)
    m = inverse_gnomonic_projection_map((16, 32), (3, 3), stride=1, device="cuda")
    a = MappedConvolution(64, 64, 9, InterpolationType.BILINEAR, activation="relu").cuda()
    b = MappedConvolution(64, 64, 9, InterpolationType.BILINEAR).cuda()
    return a, b, m


def _inputs(n):
    g = torch.Generator().manual_seed(1)
    return [torch.randn(2, 64, 16, 32, generator=g).cuda() for _ in range(n)]


def test_replays_read_the_inputs_of_their_own():
    """Captured on a tensor that a warm-up call has seen, on the warm-up's stream: replays convert what it holds then."""
    a, b, m = _layers()
    first, *others = _inputs(4)
    x = first.clone()

    def step(t):
        t = t.detach().requires_grad_(True)
        out = b(a(t, m), m)
        return out.detach(), torch.autograd.grad(out, t, out.detach())[0]

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        for _ in range(2):
            step(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        got = step(x)
    with torch.cuda.stream(stream):      # an ordinary call between capture and replay finds no copy of the capture's either
        eager = step(x)
    torch.cuda.synchronize()
    for u, v in zip(eager, step(first.clone())):
        assert torch.equal(u, v)
    for other in others:
        x.copy_(other)
        graph.replay()
        torch.cuda.synchronize()
        for u, v in zip(got, step(other.clone())):
            assert torch.equal(u, v)


def test_inference_tensors_modified_in_place():
    a, b, m = _layers()
    first, other = _inputs(2)
    with torch.inference_mode():
        x = first.clone()
        b(x, m)
        x.copy_(other)
        assert torch.equal(b(x, m), b(other.clone(), m))
        h = a(x, m)
        h += 1.0
        assert torch.equal(b(h, m), b(h.clone(), m))


def test_copies_serve_their_own_stream():
    """The copy is made behind a long queue on one stream; another one does not read it unfinished."""
    _, b, m = _layers()
    x, = _inputs(1)
    want = b(x.clone(), m)
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    big = torch.empty(1 << 30, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(one):
        for _ in range(20):
            big.fill_(1)
        late = b(x, m)
    with torch.cuda.stream(two):
        early = b(x, m)
    torch.cuda.synchronize()
    assert torch.equal(early, want) and torch.equal(late, want)
