"""Kept scatter plans and CUDA graphs: a plan is read only where it exists, and for as long as a graph reads it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case():
    from spherical_distortion import functional as F
    from spherical_distortion.nn import InterpolationType
    g = torch.Generator().manual_seed(0)
    m = (torch.rand(20, 30, 2, generator=g) * torch.tensor([15.0, 9.0])).cuda()
    x = torch.randn(2, 5, 20, 30, generator=g).cuda()
    return (lambda t, q: F.resample(t, q, (10, 16), InterpolationType.BILINEAR)), x, m


def test_a_plan_from_before_serves_a_capture_on_another_stream():
    """Warm-up on one stream, capture on another (the usual order), eviction pressure in between: replays follow the input."""
    op, x, m = _case()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        op(x, m)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = op(x, m)
    maps = [m * (i / 70) for i in range(70)]     # more than are kept
    for q in maps:
        op(x, q)
    fill = [torch.full((1 << 16,), -1, dtype=torch.int32, device="cuda") for _ in range(64)]   # (over what an evicted plan held)
    for k in range(3):
        x.copy_(torch.randn(x.shape, generator=torch.Generator().manual_seed(k)))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, op(x.clone(), m.clone()))
    del fill


def test_a_plan_built_in_a_capture_serves_that_alone():
    """An ordinary call between the capture that first met the map and its replay builds a plan of its own."""
    op, x, m = _case()
    want = op(x, m.clone())
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = op(x, m)
        z = op(x + 1, m)
    assert torch.equal(op(x, m), want)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want) and torch.equal(z, op(x + 1, m))
