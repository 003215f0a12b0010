"""Resampling and pooling over plane groups (the kernels the host extension selects by giving them scratch) against the
direct kernels of the same library, which the other tests compare with the oracle: bit-identical, at plane counts around
the group sizes, images whose pixel count is no multiple of a tile or of four, and maps whose tap table does and does not
fit shared memory."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(planes, ih, iw, oh, ow, K, P, seed=0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(1, planes, ih, iw, generator=g)
    shape = (oh, ow, K, P, 2) if P else (oh, ow, K, 2)
    m = torch.rand(*shape, generator=g) * torch.tensor([iw + 3.0, ih + 3.0]) - 2.0
    w = torch.rand(oh, ow, K, P, generator=g) if P else None
    go = torch.randn(1, planes, oh, ow, generator=g)
    return [t.cuda() if t is not None else None for t in (x, m, w, go)]


@pytest.mark.parametrize("planes", [3, 5, 8, 16, 17, 33, 70])
@pytest.mark.parametrize("interp,P", [(0, 0), (1, 0), (2, 0), (0, 3), (1, 2)])
def test_pooling_matches_direct_kernels(planes, interp, P):
    import _spherical_distortion_ext._C as C
    from sphmap import capi
    it = C.InterpolationType(interp)
    for ih, iw, oh, ow, K in ((7, 9, 6, 11, 9), (16, 20, 9, 17, 20)):
        x, m, w, go = _case(planes, ih, iw, oh, ow, K, P)
        assert capi.lib.sph_staging_bytes(1, *capi._ints(planes, ih * iw, oh * ow * K), 0) > 0
        out, idx = C.weighted_mapped_max_pool(x, m, w, K, it) if P else C.mapped_max_pool(x, m, K, it)
        ref, ridx = capi.mapped_max_pool(x, m, K, interp, w)
        assert torch.equal(out, ref) and torch.equal(idx, ridx)
        avg = C.weighted_mapped_avg_pool(x, m, w, K, it) if P else C.mapped_avg_pool(x, m, K, it)
        assert torch.equal(avg, capi.mapped_avg_pool(x, m, K, interp, w))
        idx[0, 0].view(-1)[:5] = torch.tensor([-1, -2, 1 << 40, 3, 1])          # not this output's slots: no contribution
        gin = C.weighted_mapped_max_unpool(go, idx, m, w, ih, iw, K, it) if P else C.mapped_max_unpool(go, idx, m, ih, iw, K, it)
        plan = capi.slot_plan_build(m, w, K, interp, ih, iw)
        assert torch.equal(gin, capi.mapped_max_unpool_planned(go, idx, plan, ih, iw, K, P))


@pytest.mark.parametrize("planes", [3, 5, 8, 16, 17, 33, 70])
@pytest.mark.parametrize("interp,P", [(0, 0), (1, 0), (2, 0), (0, 3), (1, 2)])
def test_resampling_matches_direct_kernels(planes, interp, P):
    import _spherical_distortion_ext._C as C
    from sphmap import capi
    it = C.InterpolationType(interp)
    for ih, iw, oh, ow in ((7, 9, 13, 11), (12, 20, 40, 33)):
        x, m, w, go = _case(planes, ih, iw, oh, ow, 1, P, seed=1)
        m, w = m[:, :, 0].contiguous(), w[:, :, 0].contiguous() if P else None
        assert capi.lib.sph_staging_bytes(0, *capi._ints(planes, ih * iw, oh * ow), 0) > 0
        y = C.weighted_resample_from_map(x, m, w, it) if P else C.resample_from_map(x, m, it)
        assert torch.equal(y, capi.resample_from_map(x, m, interp, w))
        plan = capi.plan_build(m, w, oh * ow, 1, interp, ih, iw)
        back = C.weighted_resample_to_map(go, m, w, ih, iw, it) if P else C.resample_to_map(go, m, ih, iw, it)
        assert torch.equal(back, capi.resample_to_map(go, plan, ih, iw))
        norm = C.resample_to_map_normalized(go, m, w, ih, iw, it)
        assert torch.equal(norm, capi.resample_to_map_normalized(go, plan, ih, iw))


@pytest.mark.parametrize("local", [True, False])
def test_nearest_pooling_by_locality(local):
    """The host extension reads the planes in place over a local map, once it knows that the map is one: same bits."""
    import ctypes
    from spherical_distortion.nn import InterpolationType, MappedMaxPool
    from spherical_distortion.util import inverse_gnomonic_projection_map
    from sphmap import capi
    H, W = 66, 131
    if local:
        m = inverse_gnomonic_projection_map((H, W), (3, 3), stride=2, device="cuda")
    else:
        m = torch.rand(33, 66, 9, 2, generator=torch.Generator().manual_seed(3)).mul(torch.tensor([W - 1.0, H - 1.0])).cuda()
    x = torch.randn(2, 35, H, W, generator=torch.Generator().manual_seed(4)).cuda()
    n = m.shape[0] * m.shape[1]
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")
    capi._ok(capi.lib.sph_map_locality(capi._ptr(m), ctypes.c_int64(n), ctypes.c_int64(9), capi._ptr(flag), capi._stream()), "locality")
    assert flag.item() == (1 if local else 2)
    pool = MappedMaxPool(9, InterpolationType.NEAREST, return_indices=True)
    runs = []
    for _ in range(3):
        runs.append(pool(x, m))
        torch.cuda.synchronize()
    for out, idx in runs[1:]:
        assert torch.equal(out, runs[0][0]) and torch.equal(idx, runs[0][1])
    want, at = capi.mapped_max_pool(x, m, 9, 0)
    assert torch.equal(runs[0][0], want) and torch.equal(runs[0][1], at)


@pytest.mark.parametrize("planes", [3, 8, 16])
def test_scatter_with_a_plan_of_another_size_yields_zeros(planes):
    """A plan that was built for another destination, or is none, is not followed: zeros, as from the direct kernel."""
    from sphmap import capi
    _, m, _, go = _case(planes, 6, 7, 13, 11, 1, 0)
    m = m[:, :, 0].contiguous()
    ws = capi.staging(capi.STAGE_SCATTER, planes, 13 * 11, 0, go)
    smaller = capi.plan_build(m, None, 13 * 11, 1, 1, 6, 7)
    for plan in (smaller, torch.zeros_like(smaller)):
        for scratch in (None, ws):
            assert not capi.resample_to_map(go, plan, 60, 70, ws=scratch).any()
