"""Resampling and pooling over plane groups (the entry points with scratch) against the direct kernels of the same library, which
the other tests compare with the oracle: bit-identical, at plane counts around the group sizes, images whose pixel count is no
multiple of a tile or of four, and maps whose tap table does and does not fit shared memory.  Which kernels ran is read off
the library's launch counter: a direct kernel is one launch, a chunk of plane groups two.  Then the host extension, which
chooses between the two."""
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


def _launches(fn):
    from sphmap import capi
    before = capi.lib.sph_launch_count()
    r = fn()
    return r, capi.lib.sph_launch_count() - before


def _grouped(op, ws):
    """op(ws) over plane groups: two launches, and the bits of op(None), one launch."""
    assert ws is not None
    (got, n), (want, n1) = _launches(lambda: op(ws)), _launches(lambda: op(None))
    assert n == 2 and n1 == 1
    for a, b in zip(*((t if isinstance(t, tuple) else (t,)) for t in (got, want))):
        assert torch.equal(a, b)
    return got


ANY = 1 << 40    # reads enough for the scratch to be reported


@pytest.mark.parametrize("planes", [3, 5, 8, 16, 17, 33, 70])
@pytest.mark.parametrize("interp,P", [(0, 0), (1, 0), (2, 0), (0, 3), (1, 2)])
def test_pooling_matches_direct_kernels(planes, interp, P):
    import _spherical_distortion_ext._C as C
    from sphmap import capi
    it = C.InterpolationType(interp)
    for ih, iw, oh, ow, K in ((7, 9, 6, 11, 9), (16, 20, 9, 17, 20)):
        x, m, w, go = _case(planes, ih, iw, oh, ow, K, P)
        ws = capi.staging(capi.STAGE_POOL, planes, ih * iw, ANY, x)
        ref, ridx = _grouped(lambda s: capi.mapped_max_pool(x, m, K, interp, w, ws=s), ws)
        avg = _grouped(lambda s: capi.mapped_avg_pool(x, m, K, interp, w, ws=s), ws)
        idx = ridx.clone()
        idx[0, 0].view(-1)[:5] = torch.tensor([-1, -2, 1 << 40, 3, 1])          # not this output's slots: no contribution
        plan = capi.slot_plan_build(m, w, K, interp, ih, iw)
        gin = _grouped(lambda s: capi.mapped_max_unpool_planned(go, idx, plan, ih, iw, K, P, ws=s),
                       capi.staging(capi.STAGE_ARGMAX, planes, oh * ow, 0, go))
        out, i = C.weighted_mapped_max_pool(x, m, w, K, it) if P else C.mapped_max_pool(x, m, K, it)
        assert torch.equal(out, ref) and torch.equal(i, ridx)
        assert torch.equal(avg, C.weighted_mapped_avg_pool(x, m, w, K, it) if P else C.mapped_avg_pool(x, m, K, it))
        assert torch.equal(gin, C.weighted_mapped_max_unpool(go, idx, m, w, ih, iw, K, it) if P else
                           C.mapped_max_unpool(go, idx, m, ih, iw, K, it))


@pytest.mark.parametrize("planes", [3, 5, 8, 16, 17, 33, 70])
@pytest.mark.parametrize("interp,P", [(0, 0), (1, 0), (2, 0), (0, 3), (1, 2)])
def test_resampling_matches_direct_kernels(planes, interp, P):
    import _spherical_distortion_ext._C as C
    from sphmap import capi
    it = C.InterpolationType(interp)
    for ih, iw, oh, ow in ((7, 9, 13, 11), (12, 20, 40, 33)):
        x, m, w, go = _case(planes, ih, iw, oh, ow, 1, P, seed=1)
        m, w = m[:, :, 0].contiguous(), w[:, :, 0].contiguous() if P else None
        y = _grouped(lambda s: capi.resample_from_map(x, m, interp, w, ws=s), capi.staging(capi.STAGE_GATHER, planes, ih * iw, ANY, x))
        assert torch.equal(y, C.weighted_resample_from_map(x, m, w, it) if P else C.resample_from_map(x, m, it))
        plan = capi.plan_build(m, w, oh * ow, 1, interp, ih, iw)
        ws = capi.staging(capi.STAGE_SCATTER, planes, oh * ow, 0, go)
        back = _grouped(lambda s: capi.resample_to_map(go, plan, ih, iw, ws=s), ws)
        assert torch.equal(back, C.weighted_resample_to_map(go, m, w, ih, iw, it) if P else C.resample_to_map(go, m, ih, iw, it))
        norm = _grouped(lambda s: capi.resample_to_map_normalized(go, plan, ih, iw, ws=s), ws)
        assert torch.equal(norm, C.resample_to_map_normalized(go, m, w, ih, iw, it))


def _chosen(run, first, then):
    """The host extension's launches of the first call on a map, while nothing is known of it, and of later ones; equal bits."""
    want, n = _launches(run)
    torch.cuda.synchronize()
    assert n == first
    for _ in range(2):
        got, n = _launches(run)
        assert n == then
        for a, b in zip(got, want):
            assert torch.equal(a, b)
    return want


def _map(local, h, w, oh, ow, K):
    from spherical_distortion.util import inverse_gnomonic_projection_map
    if local:
        return inverse_gnomonic_projection_map((h, w), (3, 3), stride=2, device="cuda")
    return torch.rand(oh, ow, K, 2, generator=torch.Generator().manual_seed(3)).mul(torch.tensor([w - 1.0, h - 1.0])).cuda()


@pytest.mark.parametrize("local", [True, False])
def test_nearest_pooling_by_locality(local):
    """Planes are read in place over a local map, in groups over a scattered one or one not looked at yet (one launch more)."""
    from spherical_distortion.nn import InterpolationType, MappedMaxPool
    from sphmap import capi
    m = _map(local, 144, 288, 72, 144, 9)
    assert capi.map_locality(m, 9) == (1 if local else 2)
    x = torch.randn(2, 8, 144, 288, generator=torch.Generator().manual_seed(4)).cuda()
    pool = MappedMaxPool(9, InterpolationType.NEAREST, return_indices=True)
    out, idx = _chosen(lambda: pool(x, m), 3, 1 if local else 2)
    want, at = capi.mapped_max_pool(x, m, 9, 0)
    assert torch.equal(out, want) and torch.equal(idx, at)


@pytest.mark.parametrize("planes,h,w", [(70, 65, 131), (4, 144, 288)])
def test_few_values_are_pooled_in_place(planes, h, w):
    """Nearest neighbours of few values: in place whatever the map, which is not looked at."""
    from spherical_distortion.nn import InterpolationType, MappedMaxPool
    m = _map(False, h, w, 33, 66, 9)
    x = torch.randn(1, planes, h, w, generator=torch.Generator().manual_seed(4)).cuda()
    _chosen(lambda: MappedMaxPool(9, InterpolationType.NEAREST, return_indices=True)(x, m), 1, 1)


@pytest.mark.parametrize("planes,h", [(3, 40), (8, 144), (64, 40), (64, 144)])
@pytest.mark.parametrize("interp", [1, 2])
@pytest.mark.parametrize("local", [True, False])
def test_four_tap_pooling_by_locality(local, interp, planes, h):
    """Four taps: in place over a local map, whatever the planes and the waves of blocks, in groups over a scattered one or one not looked
    at yet (one launch more)."""
    import _spherical_distortion_ext._C as C
    from spherical_distortion.nn import MappedMaxPool
    from sphmap import capi
    m = _map(local, h, 2 * h, h // 2, h, 9)
    x = torch.randn(1, planes, h, 2 * h, generator=torch.Generator().manual_seed(4)).cuda()
    out, idx = _chosen(lambda: MappedMaxPool(9, C.InterpolationType(interp), return_indices=True)(x, m), 3, 1 if local else 2)
    want, at = capi.mapped_max_pool(x, m, 9, interp, ws=capi.staging(capi.STAGE_POOL, planes, 2 * h * h, ANY, x))
    assert torch.equal(out, want) and torch.equal(idx, at)


@pytest.mark.parametrize("planes", [7, 8, 17])
@pytest.mark.parametrize("h,w,oh,ow", [(40, 83, 40, 83), (64, 128, 33, 65), (24, 10, 12, 5), (9, 200, 9, 129)])
@pytest.mark.parametrize("interp", [1, 2])
def test_squares_of_pixels(planes, h, w, oh, ow, interp):
    """Maps whose taps are mostly 2 x 2 pixels inside the image, where the kernels that read in place address them together: outputs
    around the blocks' 64 and 16 columns, taps across every edge, infinities, and coordinates that lie at a multiple of four bytes.
    Against the plane groups, bit for bit."""
    from sphmap import capi
    g = torch.Generator().manual_seed(planes)
    at = torch.stack(torch.meshgrid(torch.arange(oh) * (h / oh), torch.arange(ow) * (w / ow), indexing="ij")[::-1], -1)
    kernel = torch.tensor([[a, b] for b in (-1.25, 0.0, 1.5) for a in (-1.0, 0.25, 1.0)])
    storage = torch.empty(oh * ow * 18 + 1, device="cuda")
    m = storage[1:].view(oh, ow, 9, 2)
    m.copy_(at[:, :, None] + kernel)
    x = torch.randn(1, planes, h, w, generator=g)
    x[0, 0, 3, 5], x[0, 1, 6, 7], x[0, 2, 8, 1] = float("inf"), float("-inf"), float("nan")
    x = x.cuda()
    ws = capi.staging(capi.STAGE_POOL, planes, h * w, ANY, x)
    for smap in (m, m.clone()):
        (a, ia), (b, ib) = capi.mapped_max_pool(x, smap, 9, interp), capi.mapped_max_pool(x, smap, 9, interp, ws=ws)
        assert torch.equal(a, b) and torch.equal(ia, ib)
        one = storage[1:1 + oh * ow * 2].view(oh, ow, 2).copy_(at) if smap is m else smap[:, :, 6].contiguous()
        a, b = capi.resample_from_map(x, one, interp), capi.resample_from_map(x, one, interp, ws=ws)
        assert torch.equal(a.nan_to_num(nan=7.0), b.nan_to_num(nan=7.0))


@pytest.mark.parametrize("interp", [1, 2])
@pytest.mark.parametrize("oh,ow", [(1, 700), (700, 1), (2, 331), (331, 2), (3, 333), (9, 130), (33, 66), (4100, 3), (3, 4100)])
def test_lists_of_positions(oh, ow, interp):
    """Outputs of a few rows or columns, which take tiles of other shapes or none; gathers, pooling and scatters against the plane groups."""
    from sphmap import capi
    x, m, _, go = _case(9, 40, 83, oh, ow, 9, 0, seed=8)
    one = m[:, :, 4].contiguous()
    _grouped(lambda s: capi.resample_from_map(x, one, interp, ws=s), capi.staging(capi.STAGE_GATHER, 9, 40 * 83, ANY, x))
    ws = capi.staging(capi.STAGE_POOL, 9, 40 * 83, ANY, x)
    _grouped(lambda s: capi.mapped_max_pool(x, m, 9, interp, ws=s), ws)
    _grouped(lambda s: capi.mapped_avg_pool(x, m, 9, interp, ws=s), ws)
    at = torch.rand(40, 83, 2, generator=torch.Generator().manual_seed(9)).mul(torch.tensor([ow - 0.5, oh - 0.5])).cuda()
    plan = capi.plan_build(at, None, 40 * 83, 1, interp, oh, ow)
    ws = capi.staging(capi.STAGE_SCATTER, 9, 40 * 83, 0, x)
    _grouped(lambda s: capi.resample_to_map(x, plan, oh, ow, ws=s), ws)
    _grouped(lambda s: capi.resample_to_map_normalized(x, plan, oh, ow, ws=s), ws)


@pytest.mark.parametrize("local", [True, False])
def test_gather_by_locality(local):
    """Between one and eight reads a pixel: in place over a local map or one not looked at yet, in groups over a scattered one."""
    import _spherical_distortion_ext._C as C
    from sphmap import capi
    m = (_map(True, 80, 160, 0, 0, 9)[:, :, 4] if local else _map(False, 80, 160, 40, 80, 1)[:, :, 0]).contiguous()
    x = torch.randn(2, 8, 40, 80, generator=torch.Generator().manual_seed(4)).cuda()
    y, = _chosen(lambda: [C.resample_from_map(x, m, C.InterpolationType.BILINEAR)], 2, 1 if local else 2)
    assert torch.equal(y, capi.resample_from_map(x, m, 1))


@pytest.mark.parametrize("planes", [8, 9, 12, 13, 16, 20, 25])
@pytest.mark.parametrize("h,w", [(8, 33), (17, 64), (30, 5)])
def test_scatter_in_place(planes, h, w):
    """Threads of 8 and of 12 planes, whole and with a remainder, at the edges of blocks of 32 x 8 pixels; against the plane groups."""
    from sphmap import capi
    _, m, _, go = _case(planes, h, w, 2 * h, w, 1, 0, seed=5)
    m = m[:, :, 0].contiguous()
    plan = capi.plan_build(m, None, 2 * h * w, 1, 1, h, w)
    ws = capi.staging(capi.STAGE_SCATTER, planes, 2 * h * w, 0, go)
    _grouped(lambda s: capi.resample_to_map(go, plan, h, w, ws=s), ws)
    _grouped(lambda s: capi.resample_to_map_normalized(go, plan, h, w, ws=s), ws)


@pytest.mark.parametrize("planes", [8, 9, 12, 13, 24, 36])
def test_average_unpooling_by_planes(planes):
    """Threads of 8 and of 12 planes, whole and with a remainder: every plane as if it came alone."""
    from sphmap import capi
    x, m, _, go = _case(planes, 17, 33, 9, 17, 9, 0, seed=10)
    plan = capi.slot_plan_build(m, None, 9, 1, 17, 33)
    got = capi.mapped_avg_unpool(go, plan, 17, 33, 9)
    for j in range(planes):
        assert torch.equal(got[:, j:j + 1], capi.mapped_avg_unpool(go[:, j:j + 1].contiguous(), plan, 17, 33, 9))


def _two_by_two(values, weights, h, w):
    """A map, weights and gradients with which pixel q sums weights[q] * 0 and 1 * values[:, q]."""
    n = h * w
    q = torch.arange(n).repeat_interleave(2)
    m = torch.stack([q % w, q // w], -1).float().view(1, 2 * n, 1, 2)
    iw = torch.stack([weights, torch.ones(n)], -1).view(1, 2 * n, 1)
    go = torch.stack([torch.zeros_like(values), values], -1).view(1, -1, 1, 2 * n)
    return m.cuda(), iw.cuda(), go.cuda()


@pytest.mark.parametrize("kind", ["ordinary", "subnormal", "edges"])
def test_normalised_scatter_divides_in_bounds(kind):
    """Sums and weights between which the division goes by a reciprocal, in the kernel in place and over groups, all planes of a thread
    within its bounds: 200,000 pairs with the quotient that IEEE division gives.  `subnormal`: divisors up to its bound, under values down
    to 2^-80 whose quotients lie half way between two subnormal numbers, on top of one pair that a reciprocal rounds wrongly."""
    from sphmap import capi
    planes, h, w = 9, 160, 139
    n = h * w
    g = torch.Generator().manual_seed(7)
    power = lambda lo, hi, *shape: torch.exp2(torch.randint(lo, hi + 1, shape, generator=g).float())  # noqa: E731
    mantissa = lambda *shape: 1 + torch.rand(*shape, generator=g)  # noqa: E731
    if kind == "ordinary":
        values = torch.randn(planes, n, generator=g) * torch.tensor([1.0, 1e3, 1e-10, 0.0, 1e10, 1e-3, 1.0, 30.0, 1.0])[:, None]
        weights = mantissa(n) * power(-20, 20, n)
    elif kind == "subnormal":
        values = 3 * (2 * torch.randint(1000, 1 << 21, (planes, n), generator=g) + 1).double() * 2.0 ** -92
        weights = torch.full((n,), 3 * 2.0 ** 58)
        values[:, 0], weights[0] = float.fromhex("0x1.51b5dep-79"), float.fromhex("0x1.faep+59")
        assert torch.equal(values.float().double(), values)
        values = values.float()
    else:
        values, weights = mantissa(planes, n) * power(-62, 59, planes, n), mantissa(n) * power(-40, 59, n)
    m, iw, go = _two_by_two(values, weights, h, w)
    plan = capi.plan_build(m, iw, 2 * n, 1, 0, h, w)
    den = ((weights + 1.0) + torch.tensor(1e-12)).numpy()
    want = torch.from_numpy(values.numpy() / den).view(1, planes, h, w)
    for ws in (None, capi.staging(capi.STAGE_SCATTER, planes, 2 * n, 0, go)):
        assert torch.equal(capi.resample_to_map_normalized(go, plan, h, w, ws=ws).cpu(), want)


def test_normalised_scatter_divides():
    """sum / (weights + 1e-12) with the rounding of a division, also for values that have none of the usual magnitudes, which are
    divided.  (Such a plane takes the others of its thread along.)"""
    from sphmap import capi
    h, w = 16, 40
    _, m, iw, go = _case(9, h, w, 2 * h, w, 1, 1, seed=6)
    m, iw = m[:, :, 0].contiguous(), iw[:, :, 0].contiguous()
    scale = torch.tensor([1.0, 1e-38, 1e38, 1e-25, 0.0, 1e20, 3e-45, 1e3, float("inf")]).cuda()
    go *= scale.view(1, 9, 1, 1)
    for weights in (iw, iw * 1e-20, -iw, iw * 1e25):
        plan = capi.plan_build(m, weights, 2 * h * w, 1, 1, h, w)
        total = capi.resample_to_map(go, plan, h, w)
        den = capi.resample_to_map(torch.ones_like(go[:, :1]), plan, h, w) + 1e-12
        want = torch.where(total == 0, total, total / den)
        for ws in (None, capi.staging(capi.STAGE_SCATTER, 9, 2 * h * w, 0, go)):
            got = capi.resample_to_map_normalized(go, plan, h, w, ws=ws)
            assert torch.equal(got.nan_to_num(nan=7.0), want.nan_to_num(nan=7.0))


@pytest.mark.parametrize("local", [True, False])
def test_scatter_by_locality(local):
    """In place over a local map, in groups over a scattered one, one not looked at yet and one of many positions per pixel."""
    import _spherical_distortion_ext._C as C
    m = (_map(True, 40, 80, 0, 0, 9)[:, :, 4] if local else _map(False, 40, 80, 20, 40, 1)[:, :, 0]).contiguous()
    x = torch.randn(2, 8, 20, 40, generator=torch.Generator().manual_seed(4)).cuda()
    for run in (C.resample_to_map, lambda x, m, h, w, it: C.resample_to_map_normalized(x, m, None, h, w, it)):
        C.clear_plan_cache()
        smap = m.clone()
        run(x, smap, 40, 80, C.InterpolationType.BILINEAR)    # (the plan)
        seen, n = _launches(lambda: run(x, smap, 40, 80, C.InterpolationType.BILINEAR))
        assert n == 3                                         # (a look at the map)
        torch.cuda.synchronize()
        got, n = _launches(lambda: run(x, smap, 40, 80, C.InterpolationType.BILINEAR))
        assert n == (1 if local else 2)
        few, n = _launches(lambda: run(x, smap, 19, 20, C.InterpolationType.BILINEAR))
        assert n > 2


@pytest.mark.parametrize("h,w,face,planes,normalised,in_place", [
    (141, 282, 16, 16, False, True),      # a small image
    (141, 282, 61, 24, False, False),     # two positions per pixel of it, more than 16 planes
    (512, 1024, 84, 3, False, True),      # half-empty threads, a quarter of a position per pixel of half a million
    (512, 1024, 84, 4, True, False),      # the same, normalised
    (300, 601, 37, 8, True, True),
    (300, 601, 37, 24, False, True),      # threads of 12 planes
    (300, 601, 37, 48, False, False),     # many of them, few positions
    (300, 601, 85, 16, False, False),     # one whole group
    (256, 512, 0, 16, False, True),       # the same, a map of the image's proportions
])
def test_scatter_by_planes_and_positions(h, w, face, planes, normalised, in_place):
    """Over local maps the faster of the two kernels, with the same bits."""
    import _spherical_distortion_ext._C as C
    from sphmap import capi
    from sphmap.workloads import tangent_image_map
    m = tangent_image_map(h, w, face).cuda() if face else _map(True, h, w, 0, 0, 9)[:, :, 4].contiguous()
    x = torch.randn(1, planes, *m.shape[:2], generator=torch.Generator().manual_seed(4)).cuda()
    it = C.InterpolationType.BILINEAR
    run = lambda: C.resample_to_map_normalized(x, m, None, h, w, it) if normalised else C.resample_to_map(x, m, h, w, it)  # noqa: E731
    want = run()
    for _ in range(2):    # (the plan, a look at the map)
        run()
        torch.cuda.synchronize()
    got, n = _launches(run)
    assert n == (1 if in_place else 2)
    assert torch.equal(got, want)
    C.clear_plan_cache()


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
