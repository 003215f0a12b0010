"""float32 convolutions through three-way split operands on the tensor cores (what the host extension runs in the exact
precision) against the library's float64 kernels, beside the float32 SIMT kernels (what the C ABI runs with the smaller
scratch): no less accurate than those, at channel counts around the padding steps, row counts around the 128-row blocks,
ragged grids, every kind of map, and adjoints over down-sampling maps (multiply first)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

#        B, Cin, Cout, (H, W), (OH, OW), K, interpolation, points
CASES = [(2, 16, 32, (16, 32), (16, 32), 9, 1, 0),
         (3, 20, 37, (45, 91), (45, 91), 9, 2, 0),
         (1, 5, 33, (8, 16), (8, 16), 9, 1, 0),
         (1, 64, 129, (9, 17), (8, 15), 9, 0, 0),
         (2, 40, 200, (20, 30), (7, 11), 9, 1, 0),
         (1, 100, 50, (20, 33), (20, 33), 5, 0, 3),
         (1, 96, 16, (24, 40), (24, 40), 25, 1, 0),
         (1, 260, 256, (16, 32), (16, 32), 9, 1, 0),
         (3, 16, 40, (64, 128), (64, 128), 9, 1, 0),  # more tiles than SMs, several images: every block takes a second tile
         (2, 40, 24, (72, 136), (72, 136), 4, 0, 0),
         (4, 40, 48, (128, 256), (64, 128), 9, 1, 0), # the same where the adjoints multiply first (tiles of one segment)
         (1, 300, 320, (9, 17), (9, 17), 9, 2, 0),    # products of 90 chunks: more than one run of small products
         (1, 8200, 16, (4, 8), (4, 8), 9, 1, 0)]     # dW: the first column group of two slots is the 65th


def _rel(a, ref):
    return ((a.double() - ref).norm() / ref.norm()).item()


@pytest.mark.parametrize("case", CASES)
def test_split_products_are_float32_accurate(case):
    import _spherical_distortion_ext._C as C
    from sphmap import capi
    B, ci, co, (H, W), (OH, OW), K, interp, P = case
    g = torch.Generator().manual_seed(ci)
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    x, w, b, go = r(B, ci, H, W), r(co, ci, K) / 30, r(co), r(B, co, OH, OW)
    m = torch.rand(*((OH, OW, K, P, 2) if P else (OH, OW, K, 2)), generator=g) * torch.tensor([W + 1.0, H + 1.0]) - 1.0
    iw = torch.rand(OH, OW, K, P, generator=g) if P else None
    wt, bt, xt, got = r(ci, co, K) / 30, r(co), r(B, ci, OH, OW), r(B, co, H, W)
    dev = lambda *t: [None if v is None else v.cuda() for v in t]  # noqa: E731
    dbl = lambda *t: [None if v is None else v.double() for v in t]  # noqa: E731

    def simt(x, w, b, go, m, iw, wt, bt, xt, got):
        plan = capi.plan_build(m, iw, OH * OW, K, interp, H, W)
        return [capi.conv_forward(x, m, w, b, K, interp, iw), capi.conv_backward_input(go, plan, w, H, W, K),
                *capi.conv_backward_weight(go, x, m, K, interp, iw), capi.tconv_forward(xt, plan, wt, bt, H, W, K),
                capi.tconv_backward_input(got, m, wt, K, interp, iw), *capi.tconv_backward_weight(got, xt, m, K, interp, iw)]

    a = dev(x, w, b, go, m, iw, wt, bt, xt, got)
    ref, old = simt(*dbl(*a)), simt(*a)
    x, w, b, go, m, iw, wt, bt, xt, got = a
    it, ws = C.InterpolationType(interp), (m, iw) if P else (m,)
    name = "weighted_" if P else ""
    new = [getattr(C, name + "mapped_conv_forward")(x, *ws, w, b, K, it), *getattr(C, name + "mapped_conv_backward")(go, *ws, x, w, b, K, it),
           getattr(C, name + "mapped_transposed_conv_forward")(xt, *ws, wt, bt, H, W, K, it),
           *getattr(C, name + "mapped_transposed_conv_backward")(got, *ws, xt, wt, bt, K, it)]
    for what, n, o, f in zip(("forward", "dInput", "dW", "dBias", "t forward", "t dInput", "t dW", "t dBias"), new, old, ref):
        assert _rel(n, f) <= 1.25 * _rel(o, f) + 5e-8, (what, _rel(n, f), _rel(o, f))
    assert capi.device_status() == 0


def test_cancellation_and_one_sided_sums():
    """Sums of one sign (where truncating accumulation would drift) and sums that cancel."""
    import _spherical_distortion_ext._C as C
    from sphmap import capi
    g = torch.Generator().manual_seed(7)
    B, ci, co, H, W, K = 2, 256, 64, 16, 64, 9
    m = (torch.rand(H, W, K, 2, generator=g) * torch.tensor([W - 1.0, H - 1.0])).cuda()
    for sign in ("positive", "alternating"):
        x, w, go = (torch.rand(*s, generator=g).cuda() + 0.5 for s in ((B, ci, H, W), (co, ci, K), (B, co, H, W)))
        if sign == "alternating":
            w[:, ::2] *= -1
            go[..., ::2] *= -1
        b = torch.zeros(co, device="cuda")
        it = C.InterpolationType(1)
        new = [C.mapped_conv_forward(x, m, w, b, K, it), *C.mapped_conv_backward(go, m, x, w, b, K, it)]
        def simt(x, m, w, b, go):
            plan = capi.plan_build(m, None, H * W, K, 1, H, W)
            return [capi.conv_forward(x, m, w, b, K, 1), capi.conv_backward_input(go, plan, w, H, W, K), *capi.conv_backward_weight(go, x, m, K, 1)]
        old, ref = simt(x, m, w, b, go), simt(*(t.double() for t in (x, m, w, b, go)))
        for what, n, o, f in zip(("forward", "dInput", "dW"), new, old, ref):
            assert _rel(n, f) <= 1.25 * _rel(o, f) + 5e-8, (sign, what, _rel(n, f), _rel(o, f))


def test_long_one_sided_reduction():
    """Weight gradient whose blocks reduce 768 tiles each (147 column groups, so one split): 3072 steps of products of one sign.
    Each step cuts ten small products (2^-7 of the sum at most) and, per two steps, four large ones off toward zero, about
    5e-8 of an accumulator each.  With at most 800 small ones to an accumulator that is 4e-7 + 2e-7; rounding 1536 float32
    additions adds 2^-25 sqrt(1536 / 3) = 7e-7.  An accumulator of all 30720 would be off by 1.6e-5 on its own."""
    import _spherical_distortion_ext._C as C
    from sphmap import capi
    g = torch.Generator().manual_seed(11)
    B, ci, co, H, W, K = 768, 384, 16, 8, 16, 49
    m = (torch.rand(H, W, K, 2, generator=g) * torch.tensor([W - 1.0, H - 1.0])).cuda()
    x, w, go = (torch.rand(*s, generator=g).cuda() + 0.5 for s in ((B, ci, H, W), (co, ci, K), (B, co, H, W)))
    new = C.mapped_conv_backward(go, m, x, w, torch.zeros(co, device="cuda"), K, C.InterpolationType(1))[1]
    old = capi.conv_backward_weight(go, x, m, K, 1)[0]
    ref = capi.conv_backward_weight(go.double(), x.double(), m.double(), K, 1)[0]
    assert _rel(new, ref) <= 1.5e-6, (_rel(new, ref), _rel(old, ref))


@pytest.mark.parametrize("case", [(2, 16, 32, (16, 32), (16, 32), 9, 1, 0), (1, 40, 48, (24, 40), (11, 19), 9, 0, 0),
                                  (1, 20, 32, (9, 17), (9, 17), 4, 0, 3), (1, 300, 32, (9, 17), (9, 17), 9, 1, 0)])
@pytest.mark.parametrize("kind", ["inf", "mixed", "overflow"])
def test_infinities_and_nans_are_those_of_float32(case, kind):
    """Infinite and NaN operands (one NaN with its payload in the lower half alone) and products beyond the float32 range: the same
    elements of every result are NaN, plus and minus infinity as from the CUDA cores."""
    import _spherical_distortion_ext._C as C
    from sphmap import capi
    B, ci, co, (H, W), (OH, OW), K, interp, P = case
    g = torch.Generator().manual_seed(co)
    r = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    x, w, b, go = r(B, ci, H, W), r(co, ci, K), r(co), r(B, co, OH, OW)
    wt, bt, xt, got = r(ci, co, K), r(co), r(B, ci, OH, OW), r(B, co, H, W)
    m = torch.rand(*((OH, OW, K, P, 2) if P else (OH, OW, K, 2)), generator=g) * torch.tensor([W + 1.0, H + 1.0]) - 1.0
    iw = torch.rand(OH, OW, K, P, generator=g) if P else None
    odd_nan = torch.tensor([0x7f800001], dtype=torch.int32).view(torch.float32)
    if kind == "overflow":  # (of one sign: with two, whether a sum overflows depends on its order)
        x, w, b, go, wt, bt, xt, got = (t.abs() + 0.5 for t in (x, w, b, go, wt, bt, xt, got))
    for t in (x, go, xt, got):
        if kind == "overflow":
            t[0, 0, 3, 4] = 3e38
            continue
        t[0, 0, 3, 4] = float("inf")
        t[0, 1, 2, 7] = float("-inf")
        if kind == "mixed":
            t[-1, 2, 6, 1] = odd_nan[0]
            t[-1, 3, 5, 5] = float("nan")
    if kind == "mixed":
        w[1, 2, 3], w[2, 0, 1], wt[1, 2, 3], wt[2, 1, 0] = float("inf"), odd_nan[0], float("-inf"), float("nan")
    x, w, b, go, m, iw, wt, bt, xt, got = (None if t is None else t.cuda() for t in (x, w, b, go, m, iw, wt, bt, xt, got))
    plan = capi.plan_build(m, iw, OH * OW, K, interp, H, W)
    old = [capi.conv_forward(x, m, w, b, K, interp, iw), capi.conv_backward_input(go, plan, w, H, W, K),
           *capi.conv_backward_weight(go, x, m, K, interp, iw), capi.tconv_forward(xt, plan, wt, bt, H, W, K),
           capi.tconv_backward_input(got, m, wt, K, interp, iw), *capi.tconv_backward_weight(got, xt, m, K, interp, iw)]
    it, ws = C.InterpolationType(interp), (m, iw) if P else (m,)
    name = "weighted_" if P else ""
    new = [getattr(C, name + "mapped_conv_forward")(x, *ws, w, b, K, it), *getattr(C, name + "mapped_conv_backward")(go, *ws, x, w, b, K, it),
           getattr(C, name + "mapped_transposed_conv_forward")(xt, *ws, wt, bt, H, W, K, it),
           *getattr(C, name + "mapped_transposed_conv_backward")(got, *ws, xt, wt, bt, K, it)]
    for what, n, o in zip(("forward", "dInput", "dW", "dBias", "t forward", "t dInput", "t dW", "t dBias"), new, old):
        for which, f in (("NaN", torch.isnan), ("+inf", torch.isposinf), ("-inf", torch.isneginf)):
            assert torch.equal(f(n), f(o)), (what, which, int(f(n).sum()), int(f(o).sum()))


@pytest.mark.parametrize("case", CASES)
def test_one_pre_pass_for_all_gradients(case):
    """The combined backward, of a convolution and of a transposed one: the bits of the separate calls, one launch less; and none
    without the scratch for it."""
    from _gpu_impl import preferred_scratch
    from sphmap import capi
    B, ci, co, (H, W), (OH, OW), K, interp, P = case
    g = torch.Generator().manual_seed(ci)
    r = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    x, w, go, wt, xt, got = r(B, ci, H, W), r(co, ci, K), r(B, co, OH, OW), r(ci, co, K), r(B, ci, OH, OW), r(B, co, H, W)
    m = (torch.rand(*((OH, OW, K, P, 2) if P else (OH, OW, K, 2)), generator=g) * torch.tensor([W + 1.0, H + 1.0]) - 1.0).cuda()
    iw = torch.rand(OH, OW, K, P, generator=g).cuda() if P else None
    plan = capi.plan_build(m, iw, OH * OW, K, interp, H, W)

    def launches(fn):
        before = capi.lib.sph_launch_count()
        out = fn()
        return out, capi.lib.sph_launch_count() - before

    with preferred_scratch():
        ref, n = launches(lambda: [capi.conv_backward_input(go, plan, w, H, W, K), *capi.conv_backward_weight(go, x, m, K, interp, iw)])
        tref, tn = launches(lambda: [capi.tconv_backward_input(got, m, wt, K, interp, iw), *capi.tconv_backward_weight(got, xt, m, K, interp, iw)])
        new, nn = launches(lambda: capi.conv_backward_cl(go, None, x, None, plan, m, w, K, interp, iw, capi.EXACT))
    tnew, tnn = launches(lambda: capi.tconv_backward(got, xt, m, wt, K, interp, iw))
    assert all(torch.equal(a, b) for a, b in zip([*new, *tnew], [*ref, *tref]))
    assert nn == n - 1 and tnn == tn - 1
    for call in (lambda: capi.conv_backward_cl(go, None, x, None, plan, m, w, K, interp, iw, capi.EXACT),
                 lambda: capi.conv_backward_cl(go, go, x, None, plan, m, w, K, interp, iw, capi.EXACT),
                 lambda: capi.tconv_backward(got, xt, m, wt, K, interp, iw, ws=capi.conv_workspace(
                     capi.TCONV_BACKWARD, B, ci, co, OH, OW, H, W, K, P, capi.F32, interp, capi.EXACT, x))):
        with pytest.raises(capi.Unsupported):
            call()
    assert capi.device_status() == 0


@pytest.mark.parametrize("prec", [0, 1])
def test_phases_of_the_combined_backward(prec):
    """sph_trace_phases: the next combined call records its events, in order, whatever the precision; the list serves one call, also
    one that declines."""
    from sphmap import capi
    B, ci, co, H, W, K = 2, 32, 32, 16, 32, 9
    g = torch.Generator().manual_seed(3)
    r = lambda *s: torch.randn(*s, generator=g).cuda()  # noqa: E731
    x, w, go = r(B, ci, H, W), r(co, ci, K), r(B, co, H, W)
    m = (torch.rand(H, W, K, 2, generator=g) * torch.tensor([W - 1.0, H - 1.0])).cuda()
    plan = capi.plan_build(m, None, H * W, K, 1, H, W)
    ws = capi.conv_workspace(capi.CONV_BACKWARD, B, ci, co, H, W, H, W, K, 0, capi.F32, 1, prec, x, preferred=True)
    events, begin = ([torch.cuda.Event(enable_timing=True) for _ in range(n)] for n in (4, 1))

    def recorded(call):
        """Times of the events since the start of the call; negative: not recorded by it."""
        for e in events:
            e.record()
        torch.cuda._sleep(1000000)
        begin[0].record()
        call()
        torch.cuda.synchronize()
        return [begin[0].elapsed_time(e) for e in events]

    call = lambda: capi.conv_backward_cl(go, None, x, None, plan, m, w, K, 1, None, prec, ws=ws)  # noqa: E731
    recorded(call)
    capi.trace_phases(events)
    t = recorded(call)
    assert t[0] >= 0 and t == sorted(t) and t[3] > t[1], t
    assert max(recorded(call)) < 0
    capi.trace_phases(events)
    with pytest.raises(capi.Unsupported):
        capi.conv_backward_cl(go.double(), None, x.double(), None, plan, m.double(), w.double(), K, 1, None, capi.EXACT, ws=ws)
    assert max(recorded(call)) < 0
