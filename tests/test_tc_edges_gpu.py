"""bf16 tensor-core convolutions at the edges of their weight images (4 rows x 64 channels x 9 slots per block), of the
weight gradient's 128-row blocks and column groups, and of the plan tables (four and eight entries of a key), against the
CPU oracle; and the extra pixels of a channels-last copy that starts uninitialised."""
import pytest
import torch

from oracle import port
from test_tc_gpu import _case, _close

pytestmark = pytest.mark.gpu

CASES = [
    # seed, B, Cin, Cout, IH, IW, OH, OW, K, interp, P, gnomonic
    (21, 1, 64, 1, 9, 17, 9, 17, 1, 1, 0, False),       # one slot, one row
    (22, 2, 65, 136, 9, 17, 11, 19, 10, 1, 0, False),   # padded channels, a second slot group of one, a row block of 8
    (23, 1, 128, 200, 8, 16, 8, 16, 19, 0, 0, False),   # three slot groups, a row block of 72
    (24, 1, 64, 64, 8, 12, 12, 16, 9, 0, 3, False),     # three weighted points; six entries per key on average
    (25, 2, 72, 24, 12, 20, 17, 33, 9, 0, 1, False),    # one weighted point
    (26, 1, 64, 320, 16, 32, 16, 32, 4, 1, 0, False),   # three row blocks, the last of 64 rows
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "s%d" % c[0])
def test_edges(case):
    from _gpu_impl import CApi
    from sphmap import capi
    seed, B, Cin, Cout, IH, IW, OH, OW, K, interp, P, gn = case
    x, w, b, m, iw, go = _case(seed, B, Cin, Cout, IH, IW, OH, OW, K, interp, P, gn)
    tc = CApi(precision=1)
    _close(tc.mapped_conv_forward(x, m, w, b, K, interp, iw), port.mapped_conv_forward(x, m, w, b, K, interp, iw), "forward")
    got, want = tc.mapped_conv_backward(go, m, x, w, b, K, interp, iw), port.mapped_conv_backward(go, m, x, w, b, K, interp, iw)
    dev = lambda t: None if t is None else t.cuda()  # noqa: E731
    plan = capi.plan_build(dev(m), dev(iw), OH * OW, K, interp, IH, IW)
    for name, a, ref in zip(("grad_input", "grad_weight", "grad_bias"), got, want):
        _close(a, ref, name)
    if K <= 10:     # (more slots than a plan table holds: the separate calls only)
        both = capi.conv_backward_cl(dev(go), None, dev(x), None, plan, dev(m), dev(w), K, interp, dev(iw), capi.BF16)
        for name, a, ref in zip(("grad_input", "grad_weight", "grad_bias"), both, want):
            _close(a.cpu(), ref, name + " (combined)")
    assert capi.device_status() == 0


@pytest.mark.parametrize("cin,cout,width", [(3, 64, 32), (64, 64, 32), (3, 64, 31), (3, 8, 32), (1, 128, 33)])
def test_extra_pixels_of_an_uninitialised_copy(cin, cout, width):
    """The tensor-core kernels' pre-passes clear them, thin layers of ragged rows or few channels write them themselves."""
    from sphmap import capi
    x, w, b, m, _, _ = _case(31, 3, cin, cout, 16, width, 16, width, 9, 1)
    cl = capi.companion(3, cout, 16, width, "cuda").fill_(255)
    out = capi.conv_forward_cl(x.cuda(), None, m.cuda(), w.cuda(), b.cuda(), 9, 1, None, capi.BF16, True, out_cl=cl)
    copy = cl.view(torch.bfloat16)[:3 * (16 * width + 1) * cout].view(3, 16 * width + 1, cout)
    assert not copy[:, -1].any()
    assert torch.equal(copy[:, :-1].transpose(1, 2).reshape(3, cout, 16, width), out.bfloat16())


@pytest.mark.parametrize("cin,cout,h,w,P", [(20, 40, 140, 141, 4), (64, 96, 149, 128, 3)])
def test_weighted_input_gradient_sums_in_float32(cin, cout, h, w, P):
    """Over a weighted map as over others, the products of the output channels are summed in float32 and nothing between them and the
    result is rounded to fewer bits: whole numbers whose operands are exact in bf16 come out exact, with either scratch."""
    from sphmap import capi
    g = torch.Generator().manual_seed(41)
    whole = lambda *shape: torch.randint(-7, 8, shape, generator=g).float()  # noqa: E731
    K = 2
    x, wgt, go = whole(1, cin, h, w), whole(cout, cin, K), whole(1, cout, h, w)
    m = torch.rand(h, w, K, P, 2, generator=g) * torch.tensor([w - 1.0, h - 1.0])
    iw = torch.zeros(h, w, K, P)
    iw[..., 0] = 1.0
    want = port.mapped_conv_backward(go, m, x, wgt, torch.zeros(cout), K, 0, iw)
    assert want[0].abs().max() > 1024     # (a bf16 holds every whole number up to 256)
    x, wgt, m, iw, go = [t.cuda() for t in (x, wgt, m, iw, go)]
    plan = capi.plan_build(m, iw, h * w, K, 0, h, w)
    for preferred in (False, True):
        ws = capi.conv_workspace(capi.CONV_BACKWARD, 1, cin, cout, h, w, h, w, K, P, capi.F32, 0, capi.BF16, x, preferred=preferred)
        got = capi.conv_backward_cl(go, None, x, None, plan, m, wgt, K, 0, iw, capi.BF16, ws=ws)
        for a, ref in zip(got, want):
            assert torch.equal(a.cpu(), ref)
    assert capi.device_status() == 0
