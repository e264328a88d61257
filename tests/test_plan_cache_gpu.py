"""Measured plans where two launches differ only in how the same number of rows is laid out: the phases (0, 1) and (1, 0) of
a strided data-gradient at odd sizes (rows and columns exchanged, one side of 128 each in the last two), and launches that
follow a measurement with other options or a workspace that its plan does not fit. Against fp64 autograd."""
import pytest
import torch
import torch.nn.functional as F

from rembrandt_b200 import _native
from rembrandt_b200.ops import layout
from rembrandt_b200.ops import native_ops as K
from rembrandt_b200.ops.conv_grad import conv_dgrad

pytestmark = pytest.mark.gpu


def _operands(N, C, Ko, H, k, s, p):
    g = torch.Generator(device="cuda").manual_seed(N + H)
    rnd = lambda *d: torch.randn(d, generator=g, device="cuda").bfloat16().float()
    P = (H + 2 * p - k) // s + 1
    w, dy = rnd(Ko, C, k, k), rnd(N, Ko, P, P)
    x = torch.zeros(N, C, H, H, device="cuda", dtype=torch.float64, requires_grad=True)
    (want,) = torch.autograd.grad(F.conv2d(x, w.double(), stride=s, padding=p), x, dy.double())
    Cp, Kp = K.pad_channels(C), K.pad_channels(Ko)
    return P, Cp, Kp, layout.conv_weight_to_internal(w, Cp).bfloat16(), layout.to_nhwc_padded(dy, Kp), want


def _check(dx, want, C, terms):
    got = layout.from_nhwc_padded(dx, C).double()
    # fp32 sums of `terms` products of N(0, 1) pairs, rounded once to bf16
    assert float(((got - want).abs() - want.abs() * 2 ** -8).max()) < 1e-3 * (1 + terms ** 0.5)


@pytest.mark.parametrize("N,C,Ko,H,k,s,p", [(37, 32, 32, 73, 3, 2, 1), (37, 64, 64, 73, 3, 2, 1), (2, 32, 32, 257, 3, 2, 1),
                                            (1, 288, 32, 257, 3, 2, 1)])
def test_measured_plans_of_the_phases(N, C, Ko, H, k, s, p):
    P, Cp, Kp, w, dy, want = _operands(N, C, Ko, H, k, s, p)
    dx = torch.full((N, H, H, Cp), float("nan"), device="cuda", dtype=torch.bfloat16)
    run = lambda: conv_dgrad(dy, N, P, P, Kp, w, Ko, Cp, C, k, s, p, H, H, dx)
    K.gemm_clear_plans()
    with K.gemm_tuning():
        run()
    dx.fill_(float("nan"))
    run()
    torch.cuda.synchronize()
    assert K.read_status() == 0
    _check(dx, want, C, k * k * Ko)
    for options in (dict(force_box=0), dict(force_wide=0), dict(deterministic=1)):   # what was measured may not apply any more
        with K.gemm_options(**options):
            dx.fill_(float("nan"))
            run()
        torch.cuda.synchronize()
        assert K.read_status() == 0
        _check(dx, want, C, k * k * Ko)
    K.gemm_clear_plans()


def test_a_workspace_smaller_than_at_the_measurement():
    """7 x 7 images in few items: the plan that is measured cuts them along the reduction, in 8 MB of workspace; a launch
    with less workspace takes another plan."""
    N, C, Ko, H, k = 4, 512, 512, 7, 3
    P, Cp, Kp, w, dy, want = _operands(N, C, Ko, H, k, 1, 1)
    dx = torch.empty((N, H, H, Cp), device="cuda", dtype=torch.bfloat16)
    ws = torch.zeros(1 << 21, device="cuda")
    call = lambda nbytes: _native.cuda().rb_conv_dgrad_tc(
        dy.data_ptr(), N, P, P, Kp, w.data_ptr(), None, Ko, Cp, C, k, k, 1, 1, 1, H, H, dx.data_ptr(), None, None, ws.data_ptr(),
        nbytes, K.status_word().data_ptr(), _native.stream_handle())
    K.gemm_clear_plans()
    with K.gemm_tuning():
        assert call(ws.numel() * 4) == 0
    for nbytes in (ws.numel() * 4, 1 << 16, 0):
        dx.fill_(float("nan"))
        assert call(nbytes) == 0
        torch.cuda.synchronize()
        _check(dx, want, C, k * k * Ko)
    assert K.read_status() == 0
    K.gemm_clear_plans()
