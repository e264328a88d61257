"""Weight-gradients from whole rows against fp64 autograd: every plan that the model ranks (rows one by one and in a run, one or all
filter rows per item, one or more channel blocks), channel blocks of 32 and 64 that are and are not full, one and two blocks of
output channels, rows that are and are not multiples of 16 positions, chunks of several images and of part of one, images wider
than high, filters of 2 to 8 taps a row, paddings from none to the filter's width; values that must not be added into (channels of
the padding); and what is
remembered of a measurement."""
import pytest
import torch
import torch.nn.functional as F

from rembrandt_b200.ops import layout
from rembrandt_b200.ops import native_ops as K

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROWS = 6      # how gemm_last_launch names this kernel

SHAPES = [  # N, C, Ko, H, W, k, pad
    (3, 32, 32, 8, 8, 3, 1), (2, 64, 64, 19, 19, 3, 1), (2, 128, 96, 7, 7, 3, 1), (1, 64, 160, 28, 28, 5, 2),
    (2, 96, 64, 13, 13, 3, 1), (1, 64, 64, 9, 70, 3, 1), (1, 32, 256, 5, 130, 3, 0), (2, 256, 128, 6, 6, 3, 0),
    (1, 16, 16, 64, 64, 3, 1), (1, 64, 64, 1, 64, 3, 1), (4, 512, 512, 4, 4, 3, 1), (5, 128, 128, 16, 16, 3, 1),
    (3, 96, 256, 27, 27, 5, 2), (2, 64, 128, 20, 33, 7, 3), (3, 64, 64, 10, 10, 2, 0), (2, 64, 64, 9, 9, 4, 1),
    (7, 64, 64, 13, 13, 2, 1), (1, 160, 200, 11, 5, 3, 2), (40, 128, 128, 19, 19, 3, 1), (33, 32, 48, 16, 16, 5, 2),
    (2, 32, 32, 12, 12, 8, 4), (1, 64, 64, 3, 240, 3, 1), (9, 64, 10, 5, 6, 3, 1)]


def _case(shape):
    N, C, Ko, H, W, k, pad = shape
    g = torch.Generator(device=DEV).manual_seed(sum(shape))
    rnd = lambda *d: torch.randn(d, generator=g, device=DEV).bfloat16().float()
    Cp, Kp = K.pad_channels(C), K.pad_channels(Ko)
    P, Q = H + 2 * pad - k + 1, W + 2 * pad - k + 1
    x, dy = rnd(N, C, H, W), rnd(N, Ko, P, Q)
    w = torch.zeros(Ko, C, k, k, device=DEV, dtype=torch.float64, requires_grad=True)
    (want,) = torch.autograd.grad(F.conv2d(x.double(), w, padding=pad), w, dy.double())
    args = (layout.to_nhwc_padded(x, Cp), N, H, W, Cp, layout.to_nhwc_padded(dy, Kp), Kp, Ko, k, k, 1, pad, pad, P, Q)

    def check(run):
        dw = torch.ones((Ko, k * k, Cp), device=DEV)
        run(args, dw)
        torch.cuda.synchronize()
        assert K.read_status() == 0
        got = layout.conv_weight_from_internal(dw - 1, C, k, k).double()
        # fp32 sums of N * P * Q products of N(0, 1) pairs: a few 1e-7 of the terms' root sum of squares, and the ones
        assert float((got - want).abs().max()) < 4e-6 * (N * P * Q) ** 0.5 * 4 + 2e-6
        assert bool((dw[:, :, C:] == 1).all())
    return args, check


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("beside", [False, True])
def test_every_plan_against_autograd(shape, beside):
    args, check = _case(shape)
    seen = set()
    for nth in range(1, 9):      # the first, second ... plan by the model
        with K.gemm_options(force_rows=nth):
            check(lambda a, dw: K.conv_wgrad_tc(*a, dw, beside=beside))
        plan = tuple(K.gemm_last_launch().values())
        assert plan[6] == ROWS
        seen.add(plan)
    assert len(seen) > 1


ODD = [  # N, C, Ko, H, W, R, S, pad_h, pad_w, more rows and columns of the output, more channels per row of dy
    (3, 64, 96, 9, 13, 1, 5, 0, 2, 0, 0, 0), (2, 32, 64, 13, 9, 5, 1, 2, 0, 0, 0, 64), (2, 64, 64, 8, 10, 3, 2, 1, 0, 0, 1, 0),
    (2, 96, 32, 7, 11, 2, 3, 0, 2, 1, -1, 32), (3, 64, 160, 10, 10, 3, 3, 1, 1, -3, -2, 0), (2, 128, 64, 6, 17, 3, 3, 4, 3, 0, 0, 0),
    (2, 64, 64, 11, 6, 4, 3, 0, 1, 2, 2, 0), (1, 32, 32, 3, 3, 3, 3, 0, 0, 0, 0, 0)]


@pytest.mark.parametrize("shape", ODD)
def test_unequal_sides_and_outputs_cut_or_grown(shape):
    N, C, Ko, H, W, R, S, ph, pw, dh, dw_, more = shape
    torch.manual_seed(sum(shape))
    P, Q, ld = H + 2 * ph - R + 1 + dh, W + 2 * pw - S + 1 + dw_, K.pad_channels(Ko) + more
    x, dy = (torch.randn(N, C, H, W, device=DEV).bfloat16().float(), torch.randn(N, Ko, P, Q, device=DEV).bfloat16().float())
    w = torch.zeros(Ko, C, R, S, device=DEV, dtype=torch.float64, requires_grad=True)
    y = F.conv2d(F.pad(x.double(), (pw, pw + max(dw_, 0), ph, ph + max(dh, 0))), w)[:, :, :P, :Q]
    (want,) = torch.autograd.grad(y, w, dy.double())
    rows = torch.full((N, P, Q, ld), float("nan"), device=DEV, dtype=torch.bfloat16)      # what lies behind Ko is not read
    rows[..., :Ko] = dy.permute(0, 2, 3, 1)
    xh = layout.to_nhwc_padded(x, C)
    for beside in (False, True):
        for nth in range(1, 9):
            out = torch.zeros((Ko, R * S, C), device=DEV)
            with K.gemm_options(force_rows=nth):
                K.conv_wgrad_tc(xh, N, H, W, C, rows, ld, Ko, R, S, 1, ph, pw, P, Q, out, beside=beside)
            assert K.read_status() == 0 and (K.gemm_last_launch()["a_mode"] == ROWS) == (R > 1)      # no plans for one row of taps
            got = out.view(Ko, R, S, C).permute(0, 3, 1, 2).double()
            assert float((got - want).abs().max()) < 4e-6 * (N * P * Q) ** 0.5 * 4 + 2e-6      # as above


BORDERS = [  # N, C, Ko, H, W, R, S, pad_h, pad_w
    (2, 32, 32, 8, 8, 3, 3, 1, 1), (2, 64, 32, 11, 11, 3, 3, 1, 1), (1, 32, 64, 5, 20, 3, 3, 0, 0), (3, 32, 32, 7, 6, 5, 5, 2, 2),
    (1, 32, 32, 12, 16, 3, 3, 1, 1), (2, 32, 32, 9, 7, 2, 4, 0, 3), (1, 32, 160, 7, 7, 3, 3, 2, 2), (17, 32, 32, 3, 3, 3, 3, 1, 1)]


@pytest.mark.parametrize("shape", BORDERS)
def test_infinities_and_nan_meet_what_they_belong_to(shape):
    """A pixel at the border has no part in the taps that would put it against an output outside the image; pixels outside count as
    zeros. So every sum is what the same products give in another order: as finite, as infinite, as much a NaN."""
    N, C, Ko, H, W, R, S, ph, pw = shape
    torch.manual_seed(sum(shape))
    P, Q = H + 2 * ph - R + 1, W + 2 * pw - S + 1
    x, dy = (torch.randn(N, c, *hw).bfloat16().double() for c, hw in ((C, (H, W)), (Ko, (P, Q))))
    inf, nan = float("inf"), float("nan")
    for c, (n, h, w, v) in enumerate([(0, 0, 0, inf), (0, 0, -1, -inf), (-1, -1, 0, nan), (-1, -1, -1, inf), (0, H // 2, -1, nan),
                                      (-1, -1, W // 2, inf), (0, H // 2, W // 2, -inf), (-1, H // 2, 0, inf), (-1, 0, W // 2, nan)]):
        x[n, c, h, w] = v
    for k, (n, h, w, v) in enumerate([(0, 0, 0, inf), (-1, -1, -1, nan), (0, P // 2, Q // 2, -inf), (-1, P // 2, -1, inf)]):
        dy[n, k, h, w] = v
    dy[0, 4] = 0.0      # an infinite pixel against zeros inside the image
    padded = F.pad(x, (pw, pw, ph, ph))
    want = torch.stack([(dy[:, :, None] * padded[:, None, :, r: r + P, s: s + Q]).sum((0, 3, 4)) for r in range(R) for s in range(S)], 1)
    assert int(want.isfinite().sum()) > want.numel() // 2      # [Ko][taps][C]
    xi, dyi = (t.permute(0, 2, 3, 1).contiguous().bfloat16().to(DEV) for t in (x, dy))
    for beside in (False, True):
        for nth in range(1, 9):
            out = torch.zeros((Ko, R * S, C), device=DEV)
            with K.gemm_options(force_rows=nth):
                K.conv_wgrad_tc(xi, N, H, W, C, dyi, Ko, Ko, R, S, 1, ph, pw, P, Q, out, beside=beside)
            assert K.read_status() == 0 and K.gemm_last_launch()["a_mode"] == ROWS
            got, plan = out.double().cpu(), K.gemm_last_launch()
            assert torch.equal(got.isnan(), want.isnan()), (plan, (got.isnan() != want.isnan()).nonzero()[:9])
            assert torch.equal(got == inf, want == inf) and torch.equal(got == -inf, want == -inf), plan
            fine = want.isfinite()
            assert float((got - want)[fine].abs().max()) < 4e-6 * (N * P * Q) ** 0.5 * 4      # as above


# (row plans take three quarters of the general kernel's time here: which is kept does not hang on a percent)
@pytest.mark.parametrize("shape", [(32, 32, 32, 16, 16, 5, 2), (64, 32, 64, 12, 12, 5, 2)])
def test_what_was_measured_is_what_runs(shape):
    args, check = _case(shape)

    def runs_rows(beside):
        check(lambda a, dw: K.conv_wgrad_tc(*a, dw, beside=beside))
        return K.gemm_last_launch()["a_mode"] == ROWS

    N, H, W, Cp, _, Kp, Ko, k = args[1:9]
    tune = lambda *beside: K.tune_wgrad(N, H, W, Cp, Ko, Kp, k, k, 1, *args[11:], beside=beside)
    K.gemm_clear_plans()
    assert not runs_rows(False) and not runs_rows(True)      # not measured: the general kernel
    with K.gemm_options(autotune=0):
        tune(False, True)
    assert not runs_rows(False) and not runs_rows(True)      # nor with measuring switched off
    for first in (False, True):
        tune(first)
        assert runs_rows(first) and not runs_rows(not first)      # each form by itself
        launch = (runs_rows(first), K.gemm_last_launch())
        assert (runs_rows(first), K.gemm_last_launch()) == launch
        with K.gemm_options(deterministic=1):
            K.conv_wgrad_tc(*args, torch.zeros((Ko, k * k, Cp), device=DEV), beside=first)
            assert K.gemm_last_launch()["a_mode"] != ROWS
        tune(False, True)
        assert runs_rows(False) and runs_rows(True)
        K.gemm_clear_plans()
        assert not runs_rows(first)      # forgotten, and measured again when asked for
