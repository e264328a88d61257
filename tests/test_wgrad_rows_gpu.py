"""Weight-gradients from whole rows against fp64 autograd: every plan that the model ranks (rows one by one and in a run, one or all
filter rows per item, one or more channel blocks), channel blocks of 32 and 64 that are and are not full, one and two blocks of
output channels, rows that are and are not multiples of 16 positions, chunks of several images and of part of one, images wider
than high, filters of 2 to 8 taps a row, paddings from none to the filter's width; values that must not be added into (channels of
the padding); and what is remembered of a measurement."""
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


@pytest.mark.parametrize("shape", [SHAPES[0], SHAPES[1], SHAPES[12]])
def test_what_was_measured_is_what_runs(shape):
    args, check = _case(shape)
    run = lambda a, dw: K.conv_wgrad_tc(*a, dw)
    K.gemm_clear_plans()
    check(run)
    assert K.gemm_last_launch()["a_mode"] != ROWS      # not measured: the general kernel
    N, H, W, Cp, _, Kp, Ko, k = args[1:9]
    K._tuned_convs.clear()
    K.tune_wgrad(N, H, W, Cp, Ko, Kp, k, k, 1, *args[11:])
    check(run)
    first = K.gemm_last_launch()
    check(run)
    assert K.gemm_last_launch() == first
    with K.gemm_options(deterministic=1):
        check(run)
        assert K.gemm_last_launch()["a_mode"] != ROWS
    K.gemm_clear_plans()
