"""Weight gradient from boxes of output rows and from plain rows against fp64 autograd: rows that do and do not fill a
k-block, output rows wider than one, row groups that end past the image, padding, one tap, several taps side by side and
tiles wider than a tap; every shape also through the im2col loads, which must agree."""
import pytest
import torch
import torch.nn.functional as F

from rembrandt_b200.ops import layout
from rembrandt_b200.ops import native_ops as K

pytestmark = pytest.mark.gpu
DEV = "cuda"

SHAPES = [  # N, C, Ko, H, W, k, pad
    (3, 32, 32, 8, 8, 3, 1), (2, 64, 64, 19, 19, 3, 1), (2, 128, 96, 7, 7, 3, 1), (1, 64, 160, 28, 28, 5, 2),
    (2, 96, 64, 13, 13, 3, 1), (1, 64, 64, 9, 70, 3, 1), (1, 32, 256, 5, 130, 3, 0), (2, 256, 128, 6, 6, 3, 0),
    (5, 64, 10, 16, 16, 1, 0), (3, 320, 136, 5, 5, 1, 0), (1, 16, 16, 64, 64, 3, 1), (2, 64, 64, 12, 12, 1, 1),
    (1, 64, 64, 1, 64, 3, 1), (4, 512, 512, 4, 4, 3, 1)]


@pytest.mark.parametrize("shape", SHAPES)
def test_boxes_against_autograd(shape):
    N, C, Ko, H, W, k, pad = shape
    g = torch.Generator(device=DEV).manual_seed(sum(shape))
    rnd = lambda *d: torch.randn(d, generator=g, device=DEV).bfloat16().float()
    Cp, Kp = K.pad_channels(C), K.pad_channels(Ko)
    P, Q = H + 2 * pad - k + 1, W + 2 * pad - k + 1
    x, dy = rnd(N, C, H, W), rnd(N, Ko, P, Q)
    w = torch.zeros(Ko, C, k, k, device=DEV, dtype=torch.float64, requires_grad=True)
    (want,) = torch.autograd.grad(F.conv2d(x.double(), w, padding=pad), w, dy.double())
    xi, dyi = layout.to_nhwc_padded(x, Cp), layout.to_nhwc_padded(dy, Kp)
    for box in (-1, 0, 1):
        dw = torch.ones((Ko, k * k, Cp), device=DEV)
        with K.gemm_options(force_box=box):
            K.conv_wgrad_tc(xi, N, H, W, Cp, dyi, Kp, Ko, k, k, 1, pad, pad, P, Q, dw)
        torch.cuda.synchronize()
        assert K.read_status() == 0
        got = layout.conv_weight_from_internal(dw - 1, C, k, k).double()
        # fp32 sums of N * P * Q products of N(0, 1) pairs: a few 1e-7 of the terms' root sum of squares, and the ones
        assert float((got - want).abs().max()) < 4e-6 * (N * P * Q) ** 0.5 * 4 + 2e-6, box
        assert bool((dw[:, :, C:] == 1).all())
