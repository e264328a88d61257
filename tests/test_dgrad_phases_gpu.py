"""The output phases of a strided data-gradient in one launch, against fp64 autograd: more work items than SMs, several column
tiles, images of odd size (phases of different extents), rows that end inside a tile, a stride with more phases than a launch
takes, both forms of the filters; and the form that adds onto a gradient that is masked already."""
import pytest
import torch
import torch.nn.functional as F

from rembrandt_b200.ops import layout
from rembrandt_b200.ops import native_ops as K
from rembrandt_b200.ops.conv_grad import conv_dgrad

pytestmark = pytest.mark.gpu
DEV = "cuda"

SHAPES = [  # N, C, Ko, H, W, k, stride, pad
    (16, 64, 128, 64, 64, 3, 2, 1), (5, 320, 64, 23, 17, 3, 2, 1), (3, 32, 16, 37, 64, 5, 2, 2), (2, 512, 96, 9, 31, 3, 2, 1),
    (1, 64, 64, 3, 2, 3, 2, 1), (4, 96, 64, 15, 15, 4, 2, 1), (2, 64, 32, 13, 19, 4, 3, 1), (3, 128, 64, 11, 11, 2, 2, 0)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("how", ["default", "measured", "two sub-tiles", "onto"])
def test_against_autograd(shape, packed, how):
    N, C, Ko, H, W, k, s, p = shape
    g = torch.Generator(device=DEV).manual_seed(sum(shape))
    rnd = lambda *d: torch.randn(d, generator=g, device=DEV).bfloat16().float()
    Cp, Kp = K.pad_channels(C), K.pad_channels(Ko)
    P, Q = (H + 2 * p - k) // s + 1, (W + 2 * p - k) // s + 1
    w, dy, below = rnd(Ko, C, k, k), rnd(N, Ko, P, Q), rnd(N, C, H, W).relu()
    x = torch.zeros(N, C, H, W, device=DEV, requires_grad=True)
    (want,) = torch.autograd.grad(F.conv2d(x.double(), w.double(), stride=s, padding=p), x, dy.double())
    wi, wt = layout.conv_weight_to_internal(w, Cp).bfloat16(), None
    if packed:
        wt = torch.full((Cp, k * k, Kp), float("nan"), device=DEV, dtype=torch.bfloat16)
        K.pack_dgrad_filters(wi, wt, Ko, Kp, k * k, Cp)
    dyi, mask = layout.to_nhwc_padded(dy, Kp), layout.to_nhwc_padded(below, Cp)
    run = lambda out, **kw: conv_dgrad(dyi, N, P, Q, Kp, wi, Ko, Cp, C, k, s, p, H, W, out, mask=mask, wt=wt, **kw)
    want = want.double()
    if how == "onto":
        before = rnd(N, C, H, W) * (below > 0)
        dx = layout.to_nhwc_padded(before, Cp)
        run(dx, add=dx, add_masked=True)
        want = want + before.double()
    else:
        dx = torch.full((N, H, W, Cp), float("nan"), device=DEV, dtype=torch.bfloat16)
        if how == "measured":
            K.gemm_clear_plans()
            with K.gemm_tuning():
                run(torch.zeros_like(dx))
        with K.gemm_options(**({"force_mt": 2} if how == "two sub-tiles" else {})):
            run(dx)
    torch.cuda.synchronize()
    assert K.read_status() == 0
    want = want * (below > 0)
    got = layout.from_nhwc_padded(dx, C).double()
    # fp32 sums of up to taps * Ko products of N(0, 1) pairs, rounded once to bf16
    err = (got - want).abs() - want.abs() * 2 ** -8
    assert float(err.max()) < 1e-3 * (1 + (k * k * Ko) ** 0.5)
    assert Cp == C or bool((dx[..., C:] == 0).all())
