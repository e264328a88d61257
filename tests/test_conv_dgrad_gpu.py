"""The data-gradient that reads the filters in place or from their packed copy, and scatters the phases of a strided one,
against fp64 autograd:
channel counts below, at and off the 64-wide blocks of the operand, tiles wider than 256 columns, one and several taps,
strides 1 to 3, images wider than high and the other way round, an addend (its own tensor, or dx itself) with and without the
producer's mask, every plan option, measured plans."""
import pytest
import torch
import torch.nn.functional as F

from rembrandt_b200.ops import layout
from rembrandt_b200.ops import native_ops as K
from rembrandt_b200.ops.conv_grad import conv_dgrad

pytestmark = pytest.mark.gpu
DEV = "cuda"

SHAPES = [  # N, C, Ko, H, k, stride, pad
    (2, 16, 16, 8, 3, 1, 1), (2, 64, 64, 14, 3, 1, 1), (3, 96, 40, 9, 5, 1, 2), (2, 256, 96, 13, 3, 1, 1),
    (1, 384, 64, 7, 3, 1, 1), (2, 512, 320, 6, 1, 1, 0), (1, 3, 64, 30, 3, 1, 1), (5, 128, 128, 19, 3, 1, 1),
    (2, 64, 128, 14, 3, 2, 1), (2, 32, 64, 15, 3, 2, 1), (3, 64, 128, 14, 1, 2, 0), (2, 96, 48, 13, 1, 2, 0),
    (1, 128, 256, 8, 5, 3, 2), (2, 48, 64, 11, 2, 2, 0), (33, 32, 16, 8, 3, 2, 1)]


OBLONG = [  # ... and W
    (2, 64, 64, 14, 3, 1, 1, 9), (3, 32, 48, 6, 3, 1, 1, 40), (2, 64, 128, 14, 3, 2, 1, 21), (2, 32, 64, 15, 3, 2, 1, 6),
    (3, 64, 128, 13, 1, 2, 0, 30), (1, 128, 256, 8, 5, 3, 2, 17), (2, 48, 64, 11, 2, 2, 0, 8), (37, 64, 32, 73, 3, 2, 1, 19)]


def _run(shape, add, masked, packed=False, tuned=False, **options):
    N, C, Ko, H, k, s, p = shape[:7]
    W = shape[7] if len(shape) > 7 else H
    g = torch.Generator(device=DEV).manual_seed(sum(shape))
    rnd = lambda *d: torch.randn(d, generator=g, device=DEV).bfloat16().float()
    Cp, Kp = K.pad_channels(C), K.pad_channels(Ko)
    P, Q = (H + 2 * p - k) // s + 1, (W + 2 * p - k) // s + 1
    w, dy, extra, below = rnd(Ko, C, k, k), rnd(N, Ko, P, Q), rnd(N, C, H, W), rnd(N, C, H, W).relu()
    x = torch.zeros(N, C, H, W, device=DEV, requires_grad=True)
    (want,) = torch.autograd.grad(F.conv2d(x.double(), w.double(), stride=s, padding=p), x, dy.double())
    want = want.double()
    want = (want + extra.double() if add else want) * (below > 0 if masked else 1)
    dx = torch.full((N, H, W, Cp), float("nan"), device=DEV, dtype=torch.bfloat16)
    src = None
    if add == "own":
        src = layout.to_nhwc_padded(extra, Cp)
    elif add == "dx":
        dx = src = layout.to_nhwc_padded(extra, Cp)
    wi, wt = layout.conv_weight_to_internal(w, Cp).bfloat16(), None
    if packed:
        wt = torch.full((Cp, k * k, Kp), float("nan"), device=DEV, dtype=torch.bfloat16)
        K.pack_dgrad_filters(wi, wt, Ko, Kp, k * k, Cp)
    run = lambda out, addend: conv_dgrad(layout.to_nhwc_padded(dy, Kp), N, P, Q, Kp, wi, Ko, Cp, C, k, s, p, H, W, out,
                                         add=addend, mask=layout.to_nhwc_padded(below, Cp) if masked else None, wt=wt)
    if tuned:                                    # every plan is run several times: not on what is compared
        with K.gemm_tuning():
            run(torch.zeros_like(dx), None if src is None else src.clone())
    with K.gemm_options(**options):
        run(dx, src)
    torch.cuda.synchronize()
    assert K.read_status() == 0
    got = layout.from_nhwc_padded(dx, C).double()
    # fp32 sums of up to taps * Ko products of N(0, 1) pairs, rounded once to bf16
    err = (got - want).abs() - want.abs() * 2 ** -8
    assert float(err.max()) < 1e-3 * (1 + (k * k * Ko) ** 0.5)
    assert Cp == C or bool((dx[..., C:] == 0).all())


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("add,masked", [(None, False), (None, True), ("own", True), ("dx", False), ("dx", True)])
@pytest.mark.parametrize("packed", [False, True])
def test_against_autograd(shape, add, masked, packed):
    _run(shape, add, masked, packed)


@pytest.mark.parametrize("shape", OBLONG)
@pytest.mark.parametrize("add,masked", [(None, True), ("own", True), ("dx", True)])
@pytest.mark.parametrize("packed,tuned", [(False, False), (True, False), (False, True), (True, True)])
def test_oblong_images_and_measured_plans(shape, add, masked, packed, tuned):
    _run(shape, add, masked, packed, tuned)


@pytest.mark.parametrize("shape", [(2, 32, 48, 9, 1, 2, 2, 12), (3, 64, 32, 11, 3, 3, 4)])
@pytest.mark.parametrize("masked", [False, True])
def test_phases_of_negative_padding_run_on_cuda_cores(shape, masked):
    _run(shape, None, masked)


@pytest.mark.parametrize("shape", [SHAPES[1], SHAPES[4], SHAPES[7], SHAPES[8], SHAPES[9]])
@pytest.mark.parametrize("options", [dict(force_mt=2), dict(force_resident=1), dict(force_box=1), dict(force_wide=1),
                                     dict(force_pair=1), dict(force_tail=1), dict(deterministic=1)])
def test_plans(shape, options):
    _run(shape, "own", True, **options)


@pytest.mark.parametrize("shape,searched", [((32, 8, 8, 32, 32, 32, 32, 3, 1, 1, 8, 8), False),
                                            ((32, 64, 64, 256, 256, 256, 256, 3, 1, 1, 64, 64), True)])
def test_the_copy_is_measured_only_where_it_can_win(monkeypatch, shape, searched):
    from rembrandt_b200.ops import conv_grad
    seen, real = [], conv_grad.conv_dgrad
    monkeypatch.setattr(conv_grad, "conv_dgrad", lambda *a, **k: (seen.append(k.get("wt") is not None), real(*a, **k)))
    monkeypatch.setattr(conv_grad, "_measured", {})
    plan = conv_grad.DgradPlan(*shape, [(False, True), (True, True)])
    torch.cuda.synchronize()
    assert K.read_status() == 0 and any(seen) == searched
    assert searched or plan.wt is None
