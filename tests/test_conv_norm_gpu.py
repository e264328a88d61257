"""A convolution with the normalisation by running statistics in its epilogue, against fp64: every form of the tensor-core
kernel, channel counts at and off the 32-column groups, with and without residual and ReLU, strides; and the kernel that works
scale and shift out."""
import pytest
import torch
import torch.nn.functional as F

from rembrandt_b200.ops import layout
from rembrandt_b200.ops import native_ops as K

pytestmark = pytest.mark.gpu
DEV = "cuda"
FORMS = [dict(), dict(force_halo=1), dict(force_halo=1, force_pair=1), dict(force_halo=0, force_pair=1),
         dict(force_halo=0, force_box=1), dict(force_halo=0, force_wide=1), dict(force_halo=0, force_tail=1),
         dict(force_halo=0, force_mt=2, force_resident=1)]
SHAPES = [(2, 32, 16, 9, 3, 1), (3, 64, 64, 13, 3, 1), (40, 32, 50, 13, 3, 1), (3, 96, 200, 7, 3, 1), (2, 64, 320, 12, 3, 1),
          (4, 64, 256, 10, 1, 1), (3, 64, 128, 14, 3, 2), (2, 32, 64, 15, 1, 2), (1, 32, 33, 1, 1, 1)]


@pytest.mark.parametrize("options", FORMS)
@pytest.mark.parametrize("residual,relu", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("shape", SHAPES)
def test_normalised_convolution(shape, residual, relu, options):
    N, C, Ko, H, k, s = shape
    torch.manual_seed(sum(shape))
    pad, Kp = k // 2, K.pad_channels(Ko)
    P = (H + 2 * pad - k) // s + 1
    x = torch.randn(N, C, H, H, device=DEV).bfloat16().float()
    w = (torch.randn(Ko, C, k, k, device=DEV) / (C * k * k) ** 0.5).bfloat16().float()
    scale, shift = torch.randn(Kp, device=DEV), torch.randn(Kp, device=DEV)
    res = torch.randn(N, P, P, Kp, device=DEV).bfloat16() if residual else None
    y = torch.full((N, P, P, Kp), float("nan"), device=DEV, dtype=torch.bfloat16)
    with K.gemm_options(**options):
        K.conv_fprop_norm(layout.to_nhwc_padded(x, C), N, H, H, C, layout.conv_weight_to_internal(w, C).bfloat16(), Ko, k, k, s,
                          pad, pad, P, P, y, Kp, scale, shift, res, relu, n_valid=Ko, n_store=Kp)
    ref = F.conv2d(x.double(), w.double(), stride=s, padding=pad).permute(0, 2, 3, 1) * scale[:Ko] + shift[:Ko]
    ref = ref + res[..., :Ko].double() if residual else ref
    ref = ref.relu() if relu else ref
    assert K.read_status() == 0
    # operands are exact in bf16, sums are fp32: the rounding of the result, and the order of the additions of terms of size 1
    assert ((y[..., :Ko].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 2e-4).all()
    assert (y[..., Ko:].float() == 0).all()


def test_scale_and_shift_from_running_statistics():
    sizes = [(32, 16), (64, 64), (320, 300)]
    params = torch.rand(4096, device=DEV) + 0.1
    rows, at, out, offset = [], 0, [], 0
    for C, valid in sizes:
        offs = [offset + i * C for i in range(4)]
        offset += 4 * C
        eps = 1e-5 * (len(rows) + 1)
        rows.append([*offs, at, C, valid, int(torch.tensor([eps]).view(torch.int32))])
        g, b, m, v = (params[o: o + valid].double() for o in offs)
        sc = g * (v + eps).rsqrt()
        zeros = torch.zeros(C - valid, device=DEV, dtype=torch.float64)
        out += [sc, zeros, b - m * sc, zeros]
        at += 2 * C
    got = torch.full((at,), float("nan"), device=DEV)
    K.bn_fold(params, torch.tensor(rows, device=DEV), len(rows), got)
    want = torch.cat(out)
    # two roundings of fp32 and a cancellation of terms of size 3
    assert ((got.double() - want).abs() <= 4e-7 * 3).all()
