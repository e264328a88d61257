"""Column groups of which only a part exists: the epilogue of the tensor-core kernel writes the padding as zeros, whatever the
filters and the bias hold there, with every combination of bias, ReLU, mask and addend."""
import pytest
import torch
import torch.nn.functional as F

from rembrandt_b200.ops import layout
from rembrandt_b200.ops import native_ops as K
from rembrandt_b200.ops.conv_grad import conv_dgrad

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _close(got, ref):
    # operands are exact in bf16, sums are fp32: what is left is the rounding of the result (half of 2^-8 of its size) and the
    # order of 1e3 fp32 additions of terms of size 1 / sqrt(1e3)
    assert ((got.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()


@pytest.mark.parametrize("bias,relu,mask", [(False, False, False), (True, True, False), (True, False, True), (False, True, True)])
@pytest.mark.parametrize("ko", [1, 15, 16, 17, 31, 33, 50, 63, 95])
def test_forward_columns(ko, bias, relu, mask):
    torch.manual_seed(ko)
    n, c, h = 2, 32, 7
    kp = K.pad_channels(ko)
    x = torch.randn(n, c, h, h, device=DEV).bfloat16().float()
    w = (torch.randn(ko, c, 3, 3, device=DEV) / 17).bfloat16().float()
    # filters for the padded columns are not zero here
    wi = torch.randn(kp, 9, c, device=DEV).bfloat16()
    wi[:ko] = layout.conv_weight_to_internal(w, c).bfloat16()
    b = torch.randn(ko, device=DEV) if bias else None
    m = torch.randn(n, h, h, kp, device=DEV).bfloat16() if mask else None
    y = torch.full((n, h, h, kp), float("nan"), device=DEV, dtype=torch.bfloat16)
    K.conv_fprop_tc(layout.to_nhwc_padded(x, c), n, h, h, c, wi, kp, 3, 3, 1, 1, 1, h, h, y, kp, bias=b, relu=relu, mask_src=m,
                    n_valid=ko, n_store=kp)
    ref = F.conv2d(x.double(), w.double(), None if b is None else b.double(), padding=1).permute(0, 2, 3, 1)
    ref = torch.relu(ref) if relu else ref
    if mask:
        ref = ref * (m[..., :ko] > 0)
    assert K.read_status() == 0
    _close(y[..., :ko], ref)
    assert (y[..., ko:].float() == 0).all()


@pytest.mark.parametrize("mask", [False, True])
@pytest.mark.parametrize("c", [1, 16, 31, 33, 80])
def test_data_gradient_columns(c, mask):
    torch.manual_seed(c)
    n, ko, h = 2, 32, 6
    cp = K.pad_channels(c)
    w = (torch.randn(ko, c, 3, 3, device=DEV) / 17).bfloat16().float()
    dy = torch.randn(n, ko, h, h, device=DEV).bfloat16().float()
    add = torch.randn(n, h, h, cp, device=DEV).bfloat16()
    m = torch.randn(n, h, h, cp, device=DEV).bfloat16() if mask else None
    dx = torch.full((n, h, h, cp), float("nan"), device=DEV, dtype=torch.bfloat16)
    conv_dgrad(layout.to_nhwc_padded(dy, ko), n, h, h, ko, layout.conv_weight_to_internal(w, cp).bfloat16(), ko, cp, c, 3, 1, 1, h,
               h, dx, add=add, mask=m)
    ref = F.conv_transpose2d(dy.double(), w.double(), padding=1).permute(0, 2, 3, 1) + add[..., :c].double()
    if mask:
        ref = ref * (m[..., :c] > 0)
    assert K.read_status() == 0
    _close(dx[..., :c], ref)
    assert (dx[..., c:].float() == 0).all()
