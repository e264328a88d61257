"""The form of the tensor-core convolution that keeps whole input rows in shared memory for all filter taps, against fp64: rows
of one position to the longest that a load takes (and one longer, which another form runs), rows around 128 outputs, where
sub-tiles change from 128 positions to one row, paddings of zero, of more than the filter reaches and on one side only, images
of one row, filters of one row or column, several channel chunks, every number of sub-tiles per item, resident filters, pairs;
several items per CTA; data-gradients from filters read in place and packed, their strided phases, addends and masks."""
import pytest
import torch
import torch.nn.functional as F

from test_conv_dgrad_gpu import _run as data_gradient

from rembrandt_b200.ops import layout
from rembrandt_b200.ops import native_ops as K

pytestmark = pytest.mark.gpu
DEV = "cuda"
FLAT = 3      # the kernel's number of this form in `gemm_last_launch`

CASES = [  # N, C, H, W, Kout, R, S, pad_h, pad_w, more rows at the bottom, more columns at the right
    (2, 32, 1, 1, 32, 3, 3, 1, 1, 0, 0), (3, 32, 5, 1, 64, 3, 3, 1, 1, 0, 0), (1, 64, 1, 9, 32, 3, 3, 1, 1, 0, 0),
    (2, 64, 6, 112, 64, 3, 3, 1, 1, 0, 0), (2, 64, 6, 126, 64, 3, 3, 1, 1, 0, 0), (2, 64, 5, 127, 64, 3, 3, 1, 1, 0, 0), (2, 64, 5, 128, 128, 3, 3, 1, 1, 0, 0),
    (2, 32, 4, 129, 32, 3, 3, 1, 1, 0, 0), (2, 32, 4, 130, 32, 3, 3, 0, 0, 0, 0), (1, 32, 3, 255, 32, 3, 3, 1, 1, 0, 0),
    (1, 32, 3, 256, 32, 3, 3, 1, 1, 0, 0), (300, 64, 3, 3, 64, 3, 3, 1, 1, 0, 0), (2, 160, 9, 11, 96, 3, 3, 0, 0, 0, 0),
    (2, 96, 7, 8, 256, 5, 5, 4, 4, 0, 0), (2, 64, 7, 8, 32, 2, 2, 1, 0, 0, 1), (2, 64, 7, 8, 32, 2, 2, 0, 1, 1, 0),
    (3, 32, 8, 7, 320, 1, 5, 0, 2, 0, 0), (3, 32, 8, 7, 64, 5, 1, 2, 0, 0, 0), (2, 32, 9, 9, 32, 3, 3, 3, 3, 0, 0),
    (2, 64, 10, 10, 64, 3, 3, 1, 1, -3, -2), (9, 512, 4, 4, 64, 3, 3, 1, 1, 0, 0)]


@pytest.mark.parametrize("options", [dict(), dict(force_mt=1), dict(force_mt=2), dict(force_mt=3), dict(force_mt=4),
                                     dict(force_resident=1), dict(force_resident=0, force_pair=0), dict(force_pair=1)])
@pytest.mark.parametrize("case", CASES)
def test_flat_convolution(case, options):
    N, C, H, W, Ko, R, S, ph, pw, dh, dw = case
    torch.manual_seed(sum(case))
    P, Q = H + 2 * ph - R + 1 + dh, W + 2 * pw - S + 1 + dw
    x = torch.randn(N, C, H, W, device=DEV).bfloat16().float()
    w = (torch.randn(Ko, C, R, S, device=DEV) / (C * R * S) ** 0.5).bfloat16().float()
    b = torch.randn(Ko, device=DEV)
    m = torch.randn(N, P, Q, Ko, device=DEV).bfloat16()
    y = torch.full((N, P, Q, Ko), float("nan"), device=DEV, dtype=torch.bfloat16)
    wi = w.permute(0, 2, 3, 1).reshape(Ko, R * S, C).contiguous().bfloat16()
    with K.gemm_options(force_halo=1, **options):
        K.conv_fprop_tc(layout.to_nhwc_padded(x, C), N, H, W, C, wi, Ko, R, S, 1, ph, pw, P, Q, y, Ko, bias=b, mask_src=m,
                        n_valid=Ko, n_store=Ko)
        plan = K.gemm_last_launch()
    assert K.read_status() == 0
    pitch = Q + S - 1 - max(0, min(pw, S - 1, Q + S - 1 - pw - W))
    assert (plan["a_mode"] == FLAT) == (pitch <= 256)
    ref = F.conv2d(F.pad(x.double(), (pw, pw + max(dw, 0), ph, ph + max(dh, 0))), w.double(), b.double())[:, :, :P, :Q]
    ref = ref.permute(0, 2, 3, 1) * (m > 0)
    # operands are exact in bf16, sums are fp32: the rounding of the result, and the order of the additions of terms of size 1
    assert ((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4).all()


# several work items per CTA: rings of operands and both accumulator sets go on from item to item
MANY = [(1200, 64, 13, 13, 64, 3, 3, 1, 1, 0, 0), (700, 160, 13, 12, 96, 3, 3, 1, 1, 0, 0), (500, 32, 13, 13, 320, 3, 3, 0, 1, 0, 0),
        (160, 64, 8, 126, 64, 3, 3, 1, 1, 0, 0)]


@pytest.mark.parametrize("options", [dict(force_mt=1), dict(force_mt=2), dict(force_mt=3), dict(force_mt=4),
                                     dict(force_resident=1), dict(force_resident=0, force_pair=0), dict(force_pair=1)])
@pytest.mark.parametrize("case", MANY)
def test_many_items(case, options):
    test_flat_convolution(case, options)
    plan, (N, C, H, W, Ko, R, S, ph, pw) = K.gemm_last_launch(), case[:9]
    # not less than: positions without the zero columns and rows, in whole items, by column tiles
    items = N * (H + 2 * ph - R + 1) * (W + 2 * pw - S + 1) // (128 * plan["sub_tiles"]) * -(-Ko // plan["tile_width"])
    assert items > plan["grid"]


DGRADS = [  # N, C, Ko, H, k, stride, pad [, W]; the last phase of the strided ones has several taps
    (5, 128, 128, 19, 3, 1, 1), (2, 256, 96, 13, 5, 1, 2), (3, 16, 40, 9, 3, 1, 1, 14), (900, 64, 64, 13, 3, 1, 1),
    (37, 64, 32, 73, 3, 2, 1, 19), (2, 32, 64, 15, 3, 2, 1, 6), (1, 128, 256, 8, 5, 3, 2, 17), (300, 96, 64, 25, 3, 2, 1)]


@pytest.mark.parametrize("options", [dict(), dict(force_mt=1), dict(force_mt=2), dict(force_mt=3), dict(force_mt=4),
                                     dict(force_resident=1), dict(force_pair=1)])
@pytest.mark.parametrize("add,masked", [(None, False), (None, True), ("own", True), ("dx", False), ("dx", True)])
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("shape", DGRADS)
def test_flat_data_gradient(shape, packed, add, masked, options):
    data_gradient(shape, add, masked, packed, force_halo=1, **options)
    assert K.gemm_last_launch()["a_mode"] == FLAT
