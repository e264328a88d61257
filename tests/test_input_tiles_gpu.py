"""The staged input kernel against a restatement in torch: windows that overlap (a first layer's whole receptive field
per output pixel), space to depth, many channels, odd widths, crop borders, the constant channel, both paths of the
dispatch (staged, and element by element when a row does not fit)."""
import pytest
import torch
import torch.nn.functional as F

from rembrandt_b200.ops import native_ops as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("N,C,H,W,win,stride,pad,extra", [
    (2, 3, 9, 9, 3, 1, 1, 5), (3, 1, 28, 28, 5, 1, 0, 7), (1, 3, 33, 33, 7, 2, 3, 13), (2, 3, 32, 32, 5, 1, 2, 21),
    (2, 32, 19, 19, 1, 1, 0, 0), (5, 3, 17, 17, 1, 1, 0, 29), (2, 3, 23, 23, 4, 4, 0, 16), (1, 4, 300, 300, 3, 1, 1, 4),
    (1, 16, 8, 700, 3, 1, 1, 0), (150, 2, 11, 11, 2, 2, 0, 0)])
@pytest.mark.parametrize("border", [False, True])
def test_windows(N, C, H, W, win, stride, pad, extra, border):
    g = torch.Generator(device=DEV).manual_seed(N * H + win)
    src = torch.randint(0, 256, (N, C, H, W), generator=g, device=DEV, dtype=torch.uint8)
    mean = torch.rand((C, H, W), generator=g, device=DEV) * 255
    k = win * win * C
    Cp = (k + extra + 31) // 32 * 32
    ones = k if extra else -1
    ch, cw = (H, W) if H < 12 else (H - 3, W - 3)            # a centred crop
    lo_y, hi_y, lo_x, hi_x = -pad, H - ch - pad, -pad, W - cw - pad
    eh, ew = ch + 2 * pad, cw + 2 * pad
    OH, OW = (eh - win) // stride + 1, (ew - win) // stride + 1
    dst = torch.full((N, OH, OW, Cp), float("nan"), device=DEV, dtype=torch.bfloat16)
    K.input_u8(src, mean, dst, N, C, H, W, eh, ew, OH, OW, Cp, win, lo_y, hi_y, lo_x, hi_x, False, False, False, 0.5, 0.25,
               0.0, None, None, 1, 0, stride=stride, border=pad if border else 0, ones=ones)
    img = src.float() * 0.5 - 0.25 * mean
    oy, ox = (H - ch) // 2 - pad, (W - cw) // 2 - pad         # centred on the crop, whatever padding surrounds it
    big = F.pad(img, (pad + ew, pad + ew, pad + eh, pad + eh))[:, :, pad + eh + oy: pad + 2 * eh + oy,
                                                             pad + ew + ox: pad + 2 * ew + ox].clone()
    if border and pad:
        inner = torch.zeros_like(big)
        inner[:, :, pad:-pad, pad:-pad] = big[:, :, pad:-pad, pad:-pad]
        big = inner
    cols = big.unfold(2, win, stride).unfold(3, win, stride)[:, :, :OH, :OW]       # N, C, OH, OW, dy, dx
    want = torch.zeros((N, OH, OW, Cp), device=DEV)
    want[..., :k] = cols.permute(0, 2, 3, 4, 5, 1).reshape(N, OH, OW, k)
    if ones >= 0:
        want[..., ones] = 1.0
    # one rounding to bf16; the product and difference before it may be fused
    assert float(((dst.float() - want).abs() - want.abs() * 2 ** -8).max()) < 2e-5
