"""The staged input kernel where groups of four pixels straddle an edge: crops that start at every offset from such a group, outside
the image on either side, flipped and not, with and without a mean and a border, tiles of one to sixteen rows, widths that are
no multiple of four; and that a network without augmentation draws nothing."""
import pytest
import torch

from rembrandt_b200.ops import native_ops as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("N,H,W", [(3, 5, 7), (40, 50, 61), (300, 18, 18), (2, 33, 40)])
@pytest.mark.parametrize("offset", [-3, -2, -1, 0, 1, 2, 3])
@pytest.mark.parametrize("flip", [False, True])
@pytest.mark.parametrize("border", [0, 2])
def test_crops_at_every_offset(N, H, W, offset, flip, border):
    C, Cp = 3, 32
    g = torch.Generator(device=DEV).manual_seed(N + offset)
    src = torch.randint(0, 256, (N, C, H, W), generator=g, device=DEV, dtype=torch.uint8)
    mean = torch.rand((C, H, W), generator=g, device=DEV) * 255 if N != 40 else None
    ch, cw = H, W + 2      # a window that the offset moves over the image's edges
    dst = torch.full((N, ch, cw, Cp), float("nan"), device=DEV, dtype=torch.bfloat16)
    K.input_u8(src, mean, dst, N, C, H, W, ch, cw, ch, cw, Cp, 1, offset, offset, offset, offset, False, flip, False, 1.0, 1.0,
               0.0, None, None, 1, 0, stride=1, border=border)
    torch.cuda.synchronize()
    img = src.float() if mean is None else src.float() - mean
    pad = 8
    big = torch.nn.functional.pad(img, (pad,) * 4)
    got = dst.float()[..., :C].permute(0, 3, 1, 2)
    assert bool((dst[..., C:] == 0).all())
    ys, xs = torch.arange(ch, device=DEV), torch.arange(cw, device=DEV)
    inside = ((ys >= border) & (ys < ch - border))[:, None] & ((xs >= border) & (xs < cw - border))[None, :]
    plain = big[:, :, pad + offset: pad + offset + ch, pad + offset: pad + offset + cw]
    forms = [plain] + ([plain.flip(3)] if flip else [])
    # one rounding to bf16; the difference before it may be fused. Each sample is one of the forms (a coin per sample).
    close = [((got - f * inside).abs() <= f.abs() * 2 ** -8 + 2e-5).flatten(1).all(1) for f in forms]
    assert bool(torch.stack(close).any(0).all())
    if flip and N == 300:
        assert bool((close[0] & ~close[1]).any()) and bool((close[1] & ~close[0]).any())
