"""Average pooling over windows large enough to be split over a block, against torch, where the channel groups or the
window do not divide the block, with padding and several outputs per sample."""
import pytest
import torch
import torch.nn.functional as F

from rembrandt_b200.ops import native_ops as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("N,C,H,k,stride,pad,relu", [(3, 64, 8, 8, 1, 0, False), (1, 8, 4, 4, 1, 0, False),
                                                     (2, 96, 7, 7, 7, 0, True), (5, 1024, 6, 6, 1, 0, False),
                                                     (2, 160, 13, 5, 3, 2, True), (1, 136, 9, 9, 9, 0, False)])
def test_large_window_average(N, C, H, k, stride, pad, relu):
    g = torch.Generator(device=DEV).manual_seed(C + H)
    P = (H + 2 * pad - k) // stride + 1
    x = torch.randn((N, H, H, C), generator=g, device=DEV).bfloat16()
    y = torch.full((N, P, P, C), float("nan"), device=DEV, dtype=torch.bfloat16)
    K.pool_fwd(x, y, None, N, H, H, C, P, P, k, stride, pad, False, relu)
    ref = F.avg_pool2d(x.double().permute(0, 3, 1, 2), k, stride, pad, count_include_pad=True).permute(0, 2, 3, 1)
    ref = ref.relu() if relu else ref
    # one rounding to bf16 (2^-9 of the value) after an fp32 sum
    assert float(((y.double() - ref).abs() - ref.abs() * 2 ** -8).max()) < 1e-5


@pytest.mark.parametrize("k,stride,H", [(2, 2, 16), (3, 2, 13), (3, 1, 9)])
def test_recorded_offsets_carry_the_producers_relu(k, stride, H):
    """Behind a ReLU, clamping in the max-pooling forward pass and no mask in backward give what the mask gives."""
    g = torch.Generator(device=DEV).manual_seed(k + H)
    N, C, P = 3, 64, (H - k) // stride + 1
    x = torch.randn((N, H, H, C), generator=g, device=DEV).sub_(1.0).relu_().bfloat16()      # most windows hold zeros
    dy = torch.randn((N, P, P, C), generator=g, device=DEV).bfloat16()
    got = []
    for clamp in (False, True):
        y, idx = torch.empty_like(dy), torch.empty(dy.shape, dtype=torch.uint8, device=DEV)
        dx = torch.full_like(x, float("nan"))
        K.pool_fwd(x, y, idx, N, H, H, C, P, P, k, stride, 0, True, clamp)
        K.pool_bwd(dy, idx, None, dx, None if clamp else x, N, H, H, C, P, P, k, stride, 0, True)
        got.append((y, dx))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("k,H,W,pad,C", [(2, 16, 16, 0, 64), (2, 15, 17, 0, 32), (2, 13, 12, 1, 64), (3, 13, 13, 0, 96),
                                         (3, 27, 55, 0, 64), (3, 16, 16, 1, 64), (3, 7, 6, 1, 256), (2, 2, 2, 0, 512)])
@pytest.mark.parametrize("masked", [False, True])
def test_stride_two_backward_against_a_gather(k, H, W, pad, C, masked):
    """Odd and even extents, positions that no window covers, floor and ceil output sizes: the same bits as adding the
    windows' contributions one by one in bf16."""
    g = torch.Generator(device=DEV).manual_seed(H * W + k)
    N = 3
    for ceil in (False, True):
        up = 1 if ceil else 0
        P, Q = ((e + 2 * pad - k + up) // 2 + 1 for e in (H, W))
        if (P - 1) * 2 >= H + pad or (Q - 1) * 2 >= W + pad:
            continue
        x = torch.randn((N, H, W, C), generator=g, device=DEV).bfloat16()
        dy = torch.randn((N, P, Q, C), generator=g, device=DEV).bfloat16()
        y, idx = torch.empty_like(dy), torch.empty(dy.shape, dtype=torch.uint8, device=DEV)
        K.pool_fwd(x, y, idx, N, H, W, C, P, Q, k, 2, pad, True, True)
        dx = torch.full_like(x, float("nan"))
        K.pool_bwd(dy, idx, None, dx, x if masked else None, N, H, W, C, P, Q, k, 2, pad, True)
        want = torch.zeros((N, H + 2 * pad + k, W + 2 * pad + k, C), device=DEV, dtype=torch.bfloat16)
        for r in reversed(range(k)):             # windows above come first, and hold the position at a larger offset
            for s in reversed(range(k)):
                want[:, r: r + 2 * P: 2, s: s + 2 * Q: 2] += dy * (idx == r * k + s)
        want = want[:, pad: pad + H, pad: pad + W]
        want = want * (x > 0) if masked else want
        assert torch.equal(dx, want)
