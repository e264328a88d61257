"""Max pooling over windows around the size at which one byte no longer holds every offset and the "no gradient" code:
behind a ReLU with dead channels nothing may reach an inactive unit. On CPU the operators run their device path over the
stand-ins of tests/kernel_emulation.py; on a GPU the kernels themselves, in the row-mapped and in the generic form."""
import pytest
import torch
import torch.nn.functional as F

import kernel_emulation
from rembrandt_b200.models.config import (Act, AffineCfg, Conv2dCfg, Data3dCfg, ParamsInit, Pool2dCfg, PoolKind,
                                          SequentialOperatorConfig, SoftmaxKLLossCfg)
from rembrandt_b200.models.net import Net
from rembrandt_b200.ops import native_ops as K


def _cfg(hw, k, stride, channels=8):
    n = ParamsInit.normal
    cfg = SequentialOperatorConfig().data3d(Data3dCfg((hw, hw, 2), normalize=True))
    cfg.conv2d(Conv2dCfg(3, 1, 1, channels, Act.RECT, n(0.3)), "conv1")
    cfg.pool2d(Pool2dCfg(k, stride, 0, PoolKind.MAX), "pool1")
    return cfg.affine(AffineCfg(5, Act.IDENTITY, n(0.5)), "fc").softmax_kl_loss(SoftmaxKLLossCfg(5))


def _kill(net, channels):
    """Biases that keep every other channel of the convolution at zero."""
    op = net.hidden_ops[0]
    with torch.no_grad():
        net.params[op.seg_b.offset: op.seg_b.offset + channels: 2] = -50.0
        net.params16.copy_(net.params)


def _step(net, hw, batch):
    g = torch.Generator().manual_seed(hw)
    net.load_batch(torch.randint(0, 256, (batch, 2, hw, hw), dtype=torch.uint8, generator=g),
                   torch.randint(0, 5, (batch,), dtype=torch.int32, generator=g))
    net.forward(True)
    net.backward()
    conv = net.hidden_ops[0]
    return conv.out.float(), conv.dout.float()


@pytest.mark.parametrize("hw,k,stride", [(15, 15, 1), (16, 16, 1), (17, 16, 1), (20, 17, 3)])
def test_dead_channels_get_no_delta(monkeypatch, hw, k, stride):
    kernel_emulation.install(monkeypatch)
    monkeypatch.setattr(Net, "device_path_on_cpu", True)
    net = Net(_cfg(hw, k, stride), 3, device="cpu", seed=(3, 4))
    _kill(net, 8)
    out, delta = _step(net, hw, 3)
    assert float(delta.abs().sum()) > 0 and not bool((delta[out <= 0] != 0).any())


@pytest.mark.gpu
@pytest.mark.parametrize("generic", [False, True])
@pytest.mark.parametrize("hw,k,stride", [(15, 15, 1), (16, 16, 1), (17, 16, 1), (20, 17, 3), (40, 33, 5)])
def test_operator_against_the_host_path(monkeypatch, hw, k, stride, generic):
    if generic:
        monkeypatch.setenv("RB_POOL_GENERIC", "1")
    dev, host = (Net(_cfg(hw, k, stride, 64), 3, device=d, seed=(3, 4)) for d in ("cuda", "cpu"))
    _kill(dev, 64)
    with torch.no_grad():
        host.params.copy_(dev.params16.float().cpu())
    out, delta = _step(dev, hw, 3)
    torch.cuda.synchronize()
    assert K.read_status() == 0
    assert float(delta.abs().sum()) > 0 and not bool((delta[out <= 0] != 0).any())
    g = torch.Generator().manual_seed(hw)
    host.load_batch(torch.randint(0, 256, (3, 2, hw, hw), dtype=torch.uint8, generator=g),
                    torch.randint(0, 5, (3,), dtype=torch.int32, generator=g))
    host.forward(True)
    host.backward()
    for name in ("fc.b", "conv1.b"):
        seg, ref = (next(s for s in n.segs if s.name == name) for n in (dev, host))
        a, b = dev.seg_view(seg, "grads").float().cpu(), host.seg_view(ref, "grads")
        # bf16 activations and deltas (2^-9 each); a window's maximum may be another of two positions that round alike
        assert float((a - b).norm()) < 3e-2 * float(b.norm()), name


@pytest.mark.gpu
@pytest.mark.parametrize("k,stride,H,C", [(15, 1, 18, 64), (16, 1, 16, 64), (16, 2, 19, 32), (17, 5, 30, 64), (20, 1, 21, 8),
                                          (40, 3, 50, 64)])
@pytest.mark.parametrize("generic", [False, True])
def test_codes_against_autograd(monkeypatch, k, stride, H, C, generic):
    """Forward and backward kernels, clamped or masked, in the type that `pool_code_dtype` names."""
    if generic:
        monkeypatch.setenv("RB_POOL_GENERIC", "1")
    g = torch.Generator(device="cuda").manual_seed(k + H)
    N, P = 3, (H - k) // stride + 1
    x = torch.randn((N, H, H, C), generator=g, device="cuda").sub_(3.0).relu_().bfloat16()
    x[..., ::2] = 0                                                          # dead channels
    dy = torch.randn((N, P, P, C), generator=g, device="cuda").bfloat16()
    xd = x.double().permute(0, 3, 1, 2).requires_grad_()
    (want,) = torch.autograd.grad(F.max_pool2d(xd, k, stride), xd, dy.double().permute(0, 3, 1, 2))
    want = (want * (xd > 0)).permute(0, 2, 3, 1)
    mass = torch.autograd.grad(F.max_pool2d(xd, k, stride), xd, dy.double().abs().permute(0, 3, 1, 2))[0].permute(0, 2, 3, 1)
    for clamp in (True, False):
        y, idx = torch.empty_like(dy), torch.zeros(dy.shape, dtype=K.pool_code_dtype(k), device="cuda")
        dx = torch.full_like(x, float("nan"))
        K.pool_fwd(x, y, idx, N, H, H, C, P, P, k, stride, 0, True, clamp)
        K.pool_bwd(dy, idx, None, dx, None if clamp else x, N, H, H, C, P, P, k, stride, 0, True)
        assert torch.equal(y.double().permute(0, 3, 1, 2), F.max_pool2d(xd, k, stride))
        # at most P * P windows' deltas per position, each sum rounded to bf16 (2^-9 of the sum of their magnitudes)
        assert float(((dx.double() - want).abs() - mass * P * P * 2.0 ** -9).max()) <= 0


@pytest.mark.gpu
def test_more_offsets_than_codes_are_refused_in_the_backward_pass():
    x = torch.zeros((1, 17, 17, 64), device="cuda", dtype=torch.bfloat16)
    y = torch.zeros((1, 1, 1, 64), device="cuda", dtype=torch.bfloat16)
    idx = torch.zeros(y.shape, device="cuda", dtype=torch.uint8)
    K.pool_fwd(x, y, idx, 1, 17, 17, 64, 1, 1, 17, 1, 0, True, False)        # values are right without offsets
    with pytest.raises(RuntimeError):
        K.pool_bwd(y, idx, None, torch.empty_like(x), x, 1, 17, 17, 64, 1, 1, 17, 1, 0, True)
