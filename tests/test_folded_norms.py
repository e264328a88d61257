"""Inference passes of normalised networks, whose convolutions normalise in their epilogues by running statistics, against the
host path, operator by operator: first layers of both forms, both residual blocks with every shortcut, another activation after
the normalisation, none, channel counts off the 32-column groups; a different epsilon per operator, and scales, biases and
running statistics away from their initial values. On the device path's CPU stand-ins and on a GPU, there also as the engine runs
them: again after training has moved what they read, eager and from the captured graph."""
import pytest
import torch

import kernel_emulation
from rembrandt_b200.api import build_replica, model_config
from rembrandt_b200.models.config import (Act, AffineCfg, BNormConv2dCfg, Data3dCfg, ParamsInit, Pool2dCfg, PoolKind,
                                          ProjStackResConv2dCfg, SequentialOperatorConfig, SoftmaxKLLossCfg, StackResConv2dCfg)
from rembrandt_b200.models.net import Net
from rembrandt_b200.models.resnet_ops import _BlockBase
from rembrandt_b200.ops import native_ops as K

KAIMING = ParamsInit.kaiming()


def _cfg(stem):
    cfg = SequentialOperatorConfig().data3d(Data3dCfg((18, 18, 3), normalize=True))
    k, s, p = {"plain": (3, 1, 1), "strided": (7, 2, 3)}[stem]
    cfg.bnorm_conv2d(BNormConv2dCfg(k, s, p, 24, Act.RECT, KAIMING, bnorm_epsilon=0.1), "stem")
    cfg.stack_res_conv2d(StackResConv2dCfg(KAIMING, bnorm_epsilon=0.3), "same")
    cfg.proj_stack_res_conv2d(ProjStackResConv2dCfg(40, None, KAIMING, bnorm_epsilon=0.5), "half")
    cfg.proj_stack_res_conv2d(ProjStackResConv2dCfg(64, (9 if stem == "plain" else 5), KAIMING, bnorm_epsilon=0.7), "wider")
    cfg.bnorm_conv2d(BNormConv2dCfg(1, 1, 0, 33, Act.TANH, KAIMING, bnorm_epsilon=0.9), "smooth")
    cfg.bnorm_conv2d(BNormConv2dCfg(3, 2, 1, 32, Act.IDENTITY, KAIMING, bnorm_epsilon=1.1), "plain")
    cfg.pool2d(Pool2dCfg(3, 1, 0, PoolKind.AVERAGE), "pool")
    cfg.affine(AffineCfg(10, Act.IDENTITY, ParamsInit.xavier()), "out")
    return cfg.softmax_kl_loss(SoftmaxKLLossCfg(10))


def _units(net):
    return [u for op in net.ops if isinstance(op, _BlockBase) for u in op.units]


def _randomise(net, seed):
    gen = torch.Generator().manual_seed(seed)
    for u in _units(net):
        for seg, low in ((u.seg_g, 0.5), (u.seg_b, -0.5), (u.seg_rm, -0.5), (u.seg_rv, 0.2)):
            net.seg_view(seg)[: u.ko] = (torch.rand(u.ko, generator=gen) + low).to(net.params.device)


def _host_copy(net, cfg):
    """A network on the host path with the filters and weights that the kernels use, and the rest as it is."""
    host = Net(cfg, net.batch, device="cpu", seed=(1, 2))
    with torch.no_grad():
        host.params.copy_(net.params.cpu())
        for seg in net.segs:
            if seg.name.endswith(".w"):
                host.seg_view(seg).copy_(net.seg_view(seg, "params16").float().cpu())
    return host


def _compare(net, host, x):
    live = lambda op: op.out[..., : op.out_hwc[2]].float().cpu().permute(0, 3, 1, 2)
    for op, ref in zip(net.ops[1:-1], host.ops[1:-1]):
        if not isinstance(op, _BlockBase):
            continue
        with torch.no_grad():                 # of what the operator before it has left on the device
            want = ref.ref_forward(host.input_op.ref_forward(x, False, 0) if op.prev is net.input_op else live(op.prev), False, 0)
        # rounded to bf16, 2^-9 each: the image (first layer), the first convolution, the projection, the sum
        assert float((live(op) - want).norm()) < 4 * 2.0 ** -9 * float(want.norm()), op.name
        assert float(op.out[..., op.out_hwc[2]:].float().abs().sum()) == 0.0, op.name


def _run(net, stem):
    assert net.is_cuda and net.folded_norms is not None
    first = net.hidden_ops[0].u
    assert all((u.fold is None) == (u is first and (u.windowed is not None or u.s2d is not None)) for u in _units(net))
    x = torch.randint(0, 256, (net.batch, 3, 18, 18), dtype=torch.uint8, generator=torch.Generator().manual_seed(2))
    y = torch.arange(net.batch, dtype=torch.int32) % 10
    for seed in (5, 6):                       # what the first pass works out is not kept
        _randomise(net, seed)
        net.load_batch(x.to(net.params.device), y.to(net.params.device))
        net.forward(False)
        _compare(net, _host_copy(net, _cfg(stem)), x)


@pytest.mark.parametrize("stem", ["plain", "strided"])
def test_device_path_on_the_cpu(monkeypatch, stem):
    kernel_emulation.install(monkeypatch)
    monkeypatch.setattr(Net, "device_path_on_cpu", True)
    net = Net(_cfg(stem), 4, device="cpu", seed=(3, 4))
    monkeypatch.setattr(Net, "device_path_on_cpu", False)
    _run(net, stem)


@pytest.mark.gpu
@pytest.mark.parametrize("stem", ["plain", "strided"])
def test_on_a_gpu(stem):
    _run(Net(_cfg(stem), 5, device="cuda", seed=(3, 4)), stem)
    torch.cuda.synchronize()
    assert K.read_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("use_graph", [True, False])
def test_inference_follows_training(use_graph):
    batch, hw = 16, 32
    eng = build_replica("resnet20_cifar", batch, use_graph=use_graph, seed=(5, 7))
    gen = torch.Generator().manual_seed(3)
    draw = lambda: (torch.randint(0, 256, (batch, 3, hw, hw), dtype=torch.uint8, generator=gen).pin_memory(),
                    torch.randint(0, 10, (batch,), dtype=torch.int32, generator=gen).pin_memory())
    x, y = draw()
    losses = []
    for _ in range(4):                        # eager, captured, and replays of what was captured before the weights moved
        loss, _ = eng.eval_batch(x, y)
        _compare(eng.net, _host_copy(eng.net, model_config("resnet20_cifar")), x)
        losses.append(loss)
        eng.feed(*draw())
        eng.step()
        eng.flush()
    eng.synchronize()
    assert K.read_status() == 0
    assert len(set(losses)) == 4
