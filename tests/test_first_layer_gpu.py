"""A first layer over whole receptive fields against the fp32 host path: same loss, same gradients, same layout of the
parameters. Plain and strided (space-to-depth'd) filters, with and without a spare column for the bias gradient, crops
smaller than the image, normalised layers, a layer too wide for it."""
import pytest
import torch
import torch.nn.functional as F

from rembrandt_b200.models.config import (Act, AffineCfg, BNormConv2dCfg, Conv2dCfg, Data3dCfg, ParamsInit, Preproc,
                                          SequentialOperatorConfig, SoftmaxKLLossCfg)
from rembrandt_b200.models.net import Net
from rembrandt_b200.ops import native_ops as K

pytestmark = pytest.mark.gpu


def _cfg(hw, c, k, s, p, ko, bnorm=False, crop=None):
    n = ParamsInit.normal
    pre = [Preproc("crop", crop_width=crop, crop_height=crop)] if crop else []
    cfg = SequentialOperatorConfig().data3d(Data3dCfg((hw, hw, c), normalize=True, preprocs=pre))
    if bnorm:
        cfg.bnorm_conv2d(BNormConv2dCfg(k, s, p, ko, Act.RECT, n(0.2)), "conv1")
    else:
        cfg.conv2d(Conv2dCfg(k, s, p, ko, Act.RECT, n(0.2)), "conv1")
    return cfg.affine(AffineCfg(10, Act.IDENTITY, n(0.05)), "fc").softmax_kl_loss(SoftmaxKLLossCfg(10))


@pytest.mark.parametrize("hw,c,k,s,p,ko,bnorm,crop,windows", [
    (12, 3, 3, 1, 1, 16, False, None, True), (28, 1, 5, 1, 0, 20, False, None, True), (16, 3, 5, 1, 2, 32, True, None, True),
    (20, 2, 4, 1, 0, 40, False, None, True), (33, 3, 7, 2, 3, 64, True, None, True), (31, 3, 5, 2, 0, 24, False, None, True),
    (14, 3, 3, 1, 1, 16, False, 10, True), (12, 32, 3, 1, 1, 16, False, None, False)])
def test_against_the_host_path(hw, c, k, s, p, ko, bnorm, crop, windows):
    batch = 6
    g, h = (Net(_cfg(hw, c, k, s, p, ko, bnorm, crop), batch, device=d, seed=(3, 4),
                minibatch_size=2 * batch) for d in ("cuda", "cpu"))
    op = g.hidden_ops[0]
    unit = op.u if bnorm else op
    assert (unit.windowed is not None) == windows
    gen = torch.Generator().manual_seed(hw + k)
    x = torch.randint(0, 256, (batch, c, hw, hw), dtype=torch.uint8, generator=gen)
    y = torch.randint(0, 10, (batch,), dtype=torch.int32, generator=gen)
    train = crop is None                         # the training form draws a random crop
    for _ in range(2):                           # gradients accumulate
        for net in (g, h):
            net.load_batch(x, y)
            net.forward(train)
        if train:
            g.backward()
            h.backward()
    torch.cuda.synchronize()
    assert K.read_status() == 0
    (gl, _), (hl, _) = g.read_stats(), h.read_stats()
    assert abs(gl - hl) < 2e-2 * abs(hl)
    if not train:
        return
    for gs, hs in zip(g.segs, h.segs):
        if not gs.trainable:
            continue
        a, b = g.seg_view(gs, "grads").float().cpu(), h.seg_view(hs, "grads")
        if gs is unit.seg_w:
            # nothing may arrive where the filters' internal layout has no weight
            assert abs(float(a.abs().sum()) - float(unit._w_ref(a).abs().sum())) < 1e-3 * float(a.abs().sum())
            a, b = unit._w_ref(a), unit._w_ref(b)
        # bf16 activations and deltas (2^-9 each) against fp32, ReLU signs that flip at zero; a normalisation takes the
        # mean and the projection on its output out of the delta, so what is left carries two to three times the error
        assert float((a - b).norm()) < (9e-2 if bnorm else 3e-2) * float(b.norm()) + 1e-6, gs.name


@pytest.mark.parametrize("hw,crop,k,s,p,bnorm", [
    (15, 14, 3, 1, 1, False), (17, 14, 5, 1, 2, False), (16, 15, 3, 1, 1, False), (17, 14, 4, 1, 0, False),
    (21, 20, 7, 2, 3, True), (24, 19, 5, 2, 2, False), (33, 32, 11, 4, 5, False)])
def test_the_inference_crop_is_centred(hw, crop, k, s, p, bnorm):
    """Margins that are odd and smaller than the layer's padding on both sides, in the windowed and the space-to-depth form:
    the convolution of the crop that the host path takes. One pixel off changes noise images altogether."""
    batch = 3
    g, h = (Net(_cfg(hw, 3, k, s, p, 16, bnorm, crop), batch, device=d, seed=(3, 4)) for d in ("cuda", "cpu"))
    gen = torch.Generator().manual_seed(hw + k)
    x = torch.randint(0, 256, (batch, 3, hw, hw), dtype=torch.uint8, generator=gen)
    g.load_batch(x, torch.zeros(batch, dtype=torch.int32))
    g.forward(False)
    torch.cuda.synchronize()
    op = g.hidden_ops[0]
    if bnorm:
        w, got = op.u._w_ref(g.seg_view(op.u.seg_w).float().cpu()), op.u.conv_out
    else:
        w, got = op._w_ref(g.seg_view(op.seg_w).float().cpu()), op.out
    want = F.conv2d(h.input_op.ref_forward(x, False, 0), w.bfloat16().float(), stride=s, padding=p)
    if not bnorm:
        want = want.relu()                       # the biases are zero at first
    inner = slice(2, -2)                         # the space-to-depth form sees the image beyond the crop in its padding
    a = got[..., :16].float().cpu().permute(0, 3, 1, 2)[..., inner, inner]
    # bf16 pixels and one rounding of the result: 2^-9 each
    assert float((a - want[..., inner, inner]).norm()) < 1e-2 * float(want[..., inner, inner].norm())
