"""The two-launch form of batch normalisation (statistics worked out by the kernel that applies them) against fp64 torch,
at channel counts that do and do not divide a block, more channels than one block covers, padded channels, and row counts
from one to several waves; every call runs three times on the same scratch, once without a backward pass between. And a scratch
of the three-launch form that layers of several widths share, among them one whose two-launch scratch has its length."""
import pytest
import torch
import torch.nn.functional as F

from rembrandt_b200.ops import native_ops as K

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _close(a, b, tol):
    err = (a.double() - b).norm() / b.norm().clamp_min(1e-12)
    assert float(err) < tol, float(err)


@pytest.mark.parametrize("rows,C,valid", [(1, 32, 32), (5, 8, 8), (37, 96, 96), (1000, 320, 300), (4097, 64, 64),
                                          (92416, 128, 128), (130, 2048, 2048), (77, 2112, 2100), (20011, 32, 16)])
def test_two_launch_form(rows, C, valid):
    g = torch.Generator(device=DEV).manual_seed(rows + C)
    rnd = lambda *s: torch.randn(*s, generator=g, device=DEV)
    x = (rnd(rows, C) * 2 + 1).bfloat16()
    x[:, valid:] = 0
    res = rnd(rows, C).bfloat16()
    gamma, beta = rnd(C) * 0.1 + 1, rnd(C)
    sums = K.bn_scratch(C, DEV)
    mean, istd = torch.empty(C, device=DEV), torch.empty(C, device=DEV)
    y = torch.empty(rows, C, device=DEV, dtype=torch.bfloat16)
    dy = rnd(rows, C).bfloat16()
    dy[:, valid:] = 0
    xd, m64 = x.double(), x.double().mean(0)
    v64 = ((xd - m64) ** 2).mean(0)
    s64 = torch.rsqrt(v64 + 1e-5)
    xh = (xd - m64) * s64
    out = torch.relu(xh * gamma.double() + beta.double() + res.double())[:, :valid]
    for again in range(3):
        rm, rv = torch.zeros(C, device=DEV), torch.ones(C, device=DEV)
        K.bn_fwd_train_ws(x, rows, C, valid, sums, 1e-5, 0.25, mean, istd, rm, rv, gamma, beta, res, y, True)
        # means of `rows` fp32 sums against 64 bits: 1e-4 of the deviation covers 92416 summands many times over
        assert float(((mean.double() - m64) * s64)[:valid].abs().max()) < 1e-4
        if rows > 1:
            _close(istd[:valid], s64[:valid], 1e-4)
            _close(rv[:valid], (0.75 + 0.25 * v64 * rows / (rows - 1))[:valid], 1e-4)
        if rows > 1:
            _close(y[:, :valid], out, 4e-3)      # bf16 rounding of the result: 2^-9 per value
        assert (y[:, valid:] == 0).all()
        if again == 0:
            continue
        dg, db = torch.ones(C, device=DEV), torch.ones(C, device=DEV)
        dx = torch.empty_like(x)
        K.bn_bwd_ws(x, dy, y, rows, C, valid, sums, mean, istd, gamma, dg, db, dx)
        gm = dy.double() * (y.double() > 0)
        assert float((db.double() - 1 - gm.sum(0))[:valid].abs().max()) < 1e-4 * rows ** 0.5 * 10
        if rows > 1:
            assert float((dg.double() - 1 - (gm * xh).sum(0))[:valid].abs().max()) < 1e-4 * rows ** 0.5 * 10
            want = gamma.double() * s64 * (gm - gm.mean(0) - xh * (gm * xh).mean(0))
            _close(dx[:, :valid], want[:, :valid], 6e-3)
        assert (dx[:, valid:] == 0).all() and (dg[valid:] == 1).all()
        # one of the two buffers of sums is clear for the next call, and named by the first word behind them
        spare = int(sums[4 * C:].view(torch.int32)[0])
        assert (sums[spare * 2 * C: (spare + 1) * 2 * C] == 0).all()
    K.bn_fwd_infer(x, rows, C, valid, 1e-5, rm, rv, istd, gamma, beta, res, y, False)
    want = (xd - rm.double()) * torch.rsqrt(rv.double() + 1e-5) * gamma.double() + beta.double() + res.double()
    _close(y[:, :valid], want[:, :valid], 4e-3)


def test_layers_share_a_scratch_of_the_three_launch_form():
    widths = (32, 80, 32, 80)
    sums = torch.zeros(2 * 80, device=DEV)           # 4 * 32 + 32 floats as well
    assert sums.numel() == 4 * 32 + K.BN_SCRATCH_TAIL
    g = torch.Generator(device=DEV).manual_seed(9)
    rows = 500
    for C in widths:
        x = (torch.randn(rows, C, generator=g, device=DEV) * 2 + 1).bfloat16()
        gamma, beta = torch.ones(C, device=DEV), torch.zeros(C, device=DEV)
        mean, istd, dg, db = (torch.zeros(C, device=DEV) for _ in range(4))
        y, dx = torch.empty_like(x), torch.empty_like(x)
        K.bn_fwd_train(x, rows, C, C, sums, 1e-5, 1.0, mean, istd, None, None, gamma, beta, None, y, False)
        K.bn_bwd(x, x, None, rows, C, C, sums, mean, istd, gamma, dg, db, dx)
        m64 = x.double().mean(0)
        assert float((mean.double() - m64).abs().max()) < 1e-4 and (sums == 0).all()
        assert float((db.double() - x.double().sum(0)).abs().max()) < 1e-4 * rows ** 0.5 * 10
    with pytest.raises(ValueError):
        K.bn_bwd_ws(x, x, None, rows, 80, 80, sums, mean, istd, gamma, dg, db, dx)
