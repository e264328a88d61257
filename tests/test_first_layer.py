"""Which first layers run over whole receptive fields: those whose image form was measured to be slower, at each side of the
rule's line (the GPU tests compare both forms with the host path)."""
from types import SimpleNamespace

import pytest
import torch

from rembrandt_b200.ops import layout
from rembrandt_b200.ops import native_ops as K
from rembrandt_b200.ops.first_layer import WindowedFirstLayer


@pytest.mark.parametrize("hw,c,k,s,p,windows", [
    (256, 3, 3, 1, 1, True), (256, 3, 5, 1, 2, True), (256, 3, 7, 1, 3, True), (28, 1, 5, 1, 0, True), (256, 3, 7, 2, 3, True),
    (224, 3, 5, 2, 2, True), (32, 7, 5, 1, 2, True),
    # slower than the image form, in training or at inference
    (64, 16, 3, 1, 1, False), (256, 20, 3, 1, 1, False), (224, 3, 6, 3, 0, False), (224, 3, 8, 4, 2, False),
    (224, 3, 7, 4, 2, False),
    # more columns than any that was measured
    (227, 3, 11, 4, 0, False), (64, 3, 9, 1, 4, False)])
def test_windows_are_taken_where_they_were_measured_to_pay(hw, c, k, s, p, windows):
    mode, taps, cp = "nhwc", k * k, K.pad_channels(c)
    if s > 1 and c <= 4:                         # the image form of a strided layer on few channels is space-to-depth'd
        f, r2, _, _ = layout.s2d_geometry(k, s, hw + 2 * p)
        mode, taps, cp = "s2d", r2 * r2, K.pad_channels(f * f * c)
    assert WindowedFirstLayer.fits(SimpleNamespace(mode=mode), k, c, taps * cp, torch.device("cuda")) == windows
    assert not WindowedFirstLayer.fits(SimpleNamespace(mode="flat"), k, c, taps * cp, torch.device("cuda"))
    assert not WindowedFirstLayer.fits(SimpleNamespace(mode=mode), k, c, taps * cp, torch.device("cpu"))
