"""A network on a GPU that is not the current one: the copy of a layer's filters lies where its kernels run."""
import contextlib

import torch

from rembrandt_b200.ops import conv_grad


def test_the_copy_lies_on_the_networks_device(monkeypatch):
    current, made = [0], []

    @contextlib.contextmanager
    def device(d):
        before, current[0] = current[0], torch.device(d).index
        yield
        current[0] = before

    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: current[0])
    # a plan is measured on the device that it is for, and each device's result is its own
    monkeypatch.setattr(conv_grad, "_measured", {})
    monkeypatch.setattr(conv_grad.DgradPlan, "_measure", lambda self, forms: current[0] == 1)
    monkeypatch.setattr(torch, "zeros", lambda *a, device=None, **k: made.append(torch.device(device)) or "copy")
    shape = (4, 8, 8, 32, 32, 32, 32, 3, 1, 1, 8, 8, [(False, True)])
    assert conv_grad.DgradPlan(*shape, device=torch.device("cuda", 1)).wt == "copy" and current == [0]
    assert conv_grad.DgradPlan(*shape, device=torch.device("cuda", 0)).wt is None
    assert made == [torch.device("cuda", 1)]
