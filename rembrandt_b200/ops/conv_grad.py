"""Data-gradient of a convolution, any stride, as one call: dx = mask(add + gradient).

On a GPU this is `rb_conv_dgrad_tc` (csrc/gemm_tc.cu): the filters are read as they lie (or from a transposed and flipped
copy, `DgradPlan`), the output phases of a strided convolution share a launch and are written straight to their places in dx, and
the addend (the delta of an identity path, or the gradient of a parallel branch already in dx) and the mask of the producer's ReLU
ride in the epilogue. Strided geometries that it does not take, and all with RB_STRIDED_DGRAD_TC=0, run on the CUDA-core
kernel. Without a GPU the result is put together from the kernel fronts of `native_ops`, which the CPU tests replace by
plain torch.
"""
from __future__ import annotations

import os

import torch

from .. import _native
from .._native import check, ptr, stream_handle
from . import native_ops as K
from .conv_strided import dgrad_strided_tc

NEGATIVE_PADDING = -20


def _strided_on_cuda_cores(stride) -> bool:
    """RB_STRIDED_DGRAD_TC=0 keeps strided data-gradients on the CUDA-core kernel."""
    return stride > 1 and os.environ.get("RB_STRIDED_DGRAD_TC", "1") != "1"


def _compose(dy, n, P, Q, kp, w16, ko, cp, in_c, k, stride, pad, H, W, dx, add, mask):
    """The same from several launches. On a GPU only strided convolutions come here, without phases that the tensor-core
    kernel could run."""
    out = torch.empty_like(dx) if add is not None and add.data_ptr() == dx.data_ptr() else dx
    late = mask if add is not None else None
    early = None if add is not None else mask
    if stride == 1:
        wt = torch.zeros((cp, k * k, kp), dtype=torch.bfloat16, device=dy.device)
        K.pack_dgrad_filters(w16, wt, ko, kp, k * k, cp)
        K.conv_fprop_tc(dy, n, P, Q, kp, wt, cp, k, k, 1, k - 1 - pad, k - 1 - pad, H, W, out, cp, mask_src=early,
                        n_valid=in_c, n_store=cp)
    elif dy.device.type == "cuda" or _strided_on_cuda_cores(stride) or not dgrad_strided_tc(
            dy, n, P, Q, kp, w16, ko, cp, in_c, k, k, stride, pad, H, W, out, early):
        K.conv_direct_dgrad(dy, w16, out, early, n, H, W, cp, ko, kp, k, k, stride, pad, pad, P, Q)
    if add is not None:
        K.add_bf16(out, add, out.numel())
        if late is not None:
            K.relu_mask(out, late, out.numel())
        if out is not dx:
            dx.copy_(out)


def conv_dgrad(dy, n, P, Q, kp, w16, ko, cp, in_c, k, stride, pad, H, W, dx, add=None, mask=None, wt=None, add_masked=False):
    """dy: bf16 [n, P, Q, kp]; w16: bf16 filters [ko][k * k][cp]; dx: bf16 [n, H, W, cp], overwritten; add, mask: optional,
    shaped like dx (add may be dx); dx is zero where mask <= 0 and in channels >= in_c. wt: the filters as
    `native_ops.pack_dgrad_filters` writes them, to be read instead of w16. add_masked: add is zero already where the mask is."""
    if dy.device.type != "cuda" or _strided_on_cuda_cores(stride):
        _compose(dy, n, P, Q, kp, w16, ko, cp, in_c, k, stride, pad, H, W, dx, add, mask)
        return
    ws = K.gemm_workspace()
    geom = (ptr(dy), n, P, Q, kp, ptr(w16), ptr(wt), ko, cp, in_c, k, k, stride, pad, pad, H, W, ptr(dx))
    tail = (ptr(mask), ptr(ws), ws.numel() * 4, ptr(K.status_word()), stream_handle())
    if add_masked and add is not None and add.data_ptr() == dx.data_ptr():
        rc = _native.cuda().rb_conv_dgrad_onto_tc(*geom, *tail)
    else:
        rc = _native.cuda().rb_conv_dgrad_tc(*geom, ptr(add), *tail)
    if rc == NEGATIVE_PADDING:      # e.g. a padding larger than the filter: the CUDA-core kernel takes any geometry
        _compose(dy, n, P, Q, kp, w16, ko, cp, in_c, k, stride, pad, H, W, dx, add, mask)
        return
    check(rc, "rb_conv_dgrad_tc")


_measured: dict = {}


def _device_ms(fn, reps=4):
    """Best device time of `fn`, which has run before."""
    s, best = torch.cuda.current_stream(), 1e30
    for _ in range(reps):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(s)
        fn()
        e1.record(s)
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1))
    return best


class DgradPlan:
    """How one convolution's data-gradient reads its filters: in place, or from a transposed and flipped copy made once per
    step beside the forward pass. In place saves the copy; the copy is the K-major operand, with which the large shapes run
    10 % faster (64 x 64 x 64 x 256 -> 256: 274 against 243 us). Both are measured once per shape and process, on scratch
    operands; the copy has to win by more than a launch costs and half of the time that making it takes. Where a sixth of the
    time in place is less than that, no plans are searched for the copy: it was at most 13 % faster on every shape measured,
    and the search is most of what building a small network costs."""

    LAUNCH_MS, MOST_GAIN = 0.003, 1 / 6

    def __init__(self, n, P, Q, kp, ko, cp, in_c, k, stride, pad, H, W, forms, device="cuda"):
        """`forms`: the (addend, mask) combinations that will be asked for; `device`: the network's, current or not."""
        self.geom = (n, P, Q, kp, ko, cp, in_c, k, stride, pad, H, W)
        with torch.cuda.device(device):
            key = (torch.cuda.current_device(),) + self.geom + (tuple(forms),)
            if key not in _measured:
                _measured[key] = self._measure(forms)
        self.wt = torch.zeros((cp, k * k, kp), dtype=torch.bfloat16, device=device) if _measured[key] else None

    def _measure(self, forms) -> bool:
        n, P, Q, kp, ko, cp, in_c, k, stride, pad, H, W = self.geom
        zeros = lambda *s: torch.zeros(s, dtype=torch.bfloat16, device="cuda")
        dy, w, wt, dx = zeros(n, P, Q, kp), zeros(ko, k * k, cp), zeros(cp, k * k, kp), zeros(n, H, W, cp)

        def mean_ms(packed):
            total = 0.0
            for has_add, has_mask in forms:
                extra = dict(add=torch.zeros_like(dx) if has_add else None, mask=torch.zeros_like(dx) if has_mask else None)
                run = lambda: conv_dgrad(dy, n, P, Q, kp, w, ko, cp, in_c, k, stride, pad, H, W, dx, wt=packed, **extra)
                with K.gemm_tuning():
                    run()
                total += _device_ms(run)
            return total / len(forms)

        pack = lambda: K.pack_dgrad_filters(w, wt, ko, kp, k * k, cp)
        pack()
        cost = self.LAUNCH_MS + 0.5 * _device_ms(pack)
        in_place = mean_ms(None)
        better = in_place * self.MOST_GAIN > cost and in_place - mean_ms(wt) > cost
        torch.cuda.current_stream().synchronize()
        return better

    def prepare(self, net, w16):
        """Make the copy, if there is one, beside whatever the network does next."""
        if self.wt is not None:
            n, P, Q, kp, ko, cp, in_c, k, *_ = self.geom
            net.side(lambda: K.pack_dgrad_filters(w16, self.wt, ko, kp, k * k, cp))
