"""A first convolution on few channels as a plain matrix product.

Three-channel images leave most of a filter tap's padded channels empty, and an implicit-GEMM load per tap fetches them all
the same: a 3 x 3 layer on 64 images of 256 x 256 x 3 took 604 us forward and 909 us for its weight gradient, for 0.8 GB of
real traffic each (this form: 206 and 160). Here the input operator writes the whole receptive field of every output
position, k * k * c values side by side (27 of 32 channels: no more bytes than one padded pixel), and the convolution is a
1 x 1 one over them; the weight gradient is a product of two matrices as they lie. A spare column holds ones, whose
weight-gradient column is the bias gradient. The parameters keep their layout: filters are gathered into window order before
the forward pass, and the gradient is scattered back, by two small kernels.
"""
from __future__ import annotations

import torch

from . import layout
from . import native_ops as K

# The window tensor is written once and read twice, and what it saves are the padded channels of the image form, whose reduction
# is taps x padded channels long. It pays, in training and at inference alike, where that is MIN_SAVING times as long as the
# window. Training step / inference pass of a network of this layer, a pooling and a small affine one, image form over windows
# (64 images):
#   reduction over window   layer                        step   inference
#   9.8   1568 / 160        7 x 7 x 3 on 256 x 256       3.7    2.9
#   9.0    288 / 32         3 x 3 x 3 on 256 x 256       1.7    1.5
#   3.2    512 / 160        7 x 7 x 3 / 2 on 256 x 256   1.4    1.2
#   3.0    288 / 96         5 x 5 x 3 / 2 on 224 x 224   1.3    1.1
#   3.0    288 / 96         3 x 3 x 10 on 64 x 64        1.20   1.00
#   2.25   288 / 128        3 x 3 x 12 on 64 x 64        1.15   0.94
#   2.0    128 / 64         4 x 4 x 3 / 2 on 224 x 224   1.07   0.99
#   1.8    288 / 160        3 x 3 x 16 on 64 x 64        1.05   0.84
#   1.6    256 / 160        7 x 7 x 3 / 4 on 224 x 224   0.94   0.86
#   1.3    256 / 192        8 x 8 x 3 / 4 on 224 x 224   0.89   0.82
# It takes columns x output positions of memory, at stride 1 up to MAX_COLUMNS / 32 times the padded image.
MIN_SAVING = 2.5
MAX_COLUMNS = 192


class WindowedFirstLayer:
    @staticmethod
    def fits(data_op, ksize, c, row_len, device) -> bool:
        """`row_len`: taps x padded channels of the layer's filters in the image form."""
        k = ksize * ksize * c
        return (device.type == "cuda" and ksize > 1 and k <= MAX_COLUMNS and row_len >= MIN_SAVING * K.pad_channels(k) and
                data_op.mode in ("nhwc", "s2d"))

    def __init__(self, data_op, ksize, stride, pad, P, Q, ko, c, cp, row_len, f):
        """`cp`, `row_len`, `f`: the layer's internal filters, [ko][row_len] with `cp` channels per tap, space-to-depth'd by
        `f` (None: not)."""
        k = ksize * ksize * c
        self.P, self.Q, self.ko, self.row_len = P, Q, ko, row_len
        self.cols = K.pad_channels(k)
        self.ones = k if k < self.cols else -1
        self.columns = layout.window_columns(ksize, c, cp, f)
        data_op.request_windows(ksize, stride, pad, P, Q, self.cols, self.ones)

    def alloc(self, batch, device, ldy, relu, has_bias):
        self.batch = batch
        self.index = torch.full((self.cols,), -1, dtype=torch.int32)
        self.index[: self.columns.numel()] = self.columns
        self.index = self.index.to(device)
        self.w16 = torch.zeros((self.ko, self.cols), dtype=torch.bfloat16, device=device)
        self.dw = torch.zeros((self.ko, self.cols), dtype=torch.float32, device=device)
        K.tune_conv(batch, self.P, self.Q, self.cols, self.ko, 1, 1, 1, 0, 0, self.P, self.Q, ldy, relu=relu,
                    has_bias=has_bias, n_valid=self.ko, n_store=ldy)

    def forward(self, x, w16, y, ldy, bias=None, relu=False):
        K.gather_columns(w16, self.index, self.w16, self.ko, self.row_len, self.cols)
        K.conv_fprop_tc(x, self.batch, self.P, self.Q, self.cols, self.w16, self.ko, 1, 1, 1, 0, 0, self.P, self.Q, y, ldy,
                        bias=bias, relu=relu, n_valid=self.ko, n_store=ldy)

    def backward(self, x, dy, ldy, gw, gbias=None):
        """Accumulates the filter gradient and, where there is a column of ones, the bias gradient."""
        K.gemm_tc(dy, 1, ldy, x, 1, self.cols, self.ko, self.cols, self.batch * self.P * self.Q, self.dw, self.cols,
                  epi=K.EPI_F32_ATOMIC, n_store=self.cols, split_k=0)
        K.scatter_columns(self.dw, self.index, gw, gbias if self.ones >= 0 else None, self.ko, self.row_len, self.cols,
                          self.ones)
