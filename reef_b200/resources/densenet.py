"""DenseNet schedule graphs (DenseNet-121/169/201; growth 32, bottleneck 4x).

A dense layer is BN-ReLU-conv1x1-BN-ReLU-conv3x3 whose 32 output channels are appended to the block's
feature map.  The concatenation is never materialised as a copy (the reference's TVM build emits
`fused_concatenate_N` kernels, reference: resource/inception/inception.cu:288): every producer writes its
channels at an offset of one shared channels-last buffer (`ocs`/`ooff` in the kernel name) and every
consumer reads a channel prefix of it (`ics`/`ioff`).  The first BN-ReLU of a layer acts on that prefix (with
the folded shift; its positive scale moves into the 1x1 weights): `fused_add_nn_relu` on the channels that
are older than the previous layer, off the critical path, and the epilogue of the previous layer's 3x3 conv
on its own channels (`Builder.conv_append`).  The second is folded into the 1x1 conv (`conv2d_add_nn_relu`).  Transitions: BN-ReLU, 1x1 conv, 2x2/2 average pool."""
from __future__ import annotations

import numpy as np

from .graph import Tensor
from .layers import Builder

_BLOCKS = {121: [6, 12, 24, 16], 169: [6, 12, 32, 32], 201: [6, 12, 48, 32]}


def build_densenet(depth: int = 201, *, name: str | None = None, image: int = 224, classes: int = 1000,
                   growth: int = 32, seed: int = 4002, conv_impl: str = "auto") -> Builder:
    blocks = _BLOCKS[depth]
    b = Builder(name or f"densenet{depth}", seed, conv_impl)
    g = b.g
    data = g.input("data", 3 * image * image)
    s0, t0 = b.bn(64)
    x = b.stem_conv(data, 3, image, image, 64, 7, 2, 3, out_scale=s0, bias=t0, relu=True)
    pool, c = ("max", 3, 2, 1), 64
    for bi, n_layers in enumerate(blocks):
        c_total = c + n_layers * growth
        # the stage before the block ends in a pooling: it writes the first channels of the block's concat buffer
        h, w = ((d + 2 * pool[3] - pool[1]) // pool[2] + 1 for d in (x.h, x.w))
        buf = Tensor(g.temp(h * w * c_total), h, w, c_total)
        b.pool(x, *pool, out=b.slice_of(buf, 0, c), count_include_pad=True)
        s, t = b.bn(c)
        act = b.bias_relu_slice(b.slice_of(buf, 0, c), t / s)
        for li in range(n_layers):
            cin = c + li * growth
            s2, t2 = b.bn(4 * growth)
            mid = b.conv(act, 4 * growth, 1, 1, 0, in_scale=s, out_scale=s2, bias=t2, relu=True)
            w3 = b.he_conv(growth, 3, 3, 4 * growth)
            s, t = b.bn(cin + growth)            # BN of the next layer, of the transition or of the head
            act = b.conv_append(mid, growth, 3, 1, buf, cin, t / s, weight=w3, w_gain=0.5)
        c = c_total
        if bi != len(blocks) - 1:
            x = b.conv(act, c // 2, 1, 1, 0, in_scale=s)
            pool, c = ("avg", 2, 2, 0), c // 2
    pooled = b.global_avg_pool(act)          # of the final BN-ReLU (scale dropped: it only rescales the logits' input)
    flat = b.flatten(pooled)
    logits = b.dense(flat, classes, w_std=float(np.sqrt(1.0 / c)) * 0.5)
    b.softmax_output(logits)
    b.logits_idx = logits.idx
    return b
