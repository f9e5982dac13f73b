"""Contractions whose weights have just been brought to the device, in memory that other work has just given back."""
import random
from ctypes import c_void_p

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAYERS = [(1024, 512), (512, 512), (512, 2048), (1024, 2048), (2048, 512), (2048, 1024)]   # channels in, out
ROWS = 27


def _layer(ctx, x, w, shift, cin, cout):
    from webdnn_b200.lib import ConvDesc
    y = ctx.empty_tensor([ROWS, cout])
    d = ConvDesc(batch=3, ch_in=cin, in_h=3, in_w=3, ch_out=cout, k_h=1, k_w=1, out_h=3, out_w=3, stride_h=1, stride_w=1,
                 pad_t=0, pad_l=0, dil_h=1, dil_w=1, group=1, relu=0)
    ctx.conv2d(d, x, w, None, shift, None, y)
    return y


def test_few_rows_with_fresh_weights(cuda_context):
    """The layers of a small map, one behind the other: cold weights put a cluster's CTAs far apart, and its barrier has to
    hold until the last of them has read its tensor memory.  First results against second ones, bit for bit, and both
    against fp64."""
    from webdnn_b200.backend import CPUTensor
    ctx = cuda_context
    rng, nr = random.Random(3), np.random.default_rng(0)
    sets = [([(nr.standard_normal((co, ci, 1, 1)) / np.sqrt(ci)).astype(np.float32) for ci, co in LAYERS],
             [nr.standard_normal(co).astype(np.float32) for _, co in LAYERS]) for _ in range(3)]
    xs = {ci: nr.standard_normal((ROWS, ci)).astype(np.float32) for ci in (512, 1024, 2048)}
    put = lambda a: ctx.move_tensor(CPUTensor.from_array(a))  # noqa: E731
    want = [[xs[ci].astype(np.float64) @ w[i][:, :, 0, 0].T.astype(np.float64) + s[i] for i, (ci, _) in enumerate(LAYERS)] for w, s in sets]
    dev_x = {ci: put(a) for ci, a in xs.items()}
    for _ in range(700):
        k, order = rng.randrange(3), [rng.randrange(len(LAYERS)) for _ in range(8)]
        kept, first = [], []
        for i in order:
            (ci, co), raw, shift = LAYERS[i], put(sets[k][0][i]), put(sets[k][1][i])
            w = ctx.empty_tensor([co, 1, 1, ci])
            ctx._call("wdc_pack_conv_weight", c_void_p(raw.ptr), c_void_p(w.ptr), co, ci, 1, 1)
            ctx.declare_constant(w)
            first.append(_layer(ctx, dev_x[ci], w, shift, ci, co))
            kept.append((raw, shift, w))
        second = [_layer(ctx, dev_x[LAYERS[i][0]], w, shift, *LAYERS[i]) for i, (_, shift, w) in zip(order, kept)]
        for i, a, b in zip(order, first, second):
            got = a.get_data().reshape(ROWS, -1)
            assert np.abs(got - want[k][i]).max() <= 1e-5 * np.abs(want[k][i]).max()
            assert np.array_equal(got.reshape(-1).view(np.uint32), b.get_data().view(np.uint32))
        for t in (*first, *second, *(t for ts in kept for t in ts)):
            t.dispose()
    for t in dev_x.values():
        t.dispose()
