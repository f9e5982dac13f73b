"""Products outside the prepared-weight tensor-core kernel: few rows, two activations, the LSTM recurrence."""
from ctypes import byref

import numpy as np
import pytest

from oracle import ref_runner

from util import max_err_rel_linf, run_cuda, single_op_model

pytestmark = pytest.mark.gpu


def _gemm(ctx, a, b, c=None, alpha=1.0, beta=0.0, relu=0, trans_a=False, trans_b=False):
    """wdc_gemm on [batch, m, k] x [batch, k, n]; trans_*: the operand is stored transposed."""
    from webdnn_b200.backend import CPUTensor
    from webdnn_b200.lib import GemmDesc
    batch, m, k = a.shape
    n = b.shape[2]
    put = lambda x: ctx.move_tensor(CPUTensor.from_array(np.ascontiguousarray(x)))  # noqa: E731
    da = put(a.transpose(0, 2, 1) if trans_a else a)
    db = put(b.transpose(0, 2, 1) if trans_b else b)
    dc = put(c) if c is not None else None
    y = ctx.empty_tensor([batch, m, n])
    d = GemmDesc(batch=batch, m=m, n=n, k=k, sab=m * k, sa0=1 if trans_a else k, sa1=m if trans_a else 1,
                 sbb=k * n, sb0=1 if trans_b else n, sb1=k if trans_b else 1,
                 sc0=n if c is not None and c.ndim == 2 else 0, sc1=1, alpha=alpha, beta=beta, relu=relu)
    ctx.gemm(d, da, db, dc, y)
    got = y.get_data().reshape(batch, m, n)
    for t in (da, db, dc, y):
        if t is not None:
            t.dispose()
    return got


def _want(a, b, c=None, alpha=1.0, beta=0.0, relu=0):
    y = alpha * np.matmul(a.astype(np.float64), b.astype(np.float64))
    if c is not None:
        y = y + beta * c
    return np.maximum(y, 0) if relu else y


# rows around the kernels' row counts (1, 2, 4, 8 and their multiples), K around one load per lane and warp
@pytest.mark.parametrize("m", [1, 2, 3, 5, 8, 9, 31])
@pytest.mark.parametrize("n,k,batch", [(1, 1, 1), (10, 512, 1), (33, 127, 3), (1000, 2048, 1), (130, 1028, 2), (7, 36, 1)])
@pytest.mark.parametrize("trans_b", [False, True])
def test_few_rows(cuda_context, m, n, k, batch, trans_b):
    rng = np.random.default_rng(m * 1000 + n)
    a, b = (rng.standard_normal(s).astype(np.float32) for s in ((batch, m, k), (batch, k, n)))
    c = rng.standard_normal(n).astype(np.float32)
    got = _gemm(cuda_context, a, b, c, 0.5, 2.0, 1, trans_b=trans_b)
    assert max_err_rel_linf(got, _want(a, b, c, 0.5, 2.0, 1)) <= 2e-6


# edges of the 128-row tile, of the three tile widths, of a K block (32), a TMEM segment (128) and the two stages
@pytest.mark.parametrize("batch,m,n,k", [(3, 32, 17, 1), (1, 129, 33, 31), (2, 128, 64, 32), (5, 127, 65, 33), (2, 40, 129, 128),
                                         (2, 300, 260, 129), (1, 64, 50, 161), (2, 96, 128, 256), (1, 1, 1, 5), (64, 257, 130, 67),
                                         (8, 850, 850, 32), (8, 850, 32, 850), (40, 130, 257, 1000)])
@pytest.mark.parametrize("trans_a,trans_b", [(False, False), (True, True), (False, True)])
def test_two_activations(cuda_context, batch, m, n, k, trans_a, trans_b):
    rng = np.random.default_rng(m + n + k)
    a, b = (rng.standard_normal(s).astype(np.float32) for s in ((batch, m, k), (batch, k, n)))
    got = _gemm(cuda_context, a, b, trans_a=trans_a, trans_b=trans_b)
    assert max_err_rel_linf(got, _want(a, b)) <= 2e-6


def test_two_activations_addend_and_non_finite(cuda_context):
    rng = np.random.default_rng(3)
    a, b = (rng.standard_normal(s).astype(np.float32) for s in ((2, 200, 45), (2, 45, 150)))
    c = rng.standard_normal((200, 150)).astype(np.float32)
    got = _gemm(cuda_context, a, b, c, -1.5, 0.5, 1)
    assert max_err_rel_linf(got, _want(a, b, c, -1.5, 0.5, 1)) <= 2e-6
    a[0, 3, 7], a[1, 150, 2], b[1, 11, 140] = np.inf, np.nan, 3.4e38
    a[1, :, 11] = 1e-3
    got = _gemm(cuda_context, a, b)
    with np.errstate(invalid="ignore"):
        want = _want(a, b)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    m = np.isfinite(want)
    assert np.array_equal(got[~m & ~np.isnan(want)], want[~m & ~np.isnan(want)].astype(np.float32))
    assert np.all(np.abs(got[m] - want[m]) <= 1e-5 * np.maximum(np.abs(want[m]), 1.0))


# hidden sizes around the 32 units of a CTA or a cluster, inside one cluster (up to 512) and across clusters (up to 768, their K
# slices), batches around an MMA's columns, the spread over clusters, and more rows than one launch takes; 3 steps, 28 and
# 800 units leave both kernels' range
@pytest.mark.parametrize("seq,batch,inp,hidden,state", [
    (3, 3, 8, 32, False), (4, 1, 4, 32, False), (5, 2, 12, 28, True), (6, 3, 32, 36, True), (17, 16, 40, 64, False), (5, 17, 12, 100, True), (9, 96, 64, 216, True),
    (23, 5, 100, 344, False), (12, 64, 256, 512, True), (6, 70, 32, 512, False), (5, 33, 36, 516, True), (7, 96, 48, 768, True),
    (4, 130, 32, 764, False), (3, 9, 32, 800, True), (128, 1, 80, 256, False)])
def test_lstm_recurrence(cuda_context, seq, batch, inp, hidden, state):
    rng = np.random.default_rng(seq * batch)
    lim = 1 / np.sqrt(hidden)
    uni = lambda *s: rng.uniform(-lim, lim, s).astype(np.float32)  # noqa: E731
    ins = [rng.standard_normal((seq, batch, inp)).astype(np.float32), uni(1, 4 * hidden, inp), uni(1, 4 * hidden, hidden),
           uni(1, 8 * hidden)]
    ctx = cuda_context
    if not state:
        model = single_op_model("LSTM", {"hidden_size": hidden}, ins, n_out=3, n_graph_inputs=1)
        want = ref_runner.run_model(model, ins[:1])
        got = run_cuda(model, ins[:1], ctx)
    else:
        from oracle import ops
        from webdnn_b200.backend import CPUTensor
        h0, c0 = (rng.uniform(-1, 1, (1, batch, hidden)).astype(np.float32) for _ in range(2))
        want = ops.lstm(*ins, h0, c0)
        dev = [ctx.move_tensor(CPUTensor.from_array(x)) for x in (*ins, h0, c0)]
        outs = [ctx.empty_tensor(s) for s in ((seq, 1, batch, hidden), (1, batch, hidden), (1, batch, hidden))]
        ctx._call("wdc_lstm", *(t.ptr for t in dev + outs), seq, batch, inp, hidden)
        got = [o.get_data().reshape(o.dims) for o in outs]
        for t in dev + outs:
            t.dispose()
    for g, w in zip(got, want):
        assert max_err_rel_linf(g, np.asarray(w).reshape(g.shape)) <= 1e-5


# edges of the small kernel: rows of a tile and of its shares, columns of both tile widths, K blocks per CTA of a cluster,
# more segments than accumulators, short last K blocks of a tap, strides and padding; it takes declared constants only
@pytest.mark.parametrize("n,cin,cout,size,k,stride,pad,res", [
    (1, 32, 32, (1, 1), 1, 1, 0, False), (1, 64, 36, (1, 127), 1, 1, 0, True), (1, 256, 64, (3, 43), 1, 1, 0, True),
    (1, 512, 132, (7, 7), 3, 1, 1, True), (2, 100, 68, (9, 9), 3, 2, 1, False), (1, 1024, 256, (14, 14), 1, 1, 0, False),
    (1, 36, 2048, (10, 10), 1, 1, 0, True), (1, 64, 256, (56, 56), 1, 1, 0, True), (1, 2048, 512, (5, 5), 1, 1, 0, False),
    (3, 128, 128, (28, 28), 3, 1, 1, False), (1, 2304, 64, (8, 16), 1, 1, 0, False)])
@pytest.mark.parametrize("precision", ["tf32x3", "tf32x1"])
def test_small_outputs(cuda_context, n, cin, cout, size, k, stride, pad, res, precision):
    from oracle import ops
    from webdnn_b200.backend import CPUTensor
    from webdnn_b200.lib import ConvDesc
    ctx = cuda_context
    rng = np.random.default_rng(cin + cout)
    x = rng.standard_normal((n, cin, *size)).astype(np.float32)
    w = (rng.standard_normal((cout, cin, k, k)) * np.sqrt(2.0 / (cin * k * k))).astype(np.float32)
    scale, shift = rng.uniform(0.5, 1.5, cout).astype(np.float32), rng.uniform(-1, 1, cout).astype(np.float32)
    oh, ow = ((s + 2 * pad - k) // stride + 1 for s in size)
    r = rng.standard_normal((n, cout, oh, ow)).astype(np.float32)
    want = ops.conv2d(x, w, None, (stride, stride), (pad,) * 4).astype(np.float64) * scale[:, None, None] + shift[:, None, None]
    want = np.maximum(want + r, 0) if res else want
    put = lambda a: ctx.move_tensor(CPUTensor.from_array(np.ascontiguousarray(a)))  # noqa: E731
    dx, dr = ctx.channels_last(put(x)), ctx.channels_last(put(r))
    dw, dsc, dsh = put(w.transpose(0, 2, 3, 1)), put(scale), put(shift)
    ctx.declare_constant(dw)
    ctx.declare_constant(dsc)
    y = ctx.empty_tensor([n, cout, oh, ow], layout="nhwc")
    d = ConvDesc(batch=n, ch_in=cin, in_h=size[0], in_w=size[1], ch_out=cout, k_h=k, k_w=k, out_h=oh, out_w=ow, stride_h=stride,
                 stride_w=stride, pad_t=pad, pad_l=pad, dil_h=1, dil_w=1, group=1, relu=int(res))
    ctx.set_precision(precision)
    try:
        for split_k in (1, 0):      # clusters of ranges, and one CTA per tile
            ctx.set_option("split_k", split_k)
            for _ in range(2):      # the first call splits the weights; the read waits, so the second loads them early
                ctx.conv2d(d, dx, dw, dsc, dsh, dr if res else None, y)
                got = y.get_data().reshape(want.shape)
                assert max_err_rel_linf(got, want) <= (5e-6 if precision == "tf32x3" else 3e-3)
    finally:
        ctx.set_option("split_k", 1)
        ctx.set_precision("tf32x3")
    for t in (dx, dr, dw, dsc, dsh, y):
        t.dispose()


# maps (32 to a CTA) and pixels (8 warps) around their multiples, and more maps than one round of CTAs
@pytest.mark.parametrize("batch,ch,area", [(1, 1, 1), (1, 31, 7), (3, 33, 8), (2, 64, 49), (5, 7, 130), (40, 1030, 9)])
def test_channels_last_average(cuda_context, batch, ch, area):
    from webdnn_b200.backend import CPUTensor
    x = np.random.default_rng(ch).standard_normal((batch, area, ch)).astype(np.float32)
    dx, y = cuda_context.move_tensor(CPUTensor.from_array(x)), cuda_context.empty_tensor([batch, ch])
    cuda_context._call("wdc_global_avgpool", dx.ptr, y.ptr, batch, ch, area, area * ch, 1, ch)
    assert max_err_rel_linf(y.get_data().reshape(batch, ch), x.astype(np.float64).mean(axis=1)) <= 1e-6
    dx.dispose()
    y.dispose()


# the last row of a pair missing, both sizes of CTA, more rows than one round of CTAs, rows held and re-read
@pytest.mark.parametrize("rows", [1, 2, 625, 4737, 40001])
@pytest.mark.parametrize("length", [36, 256, 300])
def test_layernorm_row_counts(cuda_context, rows, length):
    from oracle import ops
    rng = np.random.default_rng(rows)
    x = (rng.standard_normal((rows, length)) * 3 + 1).astype(np.float32)
    gamma, beta = rng.uniform(0.5, 1.5, length).astype(np.float32), rng.standard_normal(length).astype(np.float32)
    model = single_op_model("LayerNormalization", {"axis": -1, "epsilon": 1e-5}, [x, gamma, beta], opset=17)
    (got,) = run_cuda(model, [x, gamma, beta], cuda_context)
    assert max_err_rel_linf(got, ops.layernorm_chain(x, gamma, beta, 1e-5)) <= 5e-6


# clusters of 2, 4 and 8 CTAs per query tile: ranges of chunks of unequal length, a ragged last chunk and last rows
@pytest.mark.parametrize("batch,heads,tq,tk,dh", [(1, 3, 130, 257, 32), (1, 8, 625, 625, 32), (1, 8, 100, 625, 32),
                                                  (3, 1, 17, 256, 32), (1, 4, 300, 450, 64), (1, 2, 100, 640, 64)])
def test_attention_shared_by_a_cluster(cuda_context, batch, heads, tq, tk, dh):
    from ctypes import c_void_p

    from webdnn_b200.backend import CPUTensor
    from webdnn_b200.lib import AttentionDesc
    rng = np.random.default_rng(tq + tk)
    w = heads * dh
    q, k, v = (2 * rng.standard_normal((batch, t, w)).astype(np.float32) for t in (tq, tk, tk))
    qh, kh, vh = (x.reshape(batch, -1, heads, dh).transpose(0, 2, 1, 3).astype(np.float64) for x in (q, k, v))
    s = qh @ kh.transpose(0, 1, 3, 2) * dh ** -0.5
    p = np.exp(s - s.max(-1, keepdims=True))
    want = (p / p.sum(-1, keepdims=True) @ vh).transpose(0, 2, 1, 3).reshape(batch, tq, w)
    put = lambda a: cuda_context.move_tensor(CPUTensor.from_array(a))  # noqa: E731
    dq, dk, dv, y = put(q), put(k), put(v), cuda_context.empty_tensor([batch, tq, w])
    d = AttentionDesc(batch=batch, heads=heads, tq=tq, tk=tk, dh=dh, q_sb=tq * w, q_sh=dh, q_st=w, k_sb=tk * w, k_sh=dh,
                      k_st=w, v_sb=tk * w, v_sh=dh, v_st=w, y_sb=tq * w, y_sh=dh, y_st=w, scale=dh ** -0.5)
    cuda_context._call("wdc_attention", byref(d), *(c_void_p(t.ptr) for t in (dq, dk, dv, y)))
    assert max_err_rel_linf(y.get_data().reshape(want.shape), want) <= 1e-5
    for t in (dq, dk, dv, y):
        t.dispose()
