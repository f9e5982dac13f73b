"""Kernels that a rule on sizes chooses between: each of them where the rule would not, against the other, bit for bit where
the order of the additions is the same."""
from ctypes import byref, c_void_p

import numpy as np
import pytest

from util import max_err_rel_linf

pytestmark = pytest.mark.gpu


def _put(ctx, a):
    from webdnn_b200.backend import CPUTensor
    return ctx.move_tensor(CPUTensor.from_array(np.ascontiguousarray(a)))


def _conv(ctx, x, w, shift, res, pad, small_tile):
    """x NHWC, w KRSC, on the device; the result and the kernel that computed it (see wdc_stats)."""
    from webdnn_b200.lib import ConvDesc
    n, h, wd, cin = x.dims
    cout, k = w.dims[0], w.dims[1]
    oh, ow = h + 2 * pad - k + 1, wd + 2 * pad - k + 1
    y = ctx.empty_tensor([n, oh, ow, cout])
    d = ConvDesc(batch=n, ch_in=cin, in_h=h, in_w=wd, ch_out=cout, k_h=k, k_w=k, out_h=oh, out_w=ow, stride_h=1, stride_w=1,
                 pad_t=pad, pad_l=pad, dil_h=1, dil_w=1, group=1, relu=int(res is not None))
    ctx.set_option("small_tile", small_tile)
    try:
        ctx.conv2d(d, x, w, None, shift, res, y)
    finally:
        ctx.set_option("small_tile", 0)
    got = y.get_data().copy()
    y.dispose()
    return got.view(np.uint32), ctx.stats(device_memory=True)["last_contraction"]


# [rows, columns, K blocks] that tc_igemm_kernel takes whole (in 1 .. 8 and more segments) or cuts into 2 .. 8 ranges: every
# cluster size of both tile widths; a last K block, a last row tile and a last column tile that are not full
@pytest.mark.parametrize("m,n,kblocks", [
    (76, 4, 1), (50, 36, 5), (44, 4, 8), (37, 4, 14), (32, 8, 19), (36, 4, 20), (66, 4, 24), (70, 4, 30), (3488, 4, 32), (129, 68, 32),
    (8261, 4, 54), (6105, 4, 41), (4061, 4, 36), (3333, 4, 36), (2780, 4, 36), (46, 4, 33), (33, 4, 40), (49, 100, 144),
    (9841, 40, 1), (9884, 36, 9), (10109, 40, 12), (3136, 64, 18), (625, 256, 64), (320, 512, 144)])
@pytest.mark.parametrize("ragged", [0, 12])
@pytest.mark.parametrize("precision", ["tf32x3", "tf32x1"])
def test_small_outputs_are_the_same_bits(cuda_context, m, n, kblocks, ragged, precision):
    ctx = cuda_context
    rng = np.random.default_rng(m + n)
    k = 32 * kblocks - ragged
    x, w = rng.standard_normal((1, 1, m, k)).astype(np.float32), rng.standard_normal((n, 1, 1, k)).astype(np.float32)
    dx, dw = _put(ctx, x), _put(ctx, w)
    shift, res = _put(ctx, rng.standard_normal(n).astype(np.float32)), _put(ctx, rng.standard_normal((m, n)).astype(np.float32))
    ctx.declare_constant(dw)
    ctx.set_precision(precision)
    seen = set()
    try:
        for split_k in (1, 0):
            ctx.set_option("split_k", split_k)
            for s, r in ((None, None), (shift, None), (shift, res)):
                want, kernel = _conv(ctx, dx, dw, s, r, 0, -1)
                assert kernel == 0
                for tile in (32, 64):
                    got, kernel = _conv(ctx, dx, dw, s, r, 0, tile)
                    seen.add(kernel // 10)
                    assert np.array_equal(got, want), (split_k, tile, kernel)
    finally:
        ctx.set_option("split_k", 1)
        ctx.set_precision("tf32x3")
    assert any(s > 320 for s in seen) or kblocks < 8 or (m, n) == (9841, 40), seen
    for t in (dx, dw, shift, res):
        t.dispose()


# rows that are no multiple of four columns: tiles are not cut; one segment to eight of them and more; the addend comes last
@pytest.mark.parametrize("m,n,k", [(76, 1, 32), (50, 35, 148), (64, 10, 512), (129, 67, 1024), (200, 33, 64), (2048, 10, 512),
                                   (45, 62, 768), (66, 5, 640), (90, 6, 896), (33, 2, 1280), (4000, 63, 256)])
@pytest.mark.parametrize("precision", ["tf32x3", "tf32x1"])
def test_rows_of_any_length_are_the_same_bits(cuda_context, m, n, k, precision):
    from webdnn_b200.lib import GemmDesc
    ctx = cuda_context
    rng = np.random.default_rng(m + n)
    da, db = (_put(ctx, rng.standard_normal(s).astype(np.float32)) for s in ((m, k), (k, n)))
    shift, full = _put(ctx, rng.standard_normal(n).astype(np.float32)), _put(ctx, rng.standard_normal((m, (n + 3) // 4 * 4)).astype(np.float32))
    y = ctx.empty_tensor([m, n])
    ctx.declare_constant(db)
    ctx.set_precision(precision)
    seen = set()

    def product(c, beta, tile):
        d = GemmDesc(batch=1, m=m, n=n, k=k, sab=0, sa0=k, sa1=1, sbb=0, sb0=n, sb1=1, sc0=0 if c is shift else full.dims[1],
                     sc1=1, alpha=1.5, beta=beta, relu=int(beta != 1))
        ctx.set_option("small_tile", tile)
        ctx.gemm(d, da, db, c, y)
        return y.get_data().copy().view(np.uint32), ctx.stats(device_memory=True)["last_contraction"]

    try:
        for split_k in (1, 0):
            ctx.set_option("split_k", split_k)
            for c, beta in ((None, 1.0), (shift, 1.0), (shift, 0.7), (full, 0.7)):
                want, kernel = product(c, beta, -1)
                assert kernel == 0
                for tile in (32, 64):
                    got, kernel = product(c, beta, tile)
                    seen.add(kernel // 10)
                    assert np.array_equal(got, want), (split_k, beta, tile, kernel)
    finally:
        ctx.set_option("small_tile", 0)
        ctx.set_option("split_k", 1)
        ctx.set_precision("tf32x3")
    assert any(s % 10 == 1 for s in seen) and (any(s % 10 > 1 for s in seen) or not 256 <= k <= 1024), seen
    for t in (da, db, shift, full, y):
        t.dispose()


def test_every_cluster_size_is_taken(cuda_context):
    """The shapes above do reach every variant of the small kernel."""
    ctx = cuda_context
    seen = set()
    for m, n, kblocks in [(76, 4, 1), (44, 4, 8), (37, 4, 14), (32, 8, 19), (36, 4, 20), (66, 4, 24), (70, 4, 30), (3488, 4, 32),
                          (9841, 40, 1), (8261, 4, 54), (6105, 4, 41), (4061, 4, 36), (3333, 4, 36), (2780, 4, 36), (46, 4, 33),
                          (33, 4, 40)]:
        dx, dw = ctx.empty_tensor([1, 1, m, 32 * kblocks]), ctx.empty_tensor([n, 1, 1, 32 * kblocks])
        for t in (dx, dw):
            ctx._call("wdc_fill_u32", c_void_p(t.ptr), 0, t.length)
        ctx.declare_constant(dw)
        for tile in (32, 64):
            seen.add(_conv(ctx, dx, dw, None, None, 0, tile)[1] // 10)
        dx.dispose()
        dw.dispose()
    assert {10 * t + c for t in (32, 64) for c in range(1, 9)} <= seen, seen


# filter taps around the rotated start, short last blocks of a tap, padding
@pytest.mark.parametrize("n,cin,cout,size,k", [(1, 64, 64, (56, 56), 3), (2, 100, 68, (9, 9), 3), (1, 36, 132, (20, 21), 3), (1, 512, 132, (7, 7), 3),
                                               (5, 40, 36, (30, 17), 5), (3, 128, 128, (28, 28), 3)])
def test_small_convolutions_are_the_same_bits(cuda_context, n, cin, cout, size, k):
    ctx = cuda_context
    rng = np.random.default_rng(cin + cout)
    dx = _put(ctx, rng.standard_normal((n, *size, cin)).astype(np.float32))
    dw = _put(ctx, rng.standard_normal((cout, k, k, cin)).astype(np.float32))
    shift = _put(ctx, rng.standard_normal(cout).astype(np.float32))
    ctx.declare_constant(dw)
    want, kernel = _conv(ctx, dx, dw, shift, None, k // 2, -1)
    assert kernel == 0
    for tile in (32, 64, 32):      # the reads in between wait: later calls load their weights early
        got, kernel = _conv(ctx, dx, dw, shift, None, k // 2, tile)
        assert np.array_equal(got, want), (tile, kernel)
    for t in (dx, dw, shift):
        t.dispose()


# products side by side: few rows, one and several waves of tiles of the small kernel, the whole-SM kernel
@pytest.mark.parametrize("m", [5, 100, 625, 800, 5000])
@pytest.mark.parametrize("k,columns,count", [(256, 256, 2), (256, 256, 6), (36, 100, 3), (1024, 64, 2)])
def test_products_side_by_side_are_the_same_bits(cuda_context, m, k, columns, count):
    from webdnn_b200.lib import GemmDesc
    ctx = cuda_context
    rng = np.random.default_rng(m + k)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((k, columns * count)).astype(np.float32)
    c = rng.standard_normal(columns * count).astype(np.float32)
    da = _put(ctx, a)

    def product(b, c, columns):
        db, dc, n = _put(ctx, b), _put(ctx, c), b.shape[1]
        ctx.declare_constant(db)
        y = ctx.empty_tensor([m, n])
        ctx.gemm(GemmDesc(batch=1, m=m, n=n, k=k, sab=0, sa0=k, sa1=1, sbb=0, sb0=n, sb1=1, sc0=0, sc1=1, alpha=1.0, beta=1.0, relu=0),
                 da, db, dc, y, columns)
        got = y.get_data().reshape(m, n).copy()
        for t in (db, dc, y):
            t.dispose()
        return got

    got = product(b, c, columns)
    assert max_err_rel_linf(got, a.astype(np.float64) @ b + c) <= 2e-6
    for i in range(count):
        at = slice(i * columns, (i + 1) * columns)
        assert np.array_equal(got[:, at].view(np.uint32), product(b[:, at], c[at], 0).view(np.uint32)), i
    da.dispose()


# CTAs per query tile, each of them; with all chunks of a CTA's keys scored -inf (a sum of products that overflows)
@pytest.mark.parametrize("tq,tk,dh", [(130, 520, 32), (17, 2000, 32), (100, 640, 64)])
@pytest.mark.parametrize("overflow", [False, True])
def test_every_attention_cluster(cuda_context, tq, tk, dh, overflow):
    from webdnn_b200.lib import AttentionDesc
    ctx = cuda_context
    rng = np.random.default_rng(tq + tk)
    q, k, v = (2 * rng.standard_normal((1, t, dh)).astype(np.float32) for t in (tq, tk, tk))
    if overflow:
        q[:, :, 0], k[:, tk // 2:, 0], k[:, :tk // 2, 0] = 1e20, -1e20, 0.0
    with np.errstate(over="ignore"):
        s = (np.einsum("btc,bsc->bts", q.astype(np.float64), k) * dh ** -0.5).astype(np.float32).astype(np.float64)
    p = np.exp(s - s.max(-1, keepdims=True))
    want = p / p.sum(-1, keepdims=True) @ v
    dq, dk, dv, y = _put(ctx, q), _put(ctx, k), _put(ctx, v), ctx.empty_tensor([1, tq, dh])
    d = AttentionDesc(batch=1, heads=1, tq=tq, tk=tk, dh=dh, q_sb=tq * dh, q_sh=dh, q_st=dh, k_sb=tk * dh, k_sh=dh, k_st=dh,
                      v_sb=tk * dh, v_sh=dh, v_st=dh, y_sb=tq * dh, y_sh=dh, y_st=dh, scale=dh ** -0.5)
    try:
        for cs in (1, 2, 4, 8):
            ctx.set_option("attention_cluster", cs)
            ctx._call("wdc_attention", byref(d), *(c_void_p(t.ptr) for t in (dq, dk, dv, y)))
            got = y.get_data().reshape(want.shape)
            assert ctx.stats(device_memory=True)["last_attention_cluster"] == cs
            assert max_err_rel_linf(got, want) <= 1e-5, cs
    finally:
        ctx.set_option("attention_cluster", 0)
    for t in (dq, dk, dv, y):
        t.dispose()
