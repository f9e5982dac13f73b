"""The recurrence inside one cluster (csrc/lstm_local.cu): hidden sizes at the edges of its blocks of 32 units and of what
tensor memory holds, batches at the edges of its groups of 8 rows and past what one round of clusters takes, initial states
and weights of any magnitude, alone and side by side."""
import numpy as np
import pytest

from webdnn_b200.backend import CPUTensor

pytestmark = pytest.mark.gpu


def _reference(x, w, r, b, h, c):
    sig = lambda v: 0.5 * (np.tanh(0.5 * v) + 1)  # noqa: E731
    x, w, r, b, h, c = (a.astype(np.float64) for a in (x, w, r, b, h, c))
    hidden, ys = r.shape[1], []
    for t in range(x.shape[0]):
        i, o, f, g = np.split(x[t] @ w.T + h @ r.T + b[:4 * hidden] + b[4 * hidden:], 4, axis=1)
        c = sig(f) * c + sig(i) * np.tanh(g)
        h = sig(o) * np.tanh(c)
        ys.append(h)
    return np.stack(ys), h, c


@pytest.mark.parametrize("seq,batch,hidden,state", [
    (4, 1, 32, None), (5, 1185, 32, None),                                   # one CTA a cluster; more groups than CTAs
    (9, 3, 36, 1.0), (7, 17, 100, 1.0), (6, 40, 252, 1.0),                   # units past the last block's, odd clusters
    (20, 15, 256, None), (5, 121, 256, 1.0),                                 # one row a cluster; one past 8 rows
    (6, 1, 480, 1.0), (6, 90, 484, 1.0),                                     # the last sizes with 15 CTAs and the first with 16
    (6, 56, 512, None), (5, 57, 512, 1.0), (5, 113, 512, 1.0), (4, 169, 512, None), (4, 225, 512, 1.0), (4, 500, 512, None),
    (6, 10, 512, 1e6), (6, 10, 64, 1e-6),                                    # rows of h0 have scales of their own
    (5, 4, 516, 1.0),                                                        # the first size that lstm_cluster.cu keeps
])
def test_recurrence(cuda_context, seq, batch, hidden, state):
    ctx = cuda_context
    rng = np.random.default_rng(hidden + batch)
    lim, inp = 1 / np.sqrt(hidden), 12
    u = lambda *s: rng.uniform(-lim, lim, s).astype(np.float32)  # noqa: E731
    x = rng.standard_normal((seq, batch, inp)).astype(np.float32)
    w, r, b = u(4 * hidden, inp), u(4 * hidden, hidden), u(8 * hidden)
    r[1::7] *= np.float32(1e-3)                                              # rows of R too
    h0, c0 = np.zeros((batch, hidden), np.float32), np.zeros((batch, hidden), np.float32)
    if state is not None:
        h0 = (rng.standard_normal((batch, hidden)) * state ** rng.uniform(0, 1, (batch, 1))).astype(np.float32)
        c0 = rng.standard_normal((batch, hidden)).astype(np.float32)
    dev = [ctx.move_tensor(CPUTensor.from_array(a)) for a in (x, w, r, b, h0, c0)]
    outs = [ctx.empty_tensor(s) for s in ((seq, batch, hidden), (batch, hidden), (batch, hidden))]
    ptrs = [t.ptr for t in dev]
    if state is None:
        ptrs[4] = ptrs[5] = None
    results = []
    for _ in range(2):
        ctx._call("wdc_lstm", *ptrs, *(o.ptr for o in outs), seq, batch, inp, hidden)
        results.append([o.get_data().reshape(o.dims).copy() for o in outs])
    # A pre-activation's error: the recurrent sum's, 2^-21 (22 bits of every product, as in the projection) times the sum
    # of its terms' magnitudes (lim / 2 * |h| * hidden, |h| at most that of h0 in the first step), typically its root;
    # the gates pass on at most a quarter to all of it, and steps that forget little add up.
    size = np.abs(h0).max() if state is not None else 1.0
    tol = 2.0 ** -21 * max(size, 1.0) * lim * np.sqrt(hidden) * 4 + 4e-6
    for got, want in zip(results[0], _reference(x, w, r, b, h0, c0)):
        assert np.abs(got - want).max() <= tol * max(1.0, np.abs(want).max())
    for one, two in zip(*results):
        assert np.array_equal(one.view(np.uint32), two.view(np.uint32))
    for t in dev + outs:
        t.dispose()


def test_gates_are_no_further_off_than_by_tanhf(cuda_context):
    """Sigmoid and tanh of the one-cluster kernel (sequences of 4 steps and more) and of the path for shorter ones, which calls
    tanhf, against float64 on the same pre-activations: over magnitudes from 1e-5 to 40, by ranges.  Until the last step
    the forget gate is open and the candidate 0, so that the cell is 1 or 0; then units 0 .. 15 give c = sigmoid(x) and the
    others c = tanh(x), and h = tanh(c) with the output gate open."""
    from ctypes import byref

    from webdnn_b200.lib import GemmDesc
    ctx = cuda_context
    rng = np.random.default_rng(7)
    batch, inp, hidden = 40000, 4, 32
    x = np.exp(rng.uniform(np.log(1e-2), np.log(40), batch)).astype(np.float32)
    x[:200] = np.nextafter(np.float32(1), np.float32(rng.choice([0, 2], 200))) * np.float32(1 + 1e-6) ** rng.integers(-9, 9, 200)
    x[200:400] = np.float32(0.7) * np.float32(1 + 1e-6) ** rng.integers(-9, 9, 200)   # either side of where the forms change
    x[400], x[401] = 3e38, np.nan
    w = np.zeros((4, hidden, inp), np.float32)
    sign = np.where(np.arange(16) % 2 == 0, 1, -1) * 2.0 ** -(np.arange(16) % 8 // 2 * 3)
    sign[15] *= 16 * 512                                           # (3e38 times this is infinite)
    w[2, :16, 0], w[3, 16:, 0] = sign, sign
    w[2, :16, 1] = w[0, 16:, 2] = w[1, :, 2] = 1                   # gates held open by 100
    c0 = np.zeros((batch, hidden), np.float32)
    c0[:, :16] = 1
    errors = {}
    for seq in (4, 3):
        xs = np.zeros((seq, batch, inp), np.float32)
        xs[-1, :, 0], xs[:-1, :, 1], xs[:, :, 2] = x, 100, 100
        dev = [ctx.move_tensor(CPUTensor.from_array(a)) for a in (xs, w.reshape(4 * hidden, inp), np.zeros((4 * hidden, hidden), np.float32), c0)]
        outs = [ctx.empty_tensor(s) for s in ((seq, batch, hidden), (batch, hidden), (batch, hidden))]
        ctx._call("wdc_lstm", dev[0].ptr, dev[1].ptr, dev[2].ptr, None, None, dev[3].ptr, *(o.ptr for o in outs), seq, batch, inp, hidden)
        h, c = (o.get_data().reshape(o.dims).copy() for o in outs[1:])
        p = ctx.empty_tensor([seq * batch, 4 * hidden])            # the projection, as wdc_lstm computes it
        d = GemmDesc(batch=1, m=seq * batch, n=4 * hidden, k=inp, sab=0, sa0=inp, sa1=1, sbb=0, sb0=1, sb1=inp, sc0=0, sc1=0,
                     alpha=1.0, beta=0.0, relu=0)
        ctx._call("wdc_gemm", byref(d), dev[0].ptr, dev[1].ptr, None, p.ptr)
        pre = p.get_data().reshape(seq, batch, 4, hidden)[-1].astype(np.float64)
        for t in dev + outs + [p]:
            t.dispose()
        at = np.concatenate([pre[:, 2, :16], pre[:, 3, 16:]], axis=1)
        nan = np.isnan(at)
        assert nan[401].all() and np.isnan(c[401]).all() and np.isnan(h[401]).all() and not np.isnan(c[~nan]).any()
        assert np.isinf(at[400]).any()
        at, c, h = np.delete(at, 401, 0), np.delete(c, 401, 0).astype(np.float64), np.delete(h, 401, 0)
        with np.errstate(over="ignore"):
            want_s, want_t = 1 / (1 + np.exp(-at[:, :16])), np.tanh(at[:, 16:])
        parts = [("sigmoid", np.abs(at[:, :16]), np.abs(c[:, :16] - want_s)),
                 ("tanh", np.abs(at[:, 16:]), np.abs(c[:, 16:] - want_t) / np.abs(want_t)),
                 ("tanh", np.abs(c), np.abs(h - np.tanh(c)) / np.maximum(np.abs(np.tanh(c)), 1e-30))]
        for n, (name, mag, err) in enumerate(parts):
            for lo, hi in ((1e-5, .25), (.25, .65), (.65, 1), (1, 2), (2, 4), (4, np.inf)):
                e = err[(mag >= lo) & (mag <= hi)] * 2.0 ** 24
                if e.size > 2000:
                    errors.setdefault((n, name, lo), []).append((e.max(), np.sqrt(np.mean(e ** 2))))
    assert len(errors) >= 14
    # the largest errors over all floats in units of 2^-24, by tanhf 0.6, 0.9, 0.95, 1.4, 1.1, 0.8 and 1.9, 3.4, 2.95, 1.8, 1.1, 0.55
    bounds = {"sigmoid": dict(zip((1e-5, .25, .65, 1, 2, 4), (.55, .61, .69, 1.3, .91, .6))),
              "tanh": dict(zip((1e-5, .25, .65, 1, 2, 4), (1.04, 1.24, 2.9, 1.7, .87, .53)))}
    for (n, name, lo), ((top, rms), (top_tanhf, rms_tanhf)) in errors.items():
        assert top <= bounds[name][lo] and top_tanhf <= 3.4, (n, name, lo, top, top_tanhf)
        # (two samples of a range differ by a share of a percent)
        assert rms <= 1.01 * rms_tanhf, (n, name, lo, rms, rms_tanhf)


# Rms errors that the TF32 parts and K slices of csrc/lstm_cluster.cu have at these sizes (random signs, one sign): the
# one-cluster kernel is no further off.
@pytest.mark.parametrize("hidden,mixed,one_sign", [(32, 1.09e-7, 0.91e-7), (64, 1.18e-7, 0.96e-7), (128, 1.60e-7, 1.31e-7), (256, 2.59e-7, 2.42e-7),
                                                   (384, 3.65e-7, 3.66e-7), (480, 4.62e-7, 5.11e-7), (512, 9.14e-7, 1.19e-6)])
@pytest.mark.parametrize("batch", [8, 200])
def test_sums_are_no_further_off_than_tf32_parts(cuda_context, batch, hidden, mixed, one_sign):
    """The first step's y = o tanh(i tanh(s)) with pre-activations so small that its relative error is that of the sum s (and of
    the gates, 2^-24 each)."""
    ctx = cuda_context
    for positive, bound in ((False, mixed), (True, one_sign)):
        off = size = 0.0
        for seed in range(6 if batch < 100 else 2):
            rng = np.random.default_rng(seed + hidden)
            r = (rng.standard_normal((4 * hidden, hidden)) * 1e-4).astype(np.float32)
            h0 = rng.uniform(-1, 1, (batch, hidden)).astype(np.float32)
            if positive:
                r, h0 = np.abs(r), np.abs(h0)
            dev = [ctx.move_tensor(CPUTensor.from_array(a)) for a in (np.zeros((4, batch, 4), np.float32), np.zeros((4 * hidden, 4), np.float32), r, h0)]
            outs = [ctx.empty_tensor(s) for s in ((4, batch, hidden), (batch, hidden), (batch, hidden))]
            ctx._call("wdc_lstm", dev[0].ptr, dev[1].ptr, dev[2].ptr, None, dev[3].ptr, None, *(o.ptr for o in outs), 4, batch, 4, hidden)
            got = outs[0].get_data().reshape(4, batch, hidden)[0].astype(np.float64)
            i, o, f, g = np.split(h0.astype(np.float64) @ r.T.astype(np.float64), 4, axis=1)
            want = np.tanh(np.tanh(g) / (1 + np.exp(-i))) / (1 + np.exp(-o))
            off, size = off + np.sum((got - want) ** 2), size + np.sum(want ** 2)
            for t in dev + outs:
                t.dispose()
        # (5 %: samples of a few thousand values in the smallest case)
        assert np.sqrt(off / size) <= 1.05 * bound, (positive, np.sqrt(off / size), bound)


@pytest.mark.parametrize("hidden,batch", [(36, 3), (64, 8), (256, 130), (416, 260), (480, 20), (512, 57), (512, 130)])
@pytest.mark.parametrize("kind", ["weight 1e6", "weight 1e8", "weight 1e10", "weight 3e38", "dead units", "wide weights", "few small", "h0 and weights", "tiny inputs"])
def test_ranges_inside_rows(cuda_context, kind, batch, hidden):
    """Elements of R and h0 that are far below the largest of their row count as much as where they are alone: a large weight
    whose unit's output is 0 (its gate is shut), magnitudes spread over 12 decades in every row or in a few places, states
    spread likewise, outputs of 1e-8."""
    ctx = cuda_context
    rng = np.random.default_rng(hidden + batch)
    seq, inp, lim = 6, 12, 1 / np.sqrt(hidden)
    u = lambda *s: rng.uniform(-lim, lim, s).astype(np.float32)  # noqa: E731
    x, w, r, b = rng.standard_normal((seq, batch, inp)).astype(np.float32), u(4 * hidden, inp), u(4 * hidden, hidden), u(8 * hidden)
    h0 = c0 = np.zeros((batch, hidden), np.float32)
    if kind.startswith("weight"):
        r[:, 3] = float(kind.split()[1])
        r[hidden + 3], w[hidden + 3], b[hidden + 3], b[5 * hidden + 3] = 0, 0, -200, 0
    if kind in ("wide weights", "h0 and weights"):
        r *= (10.0 ** rng.uniform(-12, 0, r.shape)).astype(np.float32)
    if kind == "dead units":
        r[:, 1::2] *= np.float32(1e-11)
        x[2:4], b[:] = 0, 0                                          # (and sums that only they decide)
        r[::5, ::2] *= np.float32(1e-20)
    if kind == "few small":
        at = rng.random(r.shape) < 0.002
        r[at] *= np.float32(1e-11)
        r[:, -1] *= np.float32(1e-11)
    if kind == "h0 and weights":
        h0 = (rng.standard_normal((batch, hidden)) * 10.0 ** rng.uniform(-12, 2, (batch, hidden))).astype(np.float32)
        r[1::3, 0], h0[:, 0] = 1e8, 0                                # the small ones of both decide
        c0 = rng.standard_normal((batch, hidden)).astype(np.float32)
    if kind == "tiny inputs":
        x *= np.float32(1e-7)
        b[:] = 0
    dev = [ctx.move_tensor(CPUTensor.from_array(a)) for a in (x, w, r, b, h0, c0)]
    outs = [ctx.empty_tensor(s) for s in ((seq, batch, hidden), (batch, hidden), (batch, hidden))]
    ctx._call("wdc_lstm", *(t.ptr for t in dev), *(o.ptr for o in outs), seq, batch, inp, hidden)
    steps = 1 if kind == "h0 and weights" else seq                   # (a weight of 1e8 on h of 1 saturates the others)
    got = outs[0].get_data().reshape(seq, batch, hidden)[:steps]
    want = _reference(x, w, r, b, h0, c0)[0][:steps]
    # 22 bits of every product and the gates' 2^-23: 2e-7 to 5e-7 over the steps
    assert np.linalg.norm(got - want) <= 1e-6 * np.linalg.norm(want)
    for t in dev + outs:
        t.dispose()


@pytest.mark.parametrize("hidden,batch", [(64, 10), (512, 10), (320, 130)])
@pytest.mark.parametrize("state", [1e-30, 1e-6, 1.0, 1e6, 1e30])
def test_initial_states_of_any_magnitude(cuda_context, state, batch, hidden):
    """Rows of h0 have scales of their own: with R as much smaller as h0 is larger, a wrong one shows in the first step."""
    ctx = cuda_context
    rng = np.random.default_rng(hidden)
    r = (rng.standard_normal((4 * hidden, hidden)) / np.sqrt(hidden) / state).astype(np.float32)
    h0 = (rng.standard_normal((batch, hidden)) * state * 2.0 ** rng.uniform(-3, 1, (batch, 1))).astype(np.float32)
    x, w, b, c0 = np.zeros((4, batch, 4), np.float32), np.zeros((4 * hidden, 4), np.float32), np.zeros(8 * hidden, np.float32), np.zeros((batch, hidden), np.float32)
    dev = [ctx.move_tensor(CPUTensor.from_array(a)) for a in (x, w, r, h0)]
    outs = [ctx.empty_tensor(s) for s in ((4, batch, hidden), (batch, hidden), (batch, hidden))]
    ctx._call("wdc_lstm", dev[0].ptr, dev[1].ptr, dev[2].ptr, None, dev[3].ptr, None, *(o.ptr for o in outs), 4, batch, 4, hidden)
    got = outs[0].get_data().reshape(4, batch, hidden)[0]
    with np.errstate(over="ignore"):
        want = _reference(x[:1], w, r, b, h0, c0)[0][0]
    assert (np.abs(got - want).max(axis=1) <= 1e-6).all() and np.abs(want).max(axis=1).min() > 1e-2   # (zeros would not pass)
    for t in dev + outs:
        t.dispose()


# as tests/test_gpu_runs.py has it for smaller ones: the largest size inside one cluster, and sizes whose clusters exchange h
@pytest.mark.parametrize("batch,hidden", [(3, 512), (5, 516), (20, 768)])
@pytest.mark.parametrize("where", ["R", "R_large", "h0"])
def test_infinities_in_many_units(cuda_context, where, batch, hidden):
    ctx = cuda_context
    seq, inp, lim = 6, 8, 0.3 * np.sqrt(256 / hidden)            # (a step passes on no more of an error than at 256 units)
    rng = np.random.default_rng(hidden)
    u = lambda *s: rng.uniform(-lim, lim, s).astype(np.float32)  # noqa: E731
    x, w, r, b, h0, c0 = u(seq, batch, inp), u(4 * hidden, inp), u(4 * hidden, hidden), u(8 * hidden), u(batch, hidden), u(batch, hidden)
    if where == "h0":
        h0[batch - 1, 7] = np.inf
    else:
        r[hidden + 3, 5] = np.inf if where == "R" else np.float32(3.4028e38)
        r[3, hidden - 1] = -np.inf if where == "R" else r[3, hidden - 1]
    dev = [ctx.move_tensor(CPUTensor.from_array(a)) for a in (x, w, r, b, h0, c0)]
    outs = [ctx.empty_tensor(s) for s in ((seq, batch, hidden), (batch, hidden), (batch, hidden))]
    ctx._call("wdc_lstm", *(t.ptr for t in dev + outs), seq, batch, inp, hidden)
    with np.errstate(all="ignore"):
        wants = _reference(x, w, r, b, h0, c0)
    for got, want in zip((o.get_data().reshape(o.dims) for o in outs), wants):
        assert np.array_equal(np.isnan(got), np.isnan(want)) and np.isfinite(got).any()
        assert np.all(np.abs(np.nan_to_num(got) - np.nan_to_num(want)) <= 1e-5)
    for t in dev + outs:
        t.dispose()
