"""The recurrence inside one cluster (csrc/lstm_local.cu): hidden sizes at the edges of its blocks of 32 units and of what
tensor memory holds, batches at the edges of its groups of 8 rows and past what one round of clusters takes, initial states
of any magnitude."""
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
