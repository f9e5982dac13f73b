"""What repeats a run for the host (tapes, graphs with their transfers) and what moves its data."""
import ctypes
from ctypes import c_void_p

import numpy as np
import pytest

from webdnn_b200 import onnx_io, operator_table, zoo

pytestmark = pytest.mark.gpu


def _load(ctx, model, **options):
    from webdnn_b200.runner import load
    return load(model, backend_order=["cuda", "cpu"], backend_options={"cuda": {"context": ctx, **options}})


def _model(nodes, inputs, outputs, inits=()):
    value = lambda v: onnx_io.ValueInfo(v[0], v[2] if len(v) > 2 else onnx_io.FLOAT, list(v[1]))  # noqa: E731
    g = onnx_io.Graph("g", nodes, [onnx_io.make_tensor(n, a) for n, a in inits], [value(v) for v in inputs],
                      [value(v) for v in outputs])
    return onnx_io.Model(g, opset_import=[("", 13)])


def _cpu(a):
    from webdnn_b200.backend import CPUTensor
    return CPUTensor.from_array(np.ascontiguousarray(a))


def _bits(a):
    return np.ascontiguousarray(a).reshape(-1).view(np.uint32)


def _two_outputs(rows):
    """[rows, 40] and [rows, 40] -> their product's rectified halves, and an int32 index per row."""
    make = onnx_io.make_node
    rng = np.random.default_rng(rows)
    return _model([make("MatMul", ["a", "w"], ["m"], name="m"), make("Add", ["m", "b"], ["s"], name="s"),
                   make("Relu", ["s"], ["y"], name="r"), make("ArgMax", ["s"], ["i"], name="i", axis=-1, keepdims=0)],
                  [("a", [rows, 40]), ("b", [rows, 64])], [("y", [rows, 64]), ("i", [rows], onnx_io.INT32)],
                  [("w", rng.standard_normal((40, 64)).astype(np.float32))])


def _tape_of(runner, on_device=False):
    return [t for (dev, _), t in runner._tapes.items() if dev == on_device]


# around what a kernel moves (128 KB), what helper threads share (256 KB), a chunk (512 KB) and the ring (16 MB)
@pytest.mark.parametrize("nbytes", [1, 3, 4, 4096, (128 << 10) - 4, 128 << 10, (128 << 10) + 4, (256 << 10) - 1, 256 << 10, (256 << 10) + 1,
                                    (512 << 10) - 1, 512 << 10, (512 << 10) + 1, (16 << 20) - 1, 16 << 20, (16 << 20) + 1, 40_000_001])
@pytest.mark.parametrize("pinned", [False, True])
def test_round_trip(cuda_context, nbytes, pinned):
    ctx = cuda_context
    data = np.random.default_rng(nbytes).integers(0, 256, nbytes, dtype=np.uint8)
    host = ctx.pinned_array((nbytes,), np.uint8) if pinned else np.empty(nbytes, np.uint8)
    back = ctx.pinned_array((nbytes,), np.uint8) if pinned else np.empty(nbytes, np.uint8)
    ptr = ctx._alloc(nbytes + 16)
    for shift in (0, 4):     # the device side aligned to 16 bytes and not
        host[:] = data
        back[:] = 0
        ctx._call("wdc_upload", c_void_p(ptr + shift), host.ctypes.data_as(c_void_p), nbytes)
        if not pinned:
            host[:] = 0      # a pageable source may be reused at once
        ctx._call("wdc_download", back.ctypes.data_as(c_void_p), c_void_p(ptr + shift), nbytes)
        assert np.array_equal(back, data)
    ctx._free(ptr)
    if pinned:
        for a in (host, back):
            ctx._call("wdc_host_free", a.ctypes.data_as(c_void_p))


def test_uploads_do_not_wait_for_kernels(cuda_context):
    import time
    ctx = cuda_context
    big = ctx.empty_tensor([1 << 28])
    dst = ctx._alloc(4 << 20)
    pinned, pageable = ctx.pinned_array((1 << 20,), np.uint8), np.ones(4 << 20, np.uint8)
    for host in (pinned, pageable[:4096], pageable):
        ctx._call("wdc_upload", c_void_p(dst), host.ctypes.data_as(c_void_p), host.nbytes)   # (the ring exists from here on)
        ctx.sync()
        for _ in range(400):
            ctx._call("wdc_fill_u32", c_void_p(big.ptr), ctypes.c_uint32(1), big.length)
        t0 = time.perf_counter()
        ctx._call("wdc_upload", c_void_p(dst), host.ctypes.data_as(c_void_p), host.nbytes)
        t1 = time.perf_counter()
        ctx.sync()
        t2 = time.perf_counter()
        assert t2 - t0 > 0.01 and t1 - t0 < 0.3 * (t2 - t0), (host.nbytes, t1 - t0, t2 - t0)
    ctx._call("wdc_host_free", pinned.ctypes.data_as(c_void_p))
    ctx._free(dst)
    big.dispose()


@pytest.mark.parametrize("rows", [40, 5000])      # results within and beyond what a kernel moves
@pytest.mark.parametrize("on_device", [False, True])
def test_tape_with_new_inputs(cuda_context, rows, on_device):
    ctx = cuda_context
    runner = _load(ctx, _two_outputs(rows))
    rng = np.random.default_rng(1)
    in_use = None
    for i in range(6):
        a, b = rng.standard_normal((rows, 40)).astype(np.float32), rng.standard_normal((rows, 64)).astype(np.float32)
        where = [(0, 0), (1, 1), (0, 1), (1, 0)][i % 4]         # host and device inputs in one call
        ins = [ctx.move_tensor(_cpu(x)) if d else _cpu(x) for x, d in zip((a, b), where)]
        got = runner.run(ins, outputs_on_device=on_device)
        assert runner.nodes_on("cpu") == [] and len(runner.node_backends) >= 2
        want = runner._run_nodes([_cpu(a), _cpu(b)])
        for g, w in zip(got, want):
            assert g.backend == ("cuda" if on_device else "cpu") and g.data_type == w.data_type and list(g.dims) == list(w.dims)
            assert np.array_equal(_bits(g.get_data()), _bits(w.numpy()))
        for t in (*ins, *got):
            if t.backend == "cuda":
                t.dispose()
        if i >= 1:
            (tape,) = _tape_of(runner, on_device)
            assert tape is not None
            now = ctx.stats()["bytes_in_use"]
            assert in_use in (None, now)
            in_use = now
    runner.dispose()


def test_taped_runs_that_nobody_waited_for(cuda_context):
    """Inputs of later calls are brought into memory that the calls in flight have just given back."""
    ctx = cuda_context
    model = zoo.resnet50(48, 64, 32, (1, 1, 1, 1), 64, softmax=False)
    runner = _load(ctx, model)
    xs = [np.random.default_rng(i).standard_normal((48, 3, 64, 64)).astype(np.float32) for i in range(12)]
    want = [runner.run([_cpu(x)])[0].numpy().copy() for x in xs]
    for _ in range(3):
        runner.run([_cpu(xs[0])], outputs_on_device=True)[0].dispose()
    assert _tape_of(runner, True) != [None]
    for _ in range(5):
        queued = [runner.run([_cpu(x)], outputs_on_device=True)[0] for x in xs]
        for q, w in zip(queued, want):
            assert np.array_equal(_bits(q.get_data()), _bits(w))
            q.dispose()
        pending = []
        for x, w in [*zip(xs, want), (None, None), (None, None)]:      # three in flight
            if x is not None:
                pending.append((runner.run([_cpu(x)], wait=False), w))
            if len(pending) == 3 or x is None:
                p, expected = pending.pop(0)
                assert np.array_equal(_bits(p.result()[0].numpy()), _bits(expected))
    runner.dispose()


def test_what_a_tape_must_not_keep(cuda_context):
    """A custom operator runs every time, placement and precision may change, results may be inputs."""
    from webdnn_b200.operators.cuda import OperatorImpl
    ctx = cuda_context
    calls = []

    class Counted(OperatorImpl):
        def __init__(self):
            super().__init__("cuda")

        def run(self, context, inputs, n_outputs):
            calls.append(1)
            y = context.empty_tensor(inputs[0].dims)
            context._call("wdc_fill_u32", c_void_p(y.ptr), ctypes.c_uint32(len(calls)), y.length)
            return [y]

    operator_table.register_operators([operator_table.OperatorEntry("Counted", 1, None, "cuda", Counted)])
    x = np.ones((40, 8), np.float32)
    runner = _load(ctx, _model([onnx_io.make_node("Counted", ["x"], ["y"], name="c")], [("x", [40, 8])], [("y", [40, 8])]))
    for i in range(5):
        (y,) = runner.run([_cpu(x)])
        assert len(calls) == i + 1 and np.all(_bits(y.numpy()) == i + 1)
    runner.dispose()

    make = onnx_io.make_node
    runner = _load(ctx, _model([make("Relu", ["x"], ["r"], name="r"), make("Reshape", ["r", "s"], ["y"], name="y")],
                               [("x", [40, 8])], [("y", [80, 4]), ("x", [40, 8])], [("s", np.array([80, 4], np.int64))]))
    for i in range(4):      # a result that is an input
        y, same = runner.run([_cpu(x * (i - 2))], outputs_on_device=True)
        assert np.array_equal(y.get_data(), np.maximum(x * (i - 2), 0).reshape(-1)) and np.array_equal(same.get_data(), (x * (i - 2)).reshape(-1))
    runner.dispose()

    runner = _load(ctx, _two_outputs(70))
    ins = [_cpu(np.random.default_rng(i).standard_normal((70, n)).astype(np.float32)) for i, n in ((0, 40), (1, 64))]
    first = [runner.run(ins)[0].numpy().copy() for _ in range(3)][-1]
    assert _tape_of(runner) != [None]
    ctx.set_precision("tf32x1")
    try:
        rough = runner.run(ins)[0].numpy().copy()
        assert np.array_equal(_bits(rough), _bits(runner._run_nodes(ins)[0].numpy()))
    finally:
        ctx.set_precision("tf32x3")
    assert np.array_equal(_bits(runner.run(ins)[0].numpy()), _bits(first)) and not np.array_equal(rough, first)
    runner.force_operator_backend_order["r"] = ["cpu"]
    if any(n[0] == "r" for n in runner.node_backends):
        with pytest.raises(RuntimeError):     # no cpu implementation of Relu: asked for, so tried
            runner.run(ins)
    runner.dispose()


def test_one_tensor_as_two_inputs(cuda_context):
    ctx = cuda_context
    runner = _load(ctx, _model([onnx_io.make_node("Sub", ["a", "b"], ["y"], name="s")], [("a", [50, 8]), ("b", [50, 8])], [("y", [50, 8])]))
    for i in range(5):
        a, b = (np.random.default_rng(10 * i + j).standard_normal((50, 8)).astype(np.float32) for j in (0, 1))
        da, db = ctx.move_tensor(_cpu(a)), ctx.move_tensor(_cpu(b))
        for x, y, want in ((da, da, a - a), (da, db, a - b), (db, da, b - a), (_cpu(a), _cpu(a), a - a)):
            assert np.array_equal(runner.run([x, y])[0].numpy(), want)
        da.dispose()
        db.dispose()
    runner.dispose()


def test_more_signatures_than_tapes(cuda_context):
    ctx = cuda_context
    make = onnx_io.make_node
    runner = _load(ctx, _model([make("Relu", ["x"], ["y"], name="r")], [("x", ["n", 8])], [("y", ["n", 8])]))
    xs = [np.random.default_rng(n).standard_normal((n, 8)).astype(np.float32) for n in range(33, 33 + runner.MAX_TAPES + 6)]
    for _ in range(3):
        for x in xs:
            assert np.array_equal(runner.run([_cpu(x)])[0].numpy(), np.maximum(x, 0))
    assert len(runner._tapes) == runner.MAX_TAPES
    runner.dispose()


def test_allocation_failing_in_the_middle_of_a_tape():
    from webdnn_b200.backend import CudaBackendError, WebDNNCPUContext, WebDNNCudaContext
    ctx = WebDNNCudaContext(WebDNNCPUContext(), arena_bytes=64 << 20)
    ctx.initialize()
    make = onnx_io.make_node
    runner = _load(ctx, _model([make("Relu", ["x"], ["r"], name="r"), make("Exp", ["r"], ["e"], name="e"),
                                make("Sqrt", ["e"], ["y"], name="y")], [("x", [1 << 20])], [("y", [1 << 20])]))
    x = _cpu(np.linspace(-1, 1, 1 << 20).astype(np.float32))
    want = [runner.run([x])[0].numpy().copy() for _ in range(3)][0]
    assert _tape_of(runner) != [None]
    before = ctx.stats()["bytes_in_use"]
    hog = [ctx.empty_tensor([1 << 20]) for _ in range(14)]      # 56 of 64 MB: the input and one more fit
    full = ctx.stats()["bytes_in_use"]
    with pytest.raises(CudaBackendError):
        runner.run([x])
    for t in hog:
        t.dispose()
    assert full - before == 56 << 20
    for _ in range(4):
        assert np.array_equal(_bits(runner.run([x])[0].numpy()), _bits(want))
    runner.dispose()
    ctx.close()


# small and large inputs and results on one recorded graph, from the host and from the device in turn
@pytest.mark.parametrize("rows,width", [(8, 64), (8, 8192), (32, 2048)])
def test_graph_with_its_transfers(cuda_context, rows, width):
    ctx = cuda_context
    make = onnx_io.make_node
    model = _model([make("Relu", ["x"], ["y"], name="r"), make("Add", ["y", "z"], ["s"], name="s"),
                    make("ArgMax", ["s"], ["i"], name="i", axis=-1, keepdims=0)],
                   [("x", [rows, width]), ("z", [rows, width])], [("y", [rows, width]), ("s", [rows, width]), ("i", [rows], onnx_io.INT32)])
    runner = _load(ctx, model, graphReplay=True)
    rng = np.random.default_rng(width)
    for i in range(8):
        x, z = (rng.standard_normal((rows, width)).astype(np.float32) for _ in range(2))
        ins = [ctx.move_tensor(_cpu(a)) if i & bit and i > 2 else _cpu(a) for a, bit in ((x, 1), (z, 2))]
        y, s, idx = runner.run(ins)
        assert np.array_equal(y.numpy(), np.maximum(x, 0)) and np.array_equal(s.numpy(), np.maximum(x, 0) + z)
        assert np.array_equal(idx.numpy(), np.argmax(np.maximum(x, 0) + z, -1))
        p = runner.run([_cpu(x), _cpu(z)], wait=False)
        assert np.array_equal(p.result()[1].numpy(), np.maximum(x, 0) + z)
    assert runner.graph_replays > 6
    runner.dispose()


def test_recurrence_inside_a_graph(cuda_context):
    """The recurrence inside one cluster, a launch of clusters that are independent: recorded and replayed like the others."""
    runner = _load(cuda_context, zoo.lstm(20, 5, 24, 96), graphReplay=True)
    rng = np.random.default_rng(0)
    for _ in range(4):
        x = rng.standard_normal((20, 5, 24)).astype(np.float32)
        got = runner.run([_cpu(x)])
        want = runner._run_nodes([_cpu(x)])
        assert all(np.array_equal(_bits(g.numpy()), _bits(w.numpy())) for g, w in zip(got, want))
    assert runner.graph_replays >= 2
    runner.dispose()


# clusters that exchange h, and single CTAs: cooperative launches
@pytest.mark.parametrize("hidden", [544, 800])
def test_cooperative_recurrences_inside_a_graph(cuda_context, hidden):
    runner = _load(cuda_context, zoo.lstm(20, 5, 24, hidden), graphReplay=True)
    rng = np.random.default_rng(0)
    for _ in range(4):
        x = rng.standard_normal((20, 5, 24)).astype(np.float32)
        got, want = runner.run([_cpu(x)]), runner._run_nodes([_cpu(x)])
        assert all(np.array_equal(_bits(g.numpy()), _bits(w.numpy())) for g, w in zip(got, want))
    assert runner.graph_replays >= 2
    runner.dispose()


# an infinite weight, and one that rounding would make infinite; an infinite initial state: gates saturate as in fp32
@pytest.mark.parametrize("batch,hidden", [(1, 32), (5, 100), (33, 256)])
@pytest.mark.parametrize("where", ["R", "R_large", "h0"])
def test_recurrence_with_infinities(cuda_context, batch, hidden, where):
    ctx = cuda_context
    seq, inp = 6, 8
    rng = np.random.default_rng(hidden)
    u = lambda *s: rng.uniform(-0.3, 0.3, s).astype(np.float32)  # noqa: E731
    x, w, r, b, h0, c0 = u(seq, batch, inp), u(4 * hidden, inp), u(4 * hidden, hidden), u(8 * hidden), u(batch, hidden), u(batch, hidden)
    if where == "R":
        r[hidden + 3, 5], r[3, hidden - 1] = np.inf, -np.inf        # the output and the input gate of unit 3
    elif where == "R_large":
        r[hidden + 3, 5] = np.float32(3.4028e38)
    else:
        h0[batch - 1, 7] = np.inf
    dev = [ctx.move_tensor(_cpu(a)) for a in (x, w, r, b, h0, c0)]
    outs = [ctx.empty_tensor(s) for s in ((seq, batch, hidden), (batch, hidden), (batch, hidden))]
    ctx._call("wdc_lstm", *(t.ptr for t in dev + outs), seq, batch, inp, hidden)
    got = [o.get_data().reshape(o.dims) for o in outs]
    sig = lambda v: 0.5 * (np.tanh(0.5 * v) + 1)  # noqa: E731
    h, c, ys = h0.astype(np.float64), c0.astype(np.float64), []
    with np.errstate(all="ignore"):
        for t in range(seq):
            g = x[t].astype(np.float64) @ w.T + h @ r.T.astype(np.float64) + b[:4 * hidden] + b[4 * hidden:]
            i, o, f, cc = np.split(g, 4, axis=1)
            c = sig(f) * c + sig(i) * np.tanh(cc)
            h = sig(o) * np.tanh(c)
            ys.append(h)
    for a, e in zip(got, (np.stack(ys), h, c)):
        assert np.array_equal(np.isnan(a), np.isnan(e))
        assert np.all(np.abs(np.nan_to_num(a) - np.nan_to_num(e)) <= 1e-5)
    assert np.isfinite(got[0]).any()
    for t in dev + outs:
        t.dispose()


def test_first_results_in_used_memory(cuda_context):
    """A model loaded into memory that other work has just given back gives the same bits at every call."""
    ctx = cuda_context
    rng = np.random.default_rng(0)
    models = [zoo.resnet50(2, 64, 32, (1, 1, 1, 1), 64, softmax=False), zoo.resnet50(40, 64, 32, (1, 1, 1, 1), 64, softmax=False),
              zoo.detr(batch=1, size=128, d=64, heads=2, enc_layers=1, dec_layers=1, ffn=128, queries=9, classes=7, width=16, blocks=(1, 1, 1, 1)),
              zoo.mlp(33), zoo.lstm(9, 3, 16, 64)]
    for i in range(60):
        model = models[i % len(models)]
        x = rng.standard_normal(model.graph.input[0].shape).astype(np.float32)
        big = [ctx.empty_tensor([8 << 20]) for _ in range(4)]
        for t in big:      # a quiet NaN, large values: whatever is read without having been written shows
            ctx._call("wdc_fill_u32", c_void_p(t.ptr), ctypes.c_uint32([0x7fc00000, 0x7e000000, 0xc4fa0001][i % 3]), t.length)
            t.dispose()
        runner = _load(ctx, model)
        results = [[o.numpy().copy() for o in runner.run([_cpu(x)])] for _ in range(3)]
        for later in results[1:]:
            assert all(np.array_equal(_bits(a), _bits(b)) for a, b in zip(results[0], later))
        runner.dispose()


def test_copying_threads_of_all_contexts_stay_below_the_cpus():
    """Large transfers of several contexts in a process that is bound to three CPUs."""
    import os
    import subprocess
    import sys
    code = """
import os
os.sched_setaffinity(0, set(sorted(os.sched_getaffinity(0))[:3]))
import numpy as np
from webdnn_b200.backend import CPUTensor, WebDNNCPUContext, WebDNNCudaContext
contexts = []
for i in range(3):
    ctx = WebDNNCudaContext(WebDNNCPUContext())
    ctx.initialize()
    ctx.move_tensor(CPUTensor.from_array(np.ones(64, np.float32))).get_data()     # (whatever the driver starts for itself)
    contexts.append(ctx)
def threads():
    return len(os.listdir("/proc/self/task"))
before = threads()
data = np.random.default_rng(0).standard_normal(4 << 20).astype(np.float32)
for ctx in contexts:
    t = ctx.move_tensor(CPUTensor.from_array(data))
    assert np.array_equal(t.get_data(), data)
assert 0 < threads() - before <= 2, (before, threads())
for ctx in contexts:
    ctx.close()
ctx = WebDNNCudaContext(WebDNNCPUContext())
ctx.initialize()
ctx.move_tensor(CPUTensor.from_array(np.ones(64, np.float32))).get_data()
before = threads()
assert np.array_equal(ctx.move_tensor(CPUTensor.from_array(data)).get_data(), data)
assert 0 < threads() - before <= 2, (before, threads())      # given back by the contexts that are gone
ctx.close()
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    done = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
