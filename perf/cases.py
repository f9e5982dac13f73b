"""What a user of this framework runs, as measured cases.

A user loads an ONNX graph once (`webdnn_b200.runner.load`) and calls `Runner.run` for every input that arrives.  The
cases are the graphs this repository is benchmarked and tested on (`webdnn_b200/zoo.py`: an MLP, one fused convolution
layer, ResNet-50, an LSTM, a DETR-style detector) and the product of two activations out of the operator list of
`layer_bench.py`, each over the sizes such a graph is called with.  Everything is fp32, the one floating type of the
runtime; "tf32x1" is the reduced `precision` that `backendOptions.cuda` offers.

`io` says where a call's tensors are:
  "host"    CPU tensors in, CPU tensors out: one request, `runner.run(inputs)` as the reference's users write it
  "read"    inputs already on the GPU (a decoder or a copy stream put them there), results read by the host
  "device"  inputs and results stay on the GPU: the graph is one stage of a longer pipeline
"""
import functools
import math

import torch

from webdnn_b200 import onnx_io, zoo
from webdnn_b200.backend import CPUTensor, WebDNNCPUContext, WebDNNCudaContext
from webdnn_b200.runner import load


def listed():
    return [
        # one feature vector through a small classifier: launches, copies and host work are all there is
        dict(name="mlp_1", kind="mlp", batch=1, io="host"),
        # the first benchmark configuration: a mini-batch of host data
        dict(name="mlp_64", kind="mlp", batch=64, io="host"),
        # the second configuration: one 3x3 convolution layer with BatchNormalization and Relu, inside a GPU pipeline
        dict(name="conv_32x64x56", kind="conv", batch=32, ch=64, size=56, io="device"),
        # classification of a single image, the way the reference's demos call it
        dict(name="resnet50_1", kind="resnet", batch=1, size=224, precision="tf32x3", io="host"),
        # a few images of an uneven size at the reduced precision
        dict(name="resnet50_5_250_tf32x1", kind="resnet", batch=5, size=250, precision="tf32x1", io="read"),
        # a serving batch: one GPU's share of 256 images split over eight
        dict(name="resnet50_32", kind="resnet", batch=32, size=224, precision="tf32x3", io="read"),
        # the headline configuration
        dict(name="resnet50_256", kind="resnet", batch=256, size=224, precision="tf32x3", io="read"),
        # one short sequence of feature frames (speech, sensor data)
        dict(name="lstm_1", kind="lstm", seq=50, batch=1, input=80, hidden=256, io="host"),
        # the fourth configuration
        dict(name="lstm_64", kind="lstm", seq=128, batch=64, input=256, hidden=512, io="device"),
        # detection on a single image
        dict(name="detr_1", kind="detr", batch=1, size=800, io="host"),
        # detection on a batch
        dict(name="detr_8", kind="detr", batch=8, size=800, io="read"),
        # product of two activations with ragged sides (attention scores written out as MatMul)
        dict(name="matmul_8x850x32x850", kind="matmul", batch=8, m=850, k=32, n=850, io="device"),
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, spread evenly over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["mlp", "conv", "resnet", "lstm", "detr", "matmul"])
    if kind == "mlp":
        return dict(kind=kind, batch=_log(rng, 1, 2048), io="host")
    if kind == "conv":
        # channel counts are multiples of 4 (24, 36, 60, ... among them), up to twice the second configuration's work
        ch, size = 4 * _log(rng, 4, 128), _log(rng, 7, 112)
        most = max(1, min(64, int(2 * 32 * 64 * 64 * 56 * 56 / (ch * ch * size * size))))
        return dict(kind=kind, batch=_log(rng, 1, most), ch=ch, size=size, io="device")
    if kind == "resnet":
        size = rng.randint(128, 288)
        batch = _log(rng, 1, min(256, int(256 * 224 * 224 / (size * size))))
        precision = "tf32x1" if rng.random() < 0.2 else "tf32x3"
        return dict(kind=kind, batch=batch, size=size, precision=precision, io="host" if batch <= 2 else "read")
    if kind == "lstm":
        batch = _log(rng, 1, 96)
        return dict(kind=kind, seq=_log(rng, 16, 192), batch=batch, input=4 * _log(rng, 4, 128),
                    hidden=8 * _log(rng, 8, 96), io="host" if batch <= 2 else "device")
    if kind == "detr":
        size = rng.randint(320, 832)
        batch = _log(rng, 1, min(16, int(8 * 800 * 800 / (size * size))))
        return dict(kind=kind, batch=batch, size=size, io="host" if batch <= 2 else "read")
    return dict(kind=kind, batch=_log(rng, 1, 64), m=_log(rng, 16, 1024), k=_log(rng, 16, 1024),
                n=_log(rng, 16, 1024), io="device")


def _model(case):
    kind, b = case["kind"], case["batch"]
    if kind == "mlp":
        return zoo.mlp(b)
    if kind == "conv":
        return zoo.conv_bn_relu(b, case["ch"], case["size"])
    if kind == "resnet":
        # without the final Softmax: on random weights it is one-hot and would hide every difference
        return zoo.resnet50(b, case["size"], softmax=False)
    if kind == "lstm":
        return zoo.lstm(case["seq"], b, case["input"], case["hidden"])
    if kind == "detr":
        return zoo.detr(b, case["size"])
    node = onnx_io.make_node("MatMul", ["a", "b"], ["y"], name="matmul")
    value = lambda name, shape: onnx_io.ValueInfo(name, onnx_io.FLOAT, shape)  # noqa: E731
    graph = onnx_io.Graph("matmul", [node], [], [value(n, s) for n, s in zip("ab", _input_shapes(case))],
                          [value("y", [b, case["m"], case["n"]])])
    return onnx_io.Model(graph, opset_import=[("", 13)])


def _input_shapes(case):
    kind, b = case["kind"], case["batch"]
    if kind == "mlp":
        return [[b, 784]]
    if kind == "conv":
        return [[b, case["ch"], case["size"], case["size"]]]
    if kind == "lstm":
        return [[case["seq"], b, case["input"]]]
    if kind == "matmul":
        return [[b, case["m"], case["k"]], [b, case["k"], case["n"]]]
    return [[b, 3, case["size"], case["size"]]]


class _Program:
    """The loaded graph a program keeps for all of its calls: one context, one runner."""

    def __init__(self, case):
        self.context = WebDNNCudaContext(WebDNNCPUContext())
        self.context.initialize()
        self.runner = load(_model(case), backend_order=["cuda", "cpu"], backend_options={
            "cuda": {"context": self.context, "precision": case.get("precision", "tf32x3")}})

    def __del__(self):
        if hasattr(self, "runner"):
            self.runner.dispose()
        self.context.close()


@functools.lru_cache(maxsize=1)
def _program_of(items):
    return _Program(dict(items))


class _View:
    """A result that stays on the GPU, readable by torch in the dims of the graph, whatever its layout in memory."""

    def __init__(self, tensor, program):
        self.tensor, self.program = tensor, program
        strides = tensor.nchw_strides() if tensor.ndim == 4 else tensor.strides
        self.__cuda_array_interface__ = dict(shape=tuple(tensor.dims), strides=tuple(4 * s for s in strides),
                                             typestr="<f4", data=(tensor.ptr, False), version=2)


class _State:
    def __init__(self, program, io, inputs):
        self.program, self.io, self.inputs, self.results = program, io, inputs, []

    def release_results(self):
        for t in self.results:
            t.dispose()
        self.results = []

    def __del__(self):
        self.release_results()
        for t in self.inputs:
            t.dispose()


def prepare(case, seed):
    program = _program_of(tuple(sorted((k, v) for k, v in case.items() if k not in ("name", "io"))))
    g = torch.Generator(device="cuda").manual_seed(seed)
    inputs = []
    for shape in _input_shapes(case):
        # pixels and feature vectors of the MLP are U(0, 1), everything else N(0, 1), as in the benchmark configurations
        make = torch.rand if case["kind"] == "mlp" else torch.randn
        host = CPUTensor.from_array(make(shape, generator=g, device="cuda").cpu().numpy())
        inputs.append(host if case["io"] == "host" else program.context.move_tensor(host))
    return _State(program, case["io"], inputs)


def run(state):
    runner = state.program.runner
    if state.io != "device":
        return [t.numpy() for t in runner.run(state.inputs)]
    state.release_results()       # the previous call's results have been used
    state.results = runner.run(state.inputs, outputs_on_device=True)
    return [torch.as_tensor(_View(t, state.program), device="cuda") for t in state.results]


def _trunk_macs(size):
    """Multiply-adds of one image through the ResNet-50 trunk, its weight count, and the side of the last map."""
    half = lambda s: (s + 1) // 2  # noqa: E731
    side = half(size)
    macs, weights = side * side * 64 * 3 * 49, 64 * 3 * 49
    side, cin = half(side), 64
    for stage, blocks in enumerate((3, 4, 6, 3)):
        planes = 64 << stage
        for i in range(blocks):
            out = half(side) if i == 0 and stage > 0 else side
            for pixels, n in ((side * side, cin * planes), (out * out, 9 * planes * planes),
                              (out * out, planes * 4 * planes)) + (((out * out, cin * 4 * planes),) if i == 0 else ()):
                macs, weights = macs + pixels * n, weights + n
            side, cin = out, planes * 4
    return macs, weights, side


def work(case):
    kind, b = case["kind"], case["batch"]
    n_in = sum(math.prod(s) for s in _input_shapes(case))
    if kind == "mlp":
        macs, weights, n_out = b * (784 * 512 + 512 * 512 + 512 * 10), 784 * 512 + 512 * 512 + 512 * 10, b * 10
    elif kind == "conv":
        weights = 9 * case["ch"] * case["ch"]
        macs, n_out = b * case["size"] ** 2 * weights, n_in
    elif kind == "resnet":
        macs, weights, _ = _trunk_macs(case["size"])
        macs, weights, n_out = b * (macs + 2048 * 1000), weights + 2048 * 1000, b * 1000
    elif kind == "lstm":
        weights = 4 * case["hidden"] * (case["input"] + case["hidden"])
        macs, n_out = case["seq"] * b * weights, (case["seq"] + 2) * b * case["hidden"]
    elif kind == "matmul":
        weights, n_out = 0, b * case["m"] * case["n"]
        macs = n_out * case["k"]
    else:
        macs, weights, side = _trunk_macs(case["size"])
        t, d, q, ffn, layers = side * side, 256, 100, 2048, 6
        macs += t * 2048 * d
        macs += layers * (t * (4 * d * d + 2 * d * ffn) + 2 * t * t * d)                          # encoder
        macs += layers * (q * (6 * d * d + 2 * d * ffn) + t * 2 * d * d + 2 * q * d * (q + t))    # decoder
        macs += q * (d * 92 + 2 * d * d + d * 4)
        weights += 2048 * d + layers * (12 * d * d + 4 * d * ffn) + d * 92 + 2 * d * d + d * 4 + (t + q) * d
        macs, n_out = b * macs, b * q * 96
    return {"bytes": 4 * (n_in + weights + n_out), "flops": 2 * macs}


def tolerance(case):
    """fp32 everywhere (TF32 triples on the tensor cores, 22 bits of every product): one contraction agrees to about
    1e-6, and dozens of them in a row, whose rounding the following layers carry on, to some 1e-5.  With "tf32x1"
    every operand has 11 bits, 5e-4 a layer."""
    if case.get("precision") == "tf32x1":
        return {"rel": 1e-2}
    if case["kind"] in ("resnet", "detr"):
        return {"rel": 5e-5}
    return {"rel": 1e-5}
