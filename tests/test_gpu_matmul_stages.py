"""Products of two activations (csrc/gemm_tc_direct.cu) where its K loop and its output can go wrong: fewer K blocks than stages,
segments of one block, both groups of loaders with and without a last block, more tiles than SMs, columns that allow 16-, 8-
and 4-byte accesses."""
import numpy as np
import pytest

from util import run_cuda, single_op_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 70, 132])                      # tiles of 64, 64 and 128 columns; odd, even, multiple of 4
@pytest.mark.parametrize("k", [5, 32, 33, 64, 96, 128, 129, 160, 161, 192, 256, 289, 321])
@pytest.mark.parametrize("batch,m", [(1, 40), (2, 129), (80, 130)])  # a few tiles; more than the SMs take at once
def test_matmul(cuda_context, batch, m, k, n):
    rng = np.random.default_rng(k + n)
    a, b = (rng.standard_normal(s).astype(np.float32) for s in ((batch, m, k), (batch, k, n)))
    (got,) = run_cuda(single_op_model("MatMul", {}, [a, b]), [a, b], cuda_context)
    want = a.astype(np.float64) @ b
    # 22 bits of every product (2^-21 of its size at worst), and the tensor core's fp32 accumulator loses up to 2^-23 of the
    # running sum at each of a segment's 48 steps (typically an eighth of that, and with changing signs of the addends)
    bound = (np.abs(a).astype(np.float64) @ np.abs(b)).max() * (2.0 ** -21 + 48 * 2.0 ** -23)
    assert np.abs(got - want).max() <= bound


@pytest.mark.parametrize("n", [33, 70, 132])                      # 4-, 8- and 16-byte stores, the last ones of a row cut off
@pytest.mark.parametrize("addend", ["none", "row", "column", "full"])
@pytest.mark.parametrize("relu", [0, 1])
@pytest.mark.parametrize("m,k", [(40, 33), (150, 161)])
def test_addend_and_relu(cuda_context, m, k, relu, addend, n):
    from ctypes import byref

    from webdnn_b200.backend import CPUTensor
    from webdnn_b200.lib import GemmDesc
    rng = np.random.default_rng(k + n)
    a, b = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (k, n)))
    c = rng.standard_normal({"none": (1, 1), "row": (1, n), "column": (m, 1), "full": (m, n)}[addend]).astype(np.float32)
    dev = [cuda_context.move_tensor(CPUTensor.from_array(t)) for t in (a, b, c)]
    y = cuda_context.empty_tensor([m, n])
    d = GemmDesc(batch=1, m=m, n=n, k=k, sab=0, sa0=k, sa1=1, sbb=0, sb0=n, sb1=1, sc0=c.shape[1] if c.shape[0] > 1 else 0,
                 sc1=int(c.shape[1] > 1), alpha=0.5, beta=-2.0, relu=relu)
    cuda_context._call("wdc_gemm", byref(d), dev[0].ptr, dev[1].ptr, None if addend == "none" else dev[2].ptr, y.ptr)
    want = 0.5 * (a.astype(np.float64) @ b) - (0 if addend == "none" else 2 * c.astype(np.float64))
    want = np.maximum(want, 0) if relu else want
    bound = (np.abs(a).astype(np.float64) @ np.abs(b)).max() * (2.0 ** -21 + 48 * 2.0 ** -23) + 2e-6
    assert np.abs(y.get_data().reshape(m, n) - want).max() <= bound
    for t in dev + [y]:
        t.dispose()
