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
