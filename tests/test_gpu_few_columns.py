"""Products whose rows are no multiple of four columns, by the small tensor-core kernel (one CTA a tile, and clusters) and past it."""
import numpy as np
import pytest

from util import run_cuda, single_op_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("m,k,n", [(32, 256, 1), (33, 512, 10), (64, 260, 15), (64, 512, 17), (200, 64, 33), (130, 128, 35), (64, 36, 5),
                                   (64, 1024, 62), (2048, 512, 10), (40000, 64, 3), (100, 1000, 3), (31, 512, 10)])
def test_few_columns(cuda_context, m, k, n, bias):
    rng = np.random.default_rng(m + k + n)
    a, b = rng.standard_normal((m, k)).astype(np.float32), rng.standard_normal((n, k)).astype(np.float32)
    c = rng.standard_normal(n).astype(np.float32)
    model = single_op_model("Gemm", dict(transB=1, alpha=0.5), [a, b] + ([c] if bias else []), n_graph_inputs=1)
    (got,) = run_cuda(model, [a], cuda_context)
    want = 0.5 * (a.astype(np.float64) @ b.T) + (c if bias else 0)
    # fp32 sums of k terms, or 22 bits of every product and the accumulator of at most 48 steps a segment
    bound = 0.5 * (np.abs(a).astype(np.float64) @ np.abs(b.T)).max() * (2.0 ** -21 + 48 * 2.0 ** -23) + 1e-6
    assert np.abs(got - want).max() <= bound
