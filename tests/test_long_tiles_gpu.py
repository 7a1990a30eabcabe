"""The int8 projection of few rows at the sizes that reach its k tiles of every length."""
import numpy as np
import pytest

from denograd_b200.device import Tensor
from oracle import oracle as O
from tests.test_kernels_gpu import assert_reduction_close

pytestmark = pytest.mark.gpu


# eight K slices (few features), four, two and one; one tile and a piece of 16, whole tiles, and a last tile that some slices do not reach
@pytest.mark.parametrize("M", [2, 8, 9, 16, 17])
@pytest.mark.parametrize("N,K", [(40, 2064), (48, 4096), (33, 5136), (5936, 2064), (5952, 3072), (11856, 2064), (23680, 2064)])
def test_int8_projection_of_few_rows(dev, M, N, K):
    rng = np.random.default_rng(M + N + K)
    x, res = rng.standard_normal((M, K)).astype(np.float16), rng.standard_normal((M, N)).astype(np.float16)
    w, s = rng.integers(-127, 128, (N, K), dtype=np.int8), (rng.uniform(0.5, 1.5, N) * 2e-4).astype(np.float16)
    xt, wt, st, rt, y = Tensor(x, device=dev), Tensor(w, device=dev), Tensor(s, device=dev), Tensor(res, device=dev), Tensor.zeros((M + 1, N), "float16", dev)
    dev.call("jg_linear", y.ptr, xt.ptr, wt.ptr, st.ptr, 0, M, N, K)
    want = O.linear_w8(x, w, s)
    assert_reduction_close(y.numpy()[:M], want, max_ulp=1, max_frac=0.05, what="int8 linear")
    dev.call("jg_linear", y.ptr, xt.ptr, wt.ptr, st.ptr, rt.ptr, M, N, K)
    assert_reduction_close(y.numpy()[:M], (res.astype(np.float32) + want.astype(np.float32)).astype(np.float16), max_ulp=2, max_frac=0.05, what="int8 linear + residual")
    assert (y.numpy()[M:] == 0).all()
