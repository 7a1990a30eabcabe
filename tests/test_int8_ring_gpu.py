"""The int8 tensor-core projection repeated over matrices that come from HBM: every repeat has the same bits, and the right ones."""
import numpy as np
import pytest

from denograd_b200.device import Tensor
from oracle import oracle as O
from tests.test_kernels_gpu import assert_reduction_close

pytestmark = pytest.mark.gpu


# 33, 100 and 128 rows: rings whose converting groups take turns at a stage; 20 and 300: the others.  Few and many k-blocks
@pytest.mark.parametrize("M,N,K", [(33, 1024, 4096), (100, 1024, 8192), (128, 4096, 4096), (100, 6144, 1024), (20, 1024, 4096), (300, 1024, 4096)])
def test_repeats_are_right_and_bit_equal(dev, M, N, K):
    rng = np.random.default_rng(M + N + K)
    x, res = rng.standard_normal((M, K)).astype(np.float16), rng.standard_normal((M, N)).astype(np.float16)
    q = [rng.integers(-127, 128, (N, K), dtype=np.int8) for _ in range(2)]
    s = [(rng.uniform(0.5, 1.5, N) * 2e-4).astype(np.float16) for _ in range(2)]
    w = [(a.astype(np.float16) * b[:, None]).astype(np.float16).astype(np.float32) for a, b in zip(q, s)]
    xt, rt = Tensor(x, device=dev), Tensor(res, device=dev)
    # copies of the matrices, 160 MB and more, so that a repeat finds none of its own in L2
    wt = [[Tensor(a, device=dev) for a in q] for _ in range(max(2, 80_000_000 // (N * K)))]
    st = [Tensor(b, device=dev) for b in s]
    acc, up = x.astype(np.float32) @ w[0].T, x.astype(np.float32) @ w[1].T
    want = acc.astype(np.float16)
    cases = {"store": (lambda y, a: dev.call("jg_linear", y.ptr, xt.ptr, a[0].ptr, st[0].ptr, 0, M, N, K), want, 1, 0.08),
             "residual": (lambda y, a: dev.call("jg_linear", y.ptr, xt.ptr, a[0].ptr, st[0].ptr, rt.ptr, M, N, K),
                          (res.astype(np.float32) + want.astype(np.float32)).astype(np.float16), 2, 0.08),
             "swiglu": (lambda y, a: dev.call("jg_norm_swiglu", y.ptr, xt.ptr, 0, 1e-5, a[0].ptr, st[0].ptr, a[1].ptr, st[1].ptr, M, N, K),
                        O.swiglu(want, up.astype(np.float16)), 3, 0.12)}
    for what, (run, ref, ulp, frac) in cases.items():
        ys = [Tensor.zeros((M, N), "float16", dev) for _ in range(60)]
        for i, y in enumerate(ys):
            run(y, wt[i % len(wt)])
        dev.synchronize()
        first = ys[0].numpy()
        assert_reduction_close(first, ref, max_ulp=ulp, max_frac=frac, what=what)
        assert all((y.numpy().view(np.uint16) == first.view(np.uint16)).all() for y in ys[1:]), what
