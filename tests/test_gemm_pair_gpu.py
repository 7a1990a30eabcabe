"""Projections of many rows on pairs of CTAs: ragged tiles, tiles shared along K, whole rounds of tiles."""
import ctypes as C

import numpy as np
import pytest

from denograd_b200 import ffi
from denograd_b200.device import Tensor
from denograd_b200.hybrid import DTYPES
from oracle import matulorn as R
from oracle import oracle as O
from tests.test_kernels_gpu import assert_reduction_close

pytestmark = pytest.mark.gpu


def bound(x, w):
    """fp32 sums of K products in any two orders: K roundings of at most the sum of the magnitudes each."""
    return 2 * x.shape[1] * 2.0 ** -24 * (np.abs(x) @ np.abs(w).T) + 1e-30


# one k-block; half a weight tile; few tiles in shares; whole rounds and remainders; the last activation row alone
@pytest.mark.parametrize("M,N,K", [(65, 128, 64), (33, 384, 2048), (129, 384, 4096), (225, 256, 1024), (513, 1280, 640), (700, 4096, 576), (1999, 2304, 192), (257, 512, 14336),
                                   (33, 12672, 128), (65, 14336, 128), (256, 12672, 576), (257, 12672, 128), (200, 18944, 64), (100, 19072, 64), (100, 12544, 128)])
def test_fp16_epilogues(dev, M, N, K):
    rng = np.random.default_rng(M + N + K)
    x, res = (rng.standard_normal(s).astype(np.float16) for s in ((M, K), (M, N)))
    w, w3 = ((rng.standard_normal((N, K)) * K ** -0.5).astype(np.float16) for _ in range(2))
    xt, wt, w3t, rt = (Tensor(a, device=dev) for a in (x, w, w3, res))
    xf, wf = x.astype(np.float32), w.astype(np.float32)
    acc, off = xf @ wf.T, bound(xf, wf)
    p32 = Tensor.zeros((M + 1, N), "float32", dev)
    for _ in range(2):  # the second launch finds the first one's flags cleared
        dev.call("jg_linear_partial", p32.ptr, xt.ptr, wt.ptr, 0, M, N, K)
        got = p32.numpy()
        assert (np.abs(got[:M] - acc) <= off).all() and (got[M:] == 0).all()
    y = Tensor.zeros((M + 1, N), "float16", dev)
    dev.call("jg_linear", y.ptr, xt.ptr, wt.ptr, 0, 0, M, N, K)
    assert (y.numpy()[:M] == got[:M].astype(np.float16)).all()  # the same sums, rounded once
    dev.call("jg_copy", y.ptr, rt.ptr, 2 * M * N)
    dev.call("jg_linear", y.ptr, xt.ptr, wt.ptr, 0, y.ptr, M, N, K)  # the residual in place
    assert (y.numpy()[:M] == (res.astype(np.float32) + got[:M].astype(np.float16)).astype(np.float16)).all()
    for gate, up, g, u in ((wt, w3t, w, w3), (w3t, wt, w3, w)):  # either matrix may lie first in memory
        dev.call("jg_norm_swiglu", y.ptr, xt.ptr, 0, 1e-5, gate.ptr, 0, up.ptr, 0, M, N, K)
        want = O.swiglu(*((xf @ a.astype(np.float32).T).astype(np.float16) for a in (g, u)))
        assert_reduction_close(y.numpy()[:M], want, max_ulp=3, max_frac=0.12, what="swiglu")
    assert (y.numpy()[M:] == 0).all()


# 12672 features, 99 tiles, and 18944, 148: a CTA per tile up to 256 rows; 12544, 98, and 19072, 149: pairs
@pytest.mark.parametrize("M,N,K", [(33, 600, 1000), (65, 513, 520), (300, 1000, 1500), (1030, 4100, 712), (131, 1, 8), (64, 12665, 576), (65, 12665, 576), (129, 18944, 136), (256, 12665, 576),
                                   (257, 12665, 136), (40, 12544, 136), (129, 19072, 136)])
@pytest.mark.parametrize("glu", [False, True])
def test_bf16_epilogues(dev, M, N, K, glu):
    """Any N and K: edges of the tiles in every direction, columns in 32 bits elsewhere, biases."""
    rng = np.random.default_rng(M)
    ld, ldy, split = (K + 7) // 8 * 8, (N + 7) // 8 * 8, N - 9 if N > 9 else N
    x, w = np.zeros((M, ld), np.float32), np.zeros((2, N, ld), np.float32)
    x[:, :K], w[:, :, :K] = R.bf16_round(rng.standard_normal((M, K))), R.bf16_round(rng.standard_normal((2, N, K)) / np.sqrt(K))
    bias = rng.standard_normal((2, N)).astype(np.float32)
    t = lambda a: Tensor.zeros(a.shape, "bfloat16", dev).assign(a)  # noqa: E731
    tx, tw, tb = t(x), [t(w[0]), t(w[1])], [Tensor(b, device=dev) for b in bias]
    y, y2 = Tensor.zeros((M + 1, ldy), "bfloat16" if glu else "float32", dev), Tensor.zeros((M + 1, 9), "float32", dev)
    d = ffi.DenseDesc(DTYPES["bfloat16"], ffi.DENSE_GLU if glu else ffi.DENSE_STORE, N, K, ld, ld, ldy, 0 if glu else 1, 0.7, 0, tx.ptr, tw[0].ptr, tw[1].ptr, 0,
                      tb[0].ptr, tb[1].ptr, 0, y.ptr)
    a, b = (x.astype(np.float64) @ w[i].T.astype(np.float64) + bias[i] for i in range(2))
    if glu:
        g, u = np.minimum(a, 0.7), np.clip(b, -0.7, 0.7)
        a = g * R.sigmoid(1.702 * g) * (u + 1)
    else:
        d.act, d.act_lo, d.act_hi = ffi.ACT_SILU, 1, split
        if split < N:
            d.split, d.ld2, d.y2 = split, 9, y2.ptr
        a[:, 1:split] = a[:, 1:split] * R.sigmoid(a[:, 1:split])
    dev.call("jg_dense", C.byref(ffi.Batch(M, 1, 0, 0, -1, 0)), d)
    # |silu'| and |glu'| stay below 1.7; a bf16 result is off by one part in 256
    off = 1.7 * np.maximum(bound(x, w[0]), bound(x, w[1])) + 1e-5 + (np.abs(a) / 256 if glu else 0)
    got = y.numpy()
    if not glu:
        got[:M, split:N] = y2.numpy()[:M, :N - split]
        assert (y2.numpy()[M:] == 0).all()
    assert (np.abs(got[:M, :N] - a) <= off).all() and (got[M:] == 0).all() and (got[:, N:] == 0).all()


def test_silu_of_every_gate(dev):
    """Both forms of the fp16 exponential: every 16-bit gate, bit for bit."""
    g = np.arange(1 << 16, dtype=np.uint32).astype(np.uint16).view(np.float16)
    g = g[np.isfinite(g)]
    for up in (1.0, -0.37):
        u = np.full(g.shape, up, np.float16)
        y, gt, ut = Tensor.zeros(g.shape, "float16", dev), Tensor(g, device=dev), Tensor(u, device=dev)
        dev.call("jg_swiglu", y.ptr, gt.ptr, ut.ptr, g.size)
        want = O.swiglu(g[None], u[None])[0]
        got = y.numpy()
        assert ((got.view(np.uint16) == want.view(np.uint16)) | (np.isnan(got) & np.isnan(want))).all()
