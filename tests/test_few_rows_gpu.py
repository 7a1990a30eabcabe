"""The projections of a few rows around the weight stream (skinny.cuh) at the edges of their tiles: outputs fewer than CTAs, a row more
than a tile, one and two tiles to a warp, a second pass; K of one run, and with a last stage that is not full."""
import os
import subprocess
import sys

import numpy as np
import pytest

from denograd_b200 import Device
from denograd_b200.device import Tensor
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CODES = [-1.0, -0.6961928009986877, -0.5250730514526367, -0.39491748809814453, -0.28444138169288635, -0.18477343022823334, -0.09105003625154495, 0.0,
         0.07958029955625534, 0.16093020141124725, 0.24611230194568634, 0.33791524171829224, 0.44070982933044434, 0.5626170039176941, 0.7229568362236023, 1.0]


@pytest.fixture(scope="module")
def dev():
    return Device["CUDA"]


def weights(rng, kind, N, K, dev):
    """(pointers of matrix and scales, dequantised values in 64 bits)"""
    if kind == "int8":
        q, s = rng.integers(-127, 128, (N, K), dtype=np.int8), (rng.uniform(0.5, 1.5, N) * 3e-4).astype(np.float16)
        return (Tensor(q, device=dev), Tensor(s, device=dev)), (q.astype(np.float16) * s[:, None]).astype(np.float64)
    w = (rng.standard_normal((N, K)) * 0.02).astype(np.float16)
    return (Tensor(w, device=dev), None), w.astype(np.float64)


@pytest.mark.parametrize("kind", ["float16", "int8"])
@pytest.mark.parametrize("M,N,K", [(3, 5, 128), (8, 149, 256), (4, 148 * 16 + 3, 1152), (7, 148 * 64 + 130, 384), (8, 148 * 136 + 9, 128), (5, 148 * 256 + 77, 128), (16, 700, 2048)])
def test_edges_of_tiles(dev, kind, M, N, K):
    """Tolerance: the fp32 sum of K exact products (relative to the sum of their magnitudes) and an fp16 rounding per elementwise op."""
    rng = np.random.default_rng(M * 7 + N + K)
    x, res = rng.standard_normal((M, K)).astype(np.float16), rng.standard_normal((M, N)).astype(np.float16)
    (w, s), dw = weights(rng, kind, N, K, dev)
    (w3, s3), dw3 = weights(rng, kind, N, K, dev)
    sp, sp3 = s.ptr if s else 0, s3.ptr if s3 else 0
    xt, rt, y = Tensor(x, device=dev), Tensor(res, device=dev), Tensor.zeros((M, N), "float16", dev)
    x64, ulp, eps = x.astype(np.float64), 2.0 ** -11, 2.0 ** -20
    g, u, mg, mu = x64 @ dw.T, x64 @ dw3.T, np.abs(x64) @ np.abs(dw).T, np.abs(x64) @ np.abs(dw3).T

    def check(want, bound):
        assert (np.abs(y.numpy().astype(np.float64) - want) <= bound + 1e-7).all()

    dev.call("jg_linear", y.ptr, xt.ptr, w.ptr, sp, 0, M, N, K)
    check(g, eps * mg + ulp * np.abs(g) * 1.01)
    dev.call("jg_linear", y.ptr, xt.ptr, w.ptr, sp, rt.ptr, M, N, K)
    check(g + res, eps * mg + ulp * (np.abs(g) + np.abs(g + res)) * 1.01)
    dev.call("jg_norm_swiglu", y.ptr, xt.ptr, 0, 1e-5, w.ptr, sp, w3.ptr, sp3, M, N, K)
    want = g / (1 + np.exp(-g)) * u
    check(want, 8 * ulp * np.abs(want) + 1.2 * np.abs(u) * (eps * mg + ulp * np.abs(g)) + np.abs(g) * eps * mu + 1e-4)
    p32 = Tensor.zeros((M, N), "float32", dev)
    dev.call("jg_linear_partial", p32.ptr, xt.ptr, w.ptr, sp, M, N, K)
    assert (np.abs(p32.numpy() - g) <= eps * mg + 1e-7).all()
    key, tok = Tensor.zeros((M,), "uint64", dev), Tensor.empty((M,), "int32", dev)
    dev.call("jg_norm_logits_argmax", y.ptr, key.ptr, xt.ptr, 0, 1e-5, w.ptr, sp, M, N, K)
    dev.call("jg_argmax_finalize", tok.ptr, key.ptr, M)
    check(g, eps * mg + ulp * np.abs(g) * 1.01)
    assert tok.numpy().tolist() == [O.argmax_f16(r) for r in y.numpy()]


@pytest.mark.parametrize("M,N,K,block", [(1, 148 * 72 + 5, 512, 64), (8, 150, 256, 32), (2, 33, 2048, 256), (1, 14, 8192, 64)])
def test_nf4_blocks_and_stages(dev, M, N, K, block):
    """Blocks of 32 to 256: the scales of a stage take 16 bytes a row at least."""
    rng = np.random.default_rng(N + block)
    code = np.array(CODES).astype(np.float16)
    x, c = rng.standard_normal((M, K)).astype(np.float16), rng.integers(0, 16, N * K).astype(np.uint8)
    s = (0.02 + 0.05 * rng.random(N * K // block)).astype(np.float16)
    d = (code[c].reshape(-1, block) * s[:, None]).astype(np.float16).reshape(N, K).astype(np.float64)
    xt, y = Tensor(x, device=dev), Tensor.zeros((M, N), "float16", dev)
    wt, st = Tensor(c[0::2] * 16 + c[1::2], device=dev), Tensor(s, device=dev)
    dev.call("jg_linear_nf4", y.ptr, xt.ptr, wt.ptr, st.ptr, 0, M, N, K, block)
    want, mag = x.astype(np.float64) @ d.T, np.abs(x.astype(np.float64)) @ np.abs(d).T
    assert (np.abs(y.numpy().astype(np.float64) - want) <= 2.0 ** -20 * mag + 2.0 ** -11 * np.abs(want) * 1.01 + 1e-7).all()


def int8_matrix(rng, N, K, dev):
    q, s = rng.integers(-127, 128, (N, K), dtype=np.int8), (rng.uniform(0.5, 1.5, N) * 3e-4).astype(np.float16)
    return q, Tensor(q, device=dev), Tensor(s, device=dev)


@pytest.mark.parametrize("M", [2, 5, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(1000, 512), (300, 2048), (6000, 2176), (4096, 5120), (6144, 3584), (12000, 2048), (24001, 2304)])
def test_int8_sums_are_the_general_kernels_to_the_bit(dev, M, N, K):
    """64 columns of zeros more keep a call off the kernel around the weight stream and add nothing: the same bits, so that a token drawn
    from a quantised model does not hang on which of the two ran."""
    rng = np.random.default_rng(N + K + M)
    x = rng.standard_normal((M, K)).astype(np.float16)
    pad = lambda a: np.pad(a, ((0, 0), (0, 64)))
    (q, w, s), (q3, w3, s3) = int8_matrix(rng, N, K, dev), int8_matrix(rng, N, K, dev)
    outs = []
    for xa, wa, w3a in ((x, w, w3), (pad(x), Tensor(pad(q), device=dev), Tensor(pad(q3), device=dev))):
        xt, k = Tensor(xa, device=dev), xa.shape[1]
        y32, y, z = Tensor.zeros((M, N), "float32", dev), Tensor.zeros((M, N), "float16", dev), Tensor.zeros((M, N), "float16", dev)
        key = Tensor.zeros((M,), "uint64", dev)
        dev.call("jg_linear_partial", y32.ptr, xt.ptr, wa.ptr, s.ptr, M, N, k)
        dev.call("jg_norm_swiglu", y.ptr, xt.ptr, 0, 1e-5, wa.ptr, s.ptr, w3a.ptr, s3.ptr, M, N, k)
        dev.call("jg_norm_logits_argmax", z.ptr, key.ptr, xt.ptr, 0, 1e-5, wa.ptr, s.ptr, M, N, k)
        outs.append([t.numpy() for t in (y32, y, z, key)])
    for a, b in zip(*outs):
        assert (a.view(np.uint8) == b.view(np.uint8)).all()


@pytest.mark.parametrize("N,K", [(14336, 4096), (6144, 4096), (4096, 14336), (8192, 2048), (1003, 512), (24001, 1536)])
def test_int8_sums_of_one_row_do_not_depend_on_where_it_is_normalised(dev, N, K):
    """A row of ones and minus ones is its own norm at eps = 0, so the launch that normalises and the one that is given the row multiply
    the same numbers: the same bits."""
    rng = np.random.default_rng(N + K)
    xt = Tensor(rng.choice(np.array([-1, 1], np.float16), (1, K)), device=dev)
    ones = Tensor(np.ones(K, np.float16), device=dev)
    (_, w, s), (_, w3, s3) = int8_matrix(rng, N, K, dev), int8_matrix(rng, N, K, dev)
    outs = []
    for norm in (0, ones.ptr):
        y, g, z, key = Tensor.zeros((1, N), "float16", dev), Tensor.zeros((1, N), "float16", dev), Tensor.zeros((1, N), "float16", dev), Tensor.zeros((1,), "uint64", dev)
        if norm:
            dev.call("jg_norm_linear", y.ptr, xt.ptr, norm, 0.0, w.ptr, s.ptr, 1, N, K)
        else:
            dev.call("jg_linear", y.ptr, xt.ptr, w.ptr, s.ptr, 0, 1, N, K)
        dev.call("jg_norm_swiglu", g.ptr, xt.ptr, norm, 0.0, w.ptr, s.ptr, w3.ptr, s3.ptr, 1, N, K)
        dev.call("jg_norm_logits_argmax", z.ptr, key.ptr, xt.ptr, norm, 0.0, w.ptr, s.ptr, 1, N, K)
        outs.append([t.numpy() for t in (y, g, z, key)])
    for a, b in zip(*outs):
        assert (a.view(np.uint8) == b.view(np.uint8)).all()


@pytest.mark.parametrize("M", [1, 8])
@pytest.mark.parametrize("N,K", [(8192, 2048), (14336, 4096), (12289, 2048), (4096, 14336)])
@pytest.mark.parametrize("block", [32, 64, 128, 256])
def test_nf4_wide_matrices_of_every_block(dev, block, M, N, K):
    """One matrix and two, against the products of the dequantised matrix in 64 bits: fp32 sums of K exact products and one fp16 rounding
    per output and elementwise op.  Wide matrices leave few warps to a tile, so that large blocks need many runs for 16 bytes of scales."""
    import torch

    rng = np.random.default_rng(N + K + block)
    code = torch.tensor(CODES, dtype=torch.float64, device="cuda").half()
    x = rng.standard_normal((M, K)).astype(np.float16)
    ws, sums, mags = [], [], []
    x64 = torch.from_numpy(x).cuda().double()
    for _ in range(2):
        c = rng.integers(0, 256, N * K // 2).astype(np.uint8)
        s = (0.02 + 0.05 * rng.random(N * K // block)).astype(np.float16)
        ws.append((Tensor(c, device=dev), Tensor(s, device=dev)))
        ct = torch.from_numpy(c).cuda()
        d = (code[torch.stack([ct >> 4, ct & 15], -1).reshape(-1, block).long()] * torch.from_numpy(s).cuda()[:, None]).reshape(N, K).double()
        sums.append((x64 @ d.T).cpu().numpy())
        mags.append((x64.abs() @ d.abs().T).cpu().numpy())
    (g, u), eps, ulp = sums, 2.0 ** -20, 2.0 ** -11
    xt, y = Tensor(x, device=dev), Tensor.zeros((M, N), "float16", dev)
    dev.call("jg_linear_nf4", y.ptr, xt.ptr, ws[0][0].ptr, ws[0][1].ptr, 0, M, N, K, block)
    assert (np.abs(y.numpy().astype(np.float64) - g) <= eps * mags[0] + ulp * np.abs(g) * 1.01 + 1e-7).all()
    dev.call("jg_swiglu_nf4", y.ptr, xt.ptr, ws[0][0].ptr, ws[0][1].ptr, ws[1][0].ptr, ws[1][1].ptr, M, N, K, block)
    want = g / (1 + np.exp(-g)) * u
    bound = 8 * ulp * np.abs(want) + 1.2 * np.abs(u) * (eps * mags[0] + ulp * np.abs(g)) + np.abs(g) * eps * mags[1] + 1e-4
    assert (np.abs(y.numpy().astype(np.float64) - want) <= bound).all()


@pytest.mark.parametrize("rows,M,K", [(8, 4, 8192), (5, 8, 4096), (128, 3, 4096)])
def test_normed_rows_as_the_next_calls_weights(dev, rows, M, K):
    """The launch behind a norm starts beside it: where its weights are the norm's result it waits before it requests them."""
    rng = np.random.default_rng(rows + K)
    x, ones, y = rng.standard_normal((M, K)).astype(np.float16), Tensor(np.ones(K, np.float16), device=dev), Tensor.zeros((rows, K), "float16", dev)
    xt, out = Tensor(x, device=dev), Tensor.zeros((M, rows), "float16", dev)
    for scale in (1.0, 3.0, -2.0, 0.5):  # a stale matrix would show the sign or the rows of the turn before
        h = (scale * rng.standard_normal((rows, K))).astype(np.float16)
        ht = Tensor(h, device=dev)
        dev.synchronize()
        dev.call("jg_rmsnorm", y.ptr, ht.ptr, ones.ptr, rows, K, 1e-5)
        dev.call("jg_linear", out.ptr, xt.ptr, y.ptr, 0, 0, M, rows, K)
        w = y.numpy().astype(np.float64)
        want, mag = x.astype(np.float64) @ w.T, np.abs(x.astype(np.float64)) @ np.abs(w).T
        assert (np.abs(out.numpy() - want) <= 2.0 ** -20 * mag + 2.0 ** -11 * np.abs(want) * 1.01 + 1e-7).all()


SWITCH = """
import numpy as np
from denograd_b200 import Device
from denograd_b200.device import Tensor
dev, rng, M, N, K = Device["CUDA"], np.random.default_rng(3), 4, 14336, 4096
x, w = rng.standard_normal((M, K)).astype(np.float16), (rng.standard_normal((N, K)) * 0.02).astype(np.float16)
outs = []
for pad in (0, 8):
    xt, wt = (Tensor(np.pad(a, ((0, 0), (0, pad))), device=dev) for a in (x, w))
    y = Tensor.zeros((M, N), "float32", dev)
    dev.call("jg_linear_partial", y.ptr, xt.ptr, wt.ptr, 0, M, N, K + pad)
    outs.append(y.numpy().view(np.uint32))
print("same" if (outs[0] == outs[1]).all() else "differ")
"""


@pytest.mark.parametrize("rows,want", [("65", "same"), (None, "differ")])
def test_the_switch_between_the_tensor_core_projections_decides_for_few_rows(rows, want):
    """Eight columns of zeros more keep a call off every kernel but gemm_small.cu's.  JG_TC_MIN_M beyond the rows sends the call without
    them there, too (the same bits); unset, they go to the kernel around the weight stream, which adds K in another order."""
    env = {k: v for k, v in os.environ.items() if k != "JG_TC_MIN_M"}
    env.update({"JG_TC_MIN_M": rows} if rows else {})
    r = subprocess.run([sys.executable, "-c", SWITCH], capture_output=True, text=True, env=env, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.stdout.split()[-1:] == [want], (r.stdout, r.stderr[-2000:])
