"""Launches captured before anything else has run on a device handle: no entry point needs an eager call ahead of it."""
import numpy as np
import pytest

from denograd_b200 import ffi
from denograd_b200.device import CUDA, CUDAGraph, Tensor
from denograd_b200.llama import KVCache
from tests.test_kernels_gpu import assert_reduction_close

pytestmark = pytest.mark.gpu


@pytest.fixture
def own():
    """A handle of its own on the device."""
    d = CUDA("CUDA").init()
    yield d
    d.synchronize()


def replay(dev, launch):
    g = CUDAGraph(dev)
    with g:
        launch()
    g.launch()
    dev.synchronize()


def test_chunk_attention(own):
    B, Sc, H, G, hd = 2, 40, 4, 2, 64
    rng = np.random.default_rng(1)
    kv = KVCache(own, 1, H, G, hd, 64, B, page_size=16)
    qkv = Tensor(rng.standard_normal((B * Sc, (H + 2 * G) * hd)).astype(np.float16), device=own)
    pos, seq = (Tensor(a.astype(np.int32), device=own) for a in (np.repeat(np.arange(Sc), B), np.tile(np.arange(B), Sc)))
    freqs = Tensor.zeros((64, hd // 2, 2), "float16", own)
    ffi.call("jg_freqs_cis", own.handle, freqs.ptr, hd, 64, 10000.0)
    ffi.call("jg_rope_kvwrite_rows", own.handle, kv.handle, 0, qkv.ptr, freqs.ptr, 64, pos.ptr, seq.ptr, B * Sc, H)
    out = [Tensor.zeros((B * Sc, H * hd), "float16", own) for _ in range(2)]
    own.synchronize()
    call = lambda y: own.call("jg_attn_chunk", kv.handle, 0, y.ptr, qkv.ptr, pos.ptr, seq.ptr, B, Sc, H)  # noqa: E731
    replay(own, lambda: call(out[0]))
    call(out[1])
    a, b = out[0].numpy(), out[1].numpy()
    assert np.abs(a).max() > 0 and (a.view(np.uint16) == b.view(np.uint16)).all()
    kv.close()


def test_projection(own):
    M, N, K = 70, 256, 512  # few tiles: cut along K where the handle has room for shares, whole where it is first met in a capture
    rng = np.random.default_rng(2)
    x, w = rng.standard_normal((M, K)).astype(np.float16), (rng.standard_normal((N, K)) * 0.05).astype(np.float16)
    xt, wt, y = Tensor(x, device=own), Tensor(w, device=own), Tensor.zeros((M, N), "float16", own)
    own.synchronize()
    replay(own, lambda: own.call("jg_linear", y.ptr, xt.ptr, wt.ptr, 0, 0, M, N, K))
    assert_reduction_close(y.numpy(), (x.astype(np.float32) @ w.astype(np.float32).T).astype(np.float16), max_ulp=1, max_frac=0.08)
