"""Prompt attention of the Llama at the edges of its 128-row tiles, in both of its forms: pairs of query tiles to a CTA where they give
every SM one, single tiles with split keys below."""
import numpy as np
import pytest

from denograd_b200.device import Tensor
from denograd_b200.llama import KVCache
from oracle import oracle as O
from tests.test_kernels_gpu import assert_reduction_close

pytestmark = pytest.mark.gpu


# heads, kv heads, head size; sequences and tokens: more pairs of tiles than SMs (a second tile that is empty, part of one, whole
# ones; a last key tile of 1 to 128 keys), fewer
@pytest.mark.parametrize("H,G,hd,B,Sc", [(8, 8, 128, 10, 300), (8, 8, 64, 10, 384), (24, 8, 128, 7, 200), (24, 8, 64, 10, 85), (32, 8, 64, 10, 70), (32, 8, 128, 5, 256),
                                         (16, 2, 128, 11, 200), (64, 8, 64, 5, 97), (16, 8, 128, 10, 129), (24, 8, 64, 2, 170), (32, 8, 128, 1, 129), (16, 2, 64, 3, 31)])
@pytest.mark.parametrize("page", [16, 32, 64])
def test_tiles(dev, H, G, hd, B, Sc, page):
    rng = np.random.default_rng(H + G + hd + B + Sc + page)
    first = rng.choice([0, 1, 55, 127, 128, 200], B)  # every sequence continues at a place of its own
    first[0] = 0
    n, max_ctx = int(first.max()) + Sc, 640
    kv = KVCache(dev, 1, H, G, hd, max_ctx, B, page_size=page)
    kv.set_block_table(rng.permutation(kv.n_pages).astype(np.int32).reshape(B, kv.max_pages_per_seq))
    table = np.zeros((max_ctx, hd // 2, 2), np.float16)
    table[..., 0] = 1  # positions are not turned
    freqs = Tensor(table, device=dev)
    qkv = (rng.standard_normal((B, n, (H + 2 * G) * hd)) * 0.7).astype(np.float16)

    def rows(start, count):  # `count` positions of all sequences from start[b] on, row = s * B + b
        x = np.stack([[qkv[b, start[b] + s] for b in range(B)] for s in range(count)]).reshape(count * B, -1)
        t = Tensor(x, device=dev), Tensor((np.arange(count)[:, None] + start[None]).reshape(-1).astype(np.int32), device=dev), Tensor(np.tile(np.arange(B), count).astype(np.int32), device=dev)
        dev.call("jg_rope_kvwrite_rows", kv.handle, 0, t[0].ptr, freqs.ptr, max_ctx, t[1].ptr, t[2].ptr, count * B, H)
        return t

    if first.max():
        before = rows(np.zeros(B, np.int64), int(first.max()))  # noqa: F841  (some of it is written again below)
    x, pos, seq = rows(first, Sc)
    out = Tensor.zeros((Sc * B + 1, H * hd), "float16", dev)
    dev.call("jg_attn_chunk", kv.handle, 0, out.ptr, x.ptr, pos.ptr, seq.ptr, B, Sc, H)
    got = out.numpy()
    assert (got[Sc * B:] == 0).all()
    got = got[:Sc * B].reshape(Sc, B, H * hd)
    for b in range(B):
        k, v = (np.zeros((1, max_ctx, G, hd), np.float16) for _ in range(2))
        k[0, :n] = qkv[b, :, H * hd:(H + G) * hd].reshape(n, G, hd)
        v[0, :n] = qkv[b, :, (H + G) * hd:].reshape(n, G, hd)
        q = qkv[b, first[b]:first[b] + Sc, :H * hd].reshape(1, Sc, H, hd)
        assert_reduction_close(got[:, b], O.attention(q, k, v, int(first[b]))[0], max_ulp=2, max_frac=0.12, what=f"sequence {b} from {first[b]}")
    kv.close()
