"""Window attention over long portions in 128-row tiles: heads per kv head, pages smaller and larger than a tile, kept tokens ending
inside, at and behind a tile, windows that begin inside one, portions that wrap the ring, several sequences at once."""
import numpy as np
import pytest

from oracle import rigazen as O
from tests.test_rigazen_gpu import build, check, config, parallel, run, tokens, window

pytestmark = pytest.mark.gpu


def branch(heads, kv_heads, dim, size, keep, scale=None):
    return parallel(window(dim=dim, heads=heads, kv_heads=kv_heads, mask={"keep_first": keep, "size": size}, rot={"base": 2000.0, "dims": dim // 2},
                           scale=dim ** -0.5 if scale is None else scale, vdim=dim), right_scale=0.4)


@pytest.mark.parametrize("heads,kv_heads,dim", [(4, 1, 128), (2, 2, 64), (8, 1, 64), (6, 3, 128)])
@pytest.mark.parametrize("size,keep,page", [(4096, 0, 64), (100, 5, 16), (130, 140, 8), (129, 128, 256), (257, 64, 128)])
def test_long_portions(heads, kv_heads, dim, size, keep, page):
    cfg = config(branch(heads, kv_heads, dim, size, keep), width=64)
    params, toks = O.random_params(cfg, seed=3), tokens(cfg, 601)
    want = O.forward(params, cfg, toks)
    m = build(cfg, params, "bfloat16", max_context=640, page_size=page, max_rows=601)
    for cuts in ([601], [129, 472], [128, 200, 1, 272], [20, 300, 281], [256, 257, 88]):
        check(run(m, toks, cuts), want, "bfloat16", (size, keep, cuts))


# heads and tokens enough for two tiles of queries to a CTA (a pair of tiles for every SM): 601 and 472 tokens, or 601 alone
@pytest.mark.parametrize("heads,kv_heads,dim", [(128, 16, 64), (64, 8, 128)])
@pytest.mark.parametrize("size,keep,page", [(4096, 0, 64), (100, 5, 16), (130, 140, 8), (257, 64, 128)])
def test_pairs_of_query_tiles(heads, kv_heads, dim, size, keep, page):
    cfg = config(branch(heads, kv_heads, dim, size, keep), width=64)
    params, toks = O.random_params(cfg, seed=7), tokens(cfg, 601)
    want = O.forward(params, cfg, toks)
    m = build(cfg, params, "bfloat16", max_context=640, page_size=page, max_rows=601)
    for cuts in ([601], [129, 472], [20, 300, 281]):
        check(run(m, toks, cuts), want, "bfloat16", (size, keep, cuts))


def test_two_sequences_at_once():
    cfg = config(branch(4, 2, 128, 150, 70), width=64)
    params, rows = O.random_params(cfg, seed=4), np.stack([tokens(cfg, 620, seed=s) for s in (5, 6)])
    m = build(cfg, params, "bfloat16", max_context=640, max_batch=2, max_rows=1280)
    m.forward(rows[:, :20], 0)
    m.forward(rows[:, 20:], 20)
    got = m.last_logits(2)
    for b in range(2):
        check(got[b:b + 1], O.forward(params, cfg, rows[b].tolist())[-1:], "bfloat16")


@pytest.mark.parametrize("scale", [0.0, -0.11])
def test_scales_that_are_not_positive(scale):
    cfg = config(branch(4, 1, 128, 150, 70, scale), width=64)
    params, toks = O.random_params(cfg, seed=6), tokens(cfg, 300)
    want = O.forward(params, cfg, toks)
    m = build(cfg, params, "bfloat16", max_context=320, max_rows=300)
    for cuts in ([300], [255, 45], [43, 257]):
        check(run(m, toks, cuts), want, "bfloat16", (scale, cuts))
