"""GPU parity of the stochastic `sample` kernel (jg_sample) against the CPU checker's restatement of
jsgrad/models/llama.ts:131-185: the chosen token ids must be identical — the kernel adds its float32 sums in the
reference's own order, so there is no tolerance to state."""
import numpy as np
import pytest

from denograd_b200 import ffi, rand
from denograd_b200.device import Tensor
from denograd_b200.llama import sample
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _logits(rng, rows, V, spread):
    return (rng.standard_normal((rows, V)) * spread).astype(np.float16)


@pytest.mark.parametrize("V", [1000, 2048, 40000, 128256])
@pytest.mark.parametrize("k,p", [(0, 0.0), (1, 0.0), (40, 0.8), (40, 0.0), (7, 1.0), (200, 0.95)])
def test_sampled_ids_equal_the_checker(dev, V, k, p):
    rng = np.random.default_rng(V + 31 * k)
    rows = 3
    lg = _logits(rng, rows, V, 3.0)
    lg[1, 5] = lg[1, 900] = lg[1].max() + np.float16(1.0)  # a tie at the top: the lowest index must win a round
    lt = Tensor(lg, device=dev)
    out = Tensor.empty((rows,), "int32", dev)
    for temp in (0.95, 0.3):
        for trial in range(4):
            u = rng.random(rows, dtype=np.float32)
            dev.call("jg_sample", out.ptr, lt.ptr, Tensor(u, device=dev).ptr, 0, rows, V, temp, k, p, 0.0, 0.0)
            got = out.numpy()
            want = [O.sample(lg[r].astype(np.float32), temp, k, p, 0.0, 0.0, float(u[r])) for r in range(rows)]
            assert got.tolist() == want, (V, k, p, temp, trial)


def test_alpha_penalties_and_counter(dev):
    rng = np.random.default_rng(9)
    V, rows = 5000, 2
    lg = _logits(rng, rows, V, 2.0)
    lt = Tensor(lg, device=dev)
    cnt = Tensor.zeros((rows, V), "int32", dev)
    ref_cnt = np.zeros((rows, V), np.int32)
    out = Tensor.empty((rows,), "int32", dev)
    for step in range(12):  # a low temperature keeps picking the same few tokens: the penalties must move the pick on
        u = rng.random(rows, dtype=np.float32)
        dev.call("jg_sample", out.ptr, lt.ptr, Tensor(u, device=dev).ptr, cnt.ptr, rows, V, 0.2, 20, 0.9, 0.7, 0.4)
        want = [O.sample(lg[r].astype(np.float32), 0.2, 20, 0.9, 0.7, 0.4, float(u[r]), ref_cnt[r]) for r in range(rows)]
        assert out.numpy().tolist() == want, step
    assert (cnt.numpy() == ref_cnt).all() and ref_cnt.sum() == 24


def test_sample_wrapper_and_argument_checks(dev):
    rng = np.random.default_rng(2)
    V = 3000
    lg = _logits(rng, 1, V, 2.0)
    lt = Tensor(lg, device=dev)
    # temperature below 1e-6: argmax, lowest index among equals
    assert int(sample(lt, 0.0, 0, 0.0, 0.0, 0.0).numpy()[0]) == O.sample(lg[0].astype(np.float32), 0.0, 0, 0.0, 0, 0, 0.5)
    # default uniform source: the restated Tensor.rand stream
    rand.manual_seed(11)
    got = [int(sample(lt, 0.9, 0, 0.0, 0.0, 0.0).numpy()[0]) for _ in range(3)]
    rand.manual_seed(11)
    us = [float(rand.rand(1, dev.device)[0]) for _ in range(3)]
    assert got == [O.sample(lg[0].astype(np.float32), 0.9, 0, 0.0, 0, 0, u) for u in us]
    with pytest.raises(ValueError):
        sample(lt, 0.9, 0, 1.5, 0.0, 0.0)
    with pytest.raises(ValueError):
        sample(lt, 0.9, V + 1, 0.5, 0.0, 0.0)
    with pytest.raises(ffi.JgError):
        dev.call("jg_sample", lt.ptr, lt.ptr, lt.ptr, 0, 1, V, 0.9, 600, 0.5, 0.0, 0.0)  # k beyond the kernel's table


@pytest.mark.parametrize("V", [1, 300, 513, 4099, 40007, 40009 * 8, 128256])
@pytest.mark.parametrize("k", [0, 30])
def test_rows_at_the_edges_of_slices_and_chains(dev, V, k):
    """Vocabularies without a divisor for the chunked sums (one chain over all slices), with chunks longer than what a CTA
    keeps of its neighbour's slice, with one block or a padded first one; draws at both ends of the distribution; rows with
    infinities and NaN."""
    k = min(k, V)
    rng = np.random.default_rng(V + k)
    lg = _logits(rng, 5, V, 3.0)
    lg[1, V // 2:] = -np.inf
    lg[2, V // 3] = np.nan
    lg[3, :] = -np.inf
    lg[4, V - 1] = np.inf
    lt = Tensor(lg, device=dev)
    out = Tensor.empty((5,), "int32", dev)
    for u0 in (0.0, 0.37, 0.99999994):
        u = np.full(5, u0, np.float32)
        dev.call("jg_sample", out.ptr, lt.ptr, Tensor(u, device=dev).ptr, 0, 5, V, 0.95, k, 0.9, 0.0, 0.0)
        want = [O.sample(lg[r].astype(np.float32), 0.95, k, 0.9, 0.0, 0.0, u0) for r in range(5)]
        # without a finite maximum every probability is NaN: the draw then gives 0, the rounds of the top k are not defined
        rows = [r for r in range(5) if k == 0 or np.isfinite(np.where(np.isnan(lg[r]), -np.inf, lg[r]).max())]
        assert [out.numpy()[r] for r in rows] == [want[r] for r in rows], (V, k, u0)


@pytest.mark.parametrize("V", [370001, 380000, 382976])
@pytest.mark.parametrize("k", [0, 30])
def test_the_largest_vocabularies(dev, V, k):
    """Slices that leave room for no more than their padding and the head of the next one; one value more per slice is refused."""
    rng = np.random.default_rng(V + k)
    lg = _logits(rng, 2, V, 3.0)
    lt, out = Tensor(lg, device=dev), Tensor.empty((2,), "int32", dev)
    for u0 in (0.0, 0.61, 0.99999994):
        dev.call("jg_sample", out.ptr, lt.ptr, Tensor(np.full(2, u0, np.float32), device=dev).ptr, 0, 2, V, 0.95, k, 0.9, 0.0, 0.0)
        assert out.numpy().tolist() == [O.sample(r.astype(np.float32), 0.95, k, 0.9, 0.0, 0.0, u0) for r in lg], (V, k, u0)
    with pytest.raises(ffi.JgError):
        dev.call("jg_sample", out.ptr, lt.ptr, lt.ptr, 0, 2, 382977, 0.95, k, 0.9, 0.0, 0.0)
