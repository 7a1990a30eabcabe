"""Device buffers of a Llama's steps and prompts, over a recorder in the place of the library: what a captured step writes to stays
its own."""
import numpy as np

from tests.fake_ffi import recording


def model(**kw):
    from denograd_b200.llama3 import Llama3
    args = dict(dim=256, n_heads=4, n_kv_heads=2, n_layers=2, norm_eps=1e-5, rope_theta=500000, vocab_size=512, hidden_dim=576)
    return Llama3(size="1B", args=args, max_context=256, tied_output=True, temperature=0, **kw).model


def test_dequantised_copies_keep_their_place():
    """576 is no multiple of 128: of an NF4 block's matrices only w2 is dequantised in a step, all of them in a prompt."""
    with recording() as rec:
        m = model(quantize="nf4")
        for pos in (1, 2, 3):  # eager, captured, replayed
            m.call(np.zeros((1, 1), np.int32), pos)
        m.forward(np.zeros((1, 100), np.int32), 4)
        copies = {c[2] for c in rec.calls if c[0] == "jg_dequant_nf4_f16"}
        assert copies == {min(copies), min(copies) + 2 * 576 * 256}  # one allocation, with gate and up side by side


def test_prompts_of_many_lengths_share_their_buffers():
    with recording() as rec:
        m = model()
        m.forward(np.zeros((1, 33), np.int32), 0)
        first, n0 = m._workspace(33, rows=True).h.ptr, len(rec.calls)
        for n in (5, 17, 64, 9, 33, 48):
            m.forward(np.zeros((1, n), np.int32), 0)
            ws = m._workspace(n, rows=True)
            assert ws.B == n and ws.h.ptr == first and all(t.shape[0] == n for t in (ws.tokens, ws.pos, ws.seq, ws.xn, ws.qkv, ws.attn, ws.ffn, ws.part32))
        assert not [c for c in rec.calls[n0:] if c[0] in ("jg_alloc", "jg_host_alloc")]
        m.forward(np.zeros((1, 200), np.int32), 0)
        held = [c for c in rec.calls if c[0] == "jg_alloc"]
        for n in range(2, 256):
            m.forward(np.zeros((1, n), np.int32), 0)
        assert [c for c in rec.calls if c[0] == "jg_alloc"] == held
