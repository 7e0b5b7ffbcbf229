"""The prompt matrices for few tokens (blocks of 16, 32 and 48 instead of 64) at both sides of every block's end.

The integer sums, the parts a row's groups are dealt into and the order in which they are added do not depend on the block a token
travels in, and 64 positions are one key range of the attention, so the K/V rows of both layers of a two-layer model are the
same bits as in a block of 64: those of the second layer have passed all four matrices of the first.  Against the decode step the
tolerance is that of the prompt path (1e-4 of the logit range, tests/test_gpu_prefill.py)."""
import numpy as np
import pytest

from llama2j_b200 import synthetic as syn
from llama2j_b200.model_files import ModelConfig
from llama2j_b200.transformer import Transformer

pytestmark = pytest.mark.gpu

COUNTS = (1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63)


def _build(cfg, tensors):
    m = Transformer(cfg, 0)
    m.upload_all(tensors)
    m.finalize()
    return m


def _config(layers):
    # 10 groups per row of dim and 13 of hidden: odd counts for both issue lanes, parts of unequal length
    return ModelConfig(dim=2560, hidden_dim=3328, n_layers=layers, n_heads=20, n_kv_heads=4, vocab_size=600, seq_len=96,
                       shared_classifier=True)


def test_rows_are_those_of_a_full_block():
    cfg = _config(2)
    tensors = syn.synthetic_tensors(cfg, 4)
    rng = np.random.default_rng(5)
    toks, other = (rng.integers(3, cfg.vocab_size, 64).astype(np.int32) for _ in range(2))
    m = _build(cfg, tensors)

    def rows():
        return np.array([[m.read_buffer(w, cfg.kv_dim, layer, p) for layer in range(2) for w in (5, 6)] for p in range(64)])

    m.prefill(toks, 0)
    want = rows()
    for n in COUNTS:
        m.prefill(other, 0)                       # every row is another one before it is written again
        before = rows()
        assert all(not np.array_equal(before[p], want[p]) for p in range(64))
        m.prefill(toks[:64 - n], 0)
        m.prefill(toks[64 - n:], 64 - n)
        assert np.array_equal(rows(), want), n
    assert m.stats().device_status == 0
    m.close()


@pytest.mark.parametrize("n", COUNTS)
def test_step_of_n_sequences_and_prompt_of_n_tokens(n):
    cfg = _config(2)
    tensors = syn.synthetic_tensors(cfg, 6)
    toks = np.random.default_rng(7).integers(3, cfg.vocab_size, n).astype(np.int32)
    dec = _build(cfg, tensors)
    m = _build(cfg, tensors)
    m.batch_create(n, 4)
    got, ids = m.batch_forward(np.arange(n, dtype=np.int32), np.zeros(n, dtype=np.int32), toks)
    got = got.copy()
    for i in range(n):
        ref = dec.forward(int(toks[i]), 0)[0]
        assert float(np.abs(got[i] - ref).max()) <= 1e-4 * float(ref.max() - ref.min()), i
    for i in range(n):
        dec.forward(int(toks[i]), i, want_logits=False)
    m.prefill(toks, 0)
    a, b = dec.forward(9, n)[0].copy(), m.forward(9, n)[0].copy()
    assert float(np.abs(a - b).max()) <= 1e-4 * float(a.max() - a.min())
    assert m.stats().device_status == 0
    m.close()
    dec.close()
