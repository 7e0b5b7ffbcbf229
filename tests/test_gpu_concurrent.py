"""Concurrent sequences on one sweep over the weights (l2j_batch_create / l2j_batch_forward) against the
single-sequence decode path: every sequence of a batch must see exactly its own history.

Gates (the batched path adds the row sums in another order than the decode kernels, so tolerances, written
here): logits within 1e-4 of the logit range of a decode-only context that ran the same sequence alone, same
arg-max; and within the north star's 1e-3 of the CPU checker.
"""
import numpy as np
import pytest

from llama2j_b200 import lib as L
from llama2j_b200 import synthetic as syn
from llama2j_b200.model_files import ModelConfig
from llama2j_b200.transformer import Transformer
from tests.np_model import bf16_pieces as pieces
from tests.np_model import dequant

pytestmark = pytest.mark.gpu

LOGIT_TOL = 1e-4
ORACLE_TOL = 1e-3


def _tensors(cfg, seed):
    tensors = syn.synthetic_tensors(cfg, seed)
    rng = np.random.default_rng(seed + 100)
    for t in (L.T_RMS_ATT, L.T_RMS_FFN, L.T_RMS_FINAL):
        tensors[t] = syn.quant_encode(rng.uniform(0.5, 1.5, cfg.tensor_floats(t)).astype(np.float32))
    return tensors


def _build(cfg, tensors, flags=0):
    m = Transformer(cfg, 0, 0, None, flags)
    m.upload_all(tensors)
    m.finalize()
    return m


def _alone(cfg, tensors, stream):
    """Logits of every position of one forced token stream through the decode path."""
    m = _build(cfg, tensors)
    out = [m.forward(int(t), p)[0].copy() for p, t in enumerate(stream)]
    m.close()
    return out


def _check(got, ref):
    span = float(ref.max() - ref.min())
    assert float(np.abs(got - ref).max()) / span < LOGIT_TOL
    assert int(got.argmax()) == int(ref.argmax())


@pytest.mark.parametrize("cfg", [ModelConfig(256, 768, 3, 4, 4, 1000, 128, True),
                                 ModelConfig(512, 1280, 2, 8, 2, 1500, 128, False)], ids=["heads64", "grouped-query"])
def test_sequences_of_different_lengths_step_together(cfg):
    """Five sequences that start at different steps and have different tokens; one batch step per round."""
    tensors = _tensors(cfg, 11)
    rng = np.random.default_rng(12)
    n_seq, rounds = 5, 40
    starts = [0, 0, 3, 7, 20]                      # the round in which a sequence joins
    streams = [np.concatenate([[1], rng.integers(3, cfg.vocab_size, rounds)]).astype(np.int32) for _ in range(n_seq)]
    refs = [_alone(cfg, tensors, streams[s][:rounds - starts[s]]) for s in range(n_seq)]
    m = _build(cfg, tensors)
    m.batch_create(n_seq, 64)
    for r in range(rounds):
        live = [s for s in range(n_seq) if r >= starts[s]]
        pos = [r - starts[s] for s in live]
        toks = [int(streams[s][p]) for s, p in zip(live, pos)]
        logits, am = m.batch_forward(live, pos, toks)
        for i, (s, p) in enumerate(zip(live, pos)):
            _check(logits[i], refs[s][p])
            assert int(am[i]) == int(logits[i].argmax())
    assert m.stats().device_status == 0
    m.close()


@pytest.mark.parametrize("cfg", [ModelConfig(512, 1280, 2, 4, 2, 1000, 320, True),
                                 ModelConfig(512, 1280, 2, 8, 8, 1029, 320, False)], ids=["heads128", "heads64"])
def test_lengths_around_the_key_ranges(cfg):
    """Rounds of 32 keys per block, ranges of whole rounds, more ranges than a short sequence fills; alone and together."""
    lengths = [1, 7, 8, 31, 32, 33, 64, 96, 257, 300]
    tensors = _tensors(cfg, 21)
    stream = np.concatenate([[1], np.random.default_rng(22).integers(3, cfg.vocab_size, 300)]).astype(np.int32)
    refs = _alone(cfg, tensors, stream)
    m = _build(cfg, tensors)
    m.batch_create(len(lengths), 310)
    entries = [(s, p) for s, n in enumerate(lengths) for p in range(n)]
    for i in range(0, len(entries), 64):
        part = entries[i: i + 64]
        m.batch_forward([s for s, _ in part], [p for _, p in part], [int(stream[p]) for _, p in part], want_logits=False)
    for some in (list(range(len(lengths))), [8], [0], [5, 9], [3, 4, 8]):
        logits, am = m.batch_forward(some, [lengths[s] for s in some], [int(stream[lengths[s]]) for s in some])
        for i, s in enumerate(some):
            _check(logits[i], refs[lengths[s]])
            assert int(am[i]) == int(logits[i].argmax())
    assert m.stats().device_status == 0
    m.close()


@pytest.mark.parametrize("heads", [4, 8])
def test_overlapped_launches_change_nothing(heads):
    """A prompt of two chunks and a step of three sequences with programmatic dependent launch and without: same bits."""
    cfg = ModelConfig(512, 1280, 3, heads, heads // 2, 1000, 512, True)
    tensors = _tensors(cfg, 23)
    toks = np.random.default_rng(24).integers(3, cfg.vocab_size, 300).astype(np.int32)
    got = []
    for flags in (0, L.F_NO_PDL):
        m = _build(cfg, tensors, flags)
        m.prefill(toks, 0)
        out = [m.read_buffer(which, cfg.kv_dim, 2, p) for which in (5, 6) for p in (0, 130, 299)]
        m.batch_create(3, 64)
        for p in range(3):
            out.append(m.batch_forward([0, 1, 2], [p] * 3, [int(t) for t in toks[3 * p: 3 * p + 3]])[0])
        assert m.stats().device_status == 0
        m.close()
        got.append(out)
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("vocab, entries", [(127, 1), (128, 2), (129, 33), (1000, 64), (19200, 31)])
def test_classifier_of_a_step(vocab, entries):
    """Vocabularies beside the 128-row tiles, one tile and more tiles than SMs, token counts beside the 32-token halves,
    against the decode path's classifier."""
    cfg = ModelConfig(512, 1280, 1, 8, 8, vocab, 64, False)
    tensors = _tensors(cfg, 25)
    toks = np.random.default_rng(26).integers(0, vocab, entries).astype(np.int32)
    m = _build(cfg, tensors)
    m.batch_create(entries, 8)
    logits, am = m.batch_forward(np.arange(entries), np.zeros(entries, dtype=np.int32), toks)
    assert np.array_equal(am, logits.argmax(axis=1))
    for i, t in enumerate(toks):
        _check(logits[i], m.forward(int(t), 0)[0])
    assert m.stats().device_status == 0
    m.close()


@pytest.mark.parametrize("dim, heads", [(768, 12), (4096, 32)])
def test_classifier_of_a_step_against_float64(dim, heads):
    """Operands in three bf16 pieces lose nothing that FP32 holds: against float64, with layers that add nothing, the error
    stays below half of what operands of two pieces would cost (rounded here, on the CPU, to 16 bits)."""
    cfg = ModelConfig(dim, 256, 1, heads, heads, 1500, 16, False)
    tensors = syn.synthetic_tensors(cfg, 3)
    for t in (L.T_WQ, L.T_WK, L.T_WV, L.T_WO, L.T_W1, L.T_W2, L.T_W3):
        tensors[t] = syn.quant_encode(np.zeros(cfg.tensor_floats(t), dtype=np.float32))
    wcls = np.random.default_rng(1).normal(0, 6 / np.sqrt(dim), (cfg.vocab_size, dim)).astype(np.float32)
    tensors[L.T_WCLS] = wcls.reshape(-1)
    m = _build(cfg, tensors)
    m.batch_create(64, 8)
    toks = np.arange(64, dtype=np.int32) * 7 + 3
    logits, _ = m.batch_forward(np.arange(64), np.zeros(64, dtype=np.int32), toks)
    assert m.stats().device_status == 0
    m.close()
    x = np.asarray(tensors[L.T_TOKEN_EMBEDDING], dtype=np.float64).reshape(cfg.vocab_size, dim)[toks]
    x = dequant(tensors[L.T_RMS_FINAL], dim) * (x / np.sqrt((x * x).mean(1, keepdims=True) + 1e-5))
    exact = x @ wcls.astype(np.float64).T
    two = pieces(x, 2) @ pieces(wcls, 2).T
    error = lambda y: np.linalg.norm(y - exact) / np.linalg.norm(exact)
    print(f"error {error(logits):.2e}, with two pieces {error(two):.2e}")
    assert error(logits) < 0.5 * error(two)


def test_classifier_weights_at_the_end_of_the_range():
    """Weights that are infinite, NaN, or finite but above the largest bf16 number (3.3895e38): the logits of the decode
    path's FP32 classifier, infinities with their sign."""
    cfg = ModelConfig(512, 1280, 1, 8, 8, 300, 64, False)
    tensors = _tensors(cfg, 27)
    # a final norm of 0.02: 3.4e38 times an element of x stays finite
    tensors[L.T_RMS_FINAL] = syn.quant_encode(np.full(cfg.dim, 0.02, dtype=np.float32))
    wcls = tensors[L.T_WCLS].reshape(cfg.vocab_size, cfg.dim).copy()
    wcls[3, 7], wcls[130, 500], wcls[200, 64] = np.inf, -np.inf, np.nan
    wcls[10, 100], wcls[299, 511], wcls[129, 0] = 3.4e38, -3.4e38, 3.39e38
    tensors[L.T_WCLS] = wcls.reshape(-1)
    m = _build(cfg, tensors)
    m.batch_create(5, 8)
    toks = np.array([3, 50, 99, 150, 299], dtype=np.int32)
    logits, _ = m.batch_forward(np.arange(5), np.zeros(5, dtype=np.int32), toks)
    for i, t in enumerate(toks):
        want = m.forward(int(t), 0)[0]
        assert np.isinf(want[[3, 130]]).all() and np.isnan(want[200]) and np.isfinite(want[[10, 129, 299]]).all()
        assert np.array_equal(logits[i][[3, 130]], want[[3, 130]]) and np.isnan(logits[i][200])
        big = [10, 129, 299]
        assert np.abs(logits[i][big] / want[big] - 1).max() < LOGIT_TOL
        rest = np.setdiff1d(np.arange(cfg.vocab_size), big + [3, 130, 200])
        _check(logits[i][rest], want[rest])
    assert m.stats().device_status == 0
    m.close()


def test_steps_right_behind_large_new_caches():
    """Caches of several GB are still being cleared when the first step is enqueued: it comes behind the clearing, so the
    rows it writes are there for the second step."""
    import torch
    cfg = ModelConfig(1024, 1280, 1, 8, 8, 300, 4096, True)
    m = _build(cfg, _tensors(cfg, 31))
    seqs = list(range(64))
    toks = np.random.default_rng(32).integers(3, cfg.vocab_size, (3, 64)).astype(np.int32)
    got = []
    for wait, n_seq in ((True, 64), (False, 256), (False, 384)):      # 8.6 GB per 256 sequences
        m.batch_create(n_seq, 4096)
        if wait:
            torch.cuda.synchronize()
        got.append([m.batch_forward(seqs, [p] * 64, toks[p])[0] for p in range(3)])
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)
    assert m.stats().device_status == 0
    m.close()


def test_short_wait_limit_does_not_count_the_kernels_in_front():
    """The classifier's blocks start while W2 (32 groups per block here, well over the limit of 20 us) still runs; their
    time limits start when it has ended."""
    cfg = ModelConfig(8192, 16384, 1, 64, 8, 1024, 16, False)
    m = Transformer(cfg)
    m.set_wait_limit_us(20)
    for t in L.QUANT_TENSORS:
        n = cfg.tensor_floats(t)
        m.upload_quant(t, syn.quant_encode(np.ones(n, dtype=np.float32)) if t in (L.T_RMS_ATT, L.T_RMS_FFN, L.T_RMS_FINAL)
                       else syn.synth_quant(n, 41, t))
    for t in (L.T_TOKEN_EMBEDDING, L.T_WCLS):
        m.upload_f32(t, syn.synth_f32(cfg.tensor_floats(t), 41, t))
    m.finalize()
    m.batch_create(64, 4)
    first = None
    for _ in range(5):
        logits, _ = m.batch_forward(list(range(64)), [0] * 64, list(range(64)))
        assert m.stats().device_status == 0
        first = logits if first is None else first
        assert np.array_equal(logits, first)
    m.close()


def test_workspaces_of_a_step_and_of_a_long_prompt():
    """A step needs the workspaces of 64 tokens only; a longer prompt replaces them by larger ones, behind which the steps
    (captured anew) compute the same bits."""
    import torch
    cfg = ModelConfig(4096, 11008, 1, 32, 4, 300, 512, True)
    m = Transformer(cfg)
    for t in L.QUANT_TENSORS:
        m.upload_quant(t, syn.synth_quant(cfg.tensor_floats(t), 42, t))
    m.upload_f32(L.T_TOKEN_EMBEDDING, syn.synth_f32(cfg.tensor_floats(L.T_TOKEN_EMBEDDING), 42, 0))
    m.finalize()
    toks = np.random.default_rng(43).integers(3, cfg.vocab_size, 300).astype(np.int32)
    free = torch.cuda.mem_get_info()[0]
    m.batch_create(2, 8)
    before = m.batch_forward([0, 1], [0, 0], toks[:2])[0]
    one_block = 64 * 4 * (3 * 2 * 11008 + 12 * (4096 + 64) + 2 * 4096 + 5120 + 192 * 11008 // 256)   # h13, parts, x and q, qkv, limbs
    assert free - torch.cuda.mem_get_info()[0] < 2 * one_block                # (the rest: kernels that are loaded, caches)
    m.prefill(toks, 0)
    after = m.batch_forward([0, 1], [0, 0], toks[:2])[0]
    assert np.array_equal(before, after)
    m.prefill(toks[:30], 300)
    assert np.array_equal(before, m.batch_forward([0, 1], [0, 0], toks[:2])[0])
    assert m.stats().device_status == 0
    m.close()


def test_full_batch_of_64_at_the_110m_shape():
    cfg = syn.SHAPES["stories110M"]
    tensors = _tensors(cfg, 13)
    rng = np.random.default_rng(14)
    steps = 6
    streams = [np.concatenate([[1], rng.integers(3, cfg.vocab_size, steps)]).astype(np.int32) for _ in range(64)]
    m = _build(cfg, tensors)
    m.batch_create(64, 16)
    last = None
    for p in range(steps):
        last, _ = m.batch_forward(np.arange(64), np.full(64, p), [int(s[p]) for s in streams])
    m.close()
    for s in (0, 17, 63):
        _check(last[s], _alone(cfg, tensors, streams[s][:steps])[-1])


def test_a_prompt_in_slices_beside_decoding_sequences(oracle):
    """One call carries 40 positions of a new sequence's prompt and one position each of two running
    sequences; the checker runs every sequence alone."""
    cfg = ModelConfig(256, 768, 2, 4, 4, 800, 128, True)
    tensors = _tensors(cfg, 15)
    rng = np.random.default_rng(16)
    a = np.concatenate([[1], rng.integers(3, 800, 10)]).astype(np.int32)
    b = np.concatenate([[1], rng.integers(3, 800, 10)]).astype(np.int32)
    c = np.concatenate([[1], rng.integers(3, 800, 45)]).astype(np.int32)
    m = _build(cfg, tensors)
    m.batch_create(3, 64)
    for p in range(9):
        m.batch_forward([0, 1], [p, p], [int(a[p]), int(b[p])], want_logits=False)
    seq = [0, 1] + [2] * 40
    pos = [9, 9] + list(range(40))
    tok = [int(a[9]), int(b[9])] + [int(t) for t in c[:40]]
    logits, _ = m.batch_forward(seq, pos, tok)
    nxt, _ = m.batch_forward([2], [40], [int(c[40])])
    m.close()

    def checker(stream):
        om = oracle.OracleModel(cfg, tensors, oracle.SILU_EXACT, oracle.SOFTMAX_REFERENCE)
        out = [om.forward(int(t), p).copy() for p, t in enumerate(stream)]
        om.close()
        return out

    for got, ref in ((logits[0], checker(a[:10])[-1]), (logits[1], checker(b[:10])[-1]), (logits[41], checker(c[:40])[-1]),
                     (nxt[0], checker(c[:41])[-1])):
        span = float(ref.max() - ref.min())
        assert float(np.abs(got - ref).max()) / span < ORACLE_TOL
        assert int(got.argmax()) == int(ref.argmax())


def test_batch_argument_checks():
    cfg = ModelConfig(256, 768, 2, 4, 4, 500, 64, True)
    m = _build(cfg, _tensors(cfg, 17))
    with pytest.raises(L.L2jError):
        m.batch_forward([0], [0], [1])                       # before batch_create
    m.batch_create(2, 32)
    for seq, pos, tok in (([2], [0], [1]), ([0], [32], [1]), ([0], [0], [500]), ([0, 0], [3, 3], [1, 1])):
        with pytest.raises(L.L2jError):
            m.batch_forward(seq, pos, tok)
    m.batch_forward([], [], [])
    m.close()
    small = syn.SHAPES["stories15M"]
    s = _build(small, _tensors(small, 18))
    with pytest.raises(L.L2jError):
        s.batch_create(2, 32)                                 # rows that straddle quantisation groups
    s.close()
