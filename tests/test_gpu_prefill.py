"""Batched prompt processing (l2j_prefill) against the decode path it replaces and against the CPU checker.

The reference pushes every prompt token through the decode step (Run.java:623-637); l2j_prefill runs up to
256 positions per sweep over the weights on the tensor cores.  Per position it computes the decode step's
arithmetic with the row sums added in another order, so the gates are tolerances, written here: the K/V
cache rows the prompt leaves behind within 1e-4 of the row's largest magnitude, and the logits of the decode
step after the prompt within 1e-4 of the logit range of the decode-only path (and within the 1e-3 of the
north star against the CPU checker), same arg-max.
"""
import numpy as np
import pytest

from llama2j_b200 import lib as L
from llama2j_b200 import synthetic as syn
from llama2j_b200.model_files import ModelConfig
from llama2j_b200.transformer import Transformer
from tests.np_model import bf16_pieces, dequant

pytestmark = pytest.mark.gpu

CACHE_TOL = 1e-4     # of the row's largest magnitude
LOGIT_TOL = 1e-4     # of the logit range, prefill + decode step against decode only
ORACLE_TOL = 1e-3    # of the logit range, against the CPU checker (north star)


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


def _inputs(cfg, n, seed=3):
    """BOS and then the prompt: the token fed at each of the first n positions (Run.java:614,635-637)."""
    return np.concatenate([[1], syn.synthetic_prompt(n - 1, seed, cfg.vocab_size)]).astype(np.int32)


def _compare_with_decode(cfg, tensors, n, positions, layers, next_token=7):
    toks = _inputs(cfg, n)
    dec = _build(cfg, tensors)
    for i in range(n):
        dec.forward(int(toks[i]), i, want_logits=False)
    pre = _build(cfg, tensors)
    pre.prefill(toks, 0)
    assert pre.prefill_launches() > 0, "the tensor-core path did not run"
    worst = 0.0
    for layer in layers:
        for pos in positions:
            for which in (5, 6):
                a = dec.read_buffer(which, cfg.kv_dim, layer, pos)
                b = pre.read_buffer(which, cfg.kv_dim, layer, pos)
                worst = max(worst, float(np.abs(a - b).max()) / float(np.abs(a).max()))
    ref = dec.forward(next_token, n)[0].copy()
    got = pre.forward(next_token, n)[0].copy()
    status = (dec.stats().device_status, pre.stats().device_status)
    dec.close()
    pre.close()
    assert status == (0, 0)
    assert worst < CACHE_TOL, worst
    span = float(ref.max() - ref.min())
    assert float(np.abs(got - ref).max()) / span < LOGIT_TOL
    assert int(got.argmax()) == int(ref.argmax())
    return got


def test_prefill_512_tokens_110m_shape():
    cfg = syn.SHAPES["stories110M"]      # head size 64, K/V rows of 768, three groups per row
    _compare_with_decode(cfg, _tensors(cfg, 1), 512, (0, 1, 63, 64, 300, 511), (0, 5, 11))


def test_prefill_512_tokens_7b_shape():
    cfg = syn.SHAPES["llama2-7b"]
    _compare_with_decode(cfg, _tensors(cfg, 2), 512, (0, 63, 64, 511), (0, 31))


def test_prefill_ragged_lengths_and_continuation():
    """Lengths that are not multiples of 64, a second call that continues at pos0 > 0, grouped-query heads."""
    cfg = ModelConfig(512, 1280, 3, 8, 2, 1000, 512, True)      # 8 query heads on 2 K/V heads of 64
    tensors = _tensors(cfg, 4)
    toks = _inputs(cfg, 203)
    dec = _build(cfg, tensors)
    for i in range(203):
        dec.forward(int(toks[i]), i, want_logits=False)
    ref = dec.forward(9, 203)[0].copy()
    for first in (1, 63, 65, 130):
        pre = _build(cfg, tensors)
        pre.prefill(toks[:first], 0)
        pre.prefill(toks[first:], first)
        got = pre.forward(9, 203)[0].copy()
        for pos in (0, first - 1, first, 202):
            a, b = dec.read_buffer(5, cfg.kv_dim, 2, pos), pre.read_buffer(5, cfg.kv_dim, 2, pos)
            assert float(np.abs(a - b).max()) / float(np.abs(a).max()) < CACHE_TOL, (first, pos)
        assert pre.stats().device_status == 0
        pre.close()
        assert float(np.abs(got - ref).max()) / float(ref.max() - ref.min()) < LOGIT_TOL, first
    dec.close()


@pytest.mark.parametrize("heads", [4, 8])                       # head sizes 128 and 64
@pytest.mark.parametrize("n", [1, 63, 129, 192, 256, 257, 321])
def test_prefill_lengths_around_the_blocks_of_a_chunk(n, heads):
    """Blocks of 64 tokens, chunks of 256: one token, one short of a block, two, three and four blocks, a second chunk."""
    cfg = ModelConfig(512, 1280, 2, heads, heads // 2, 1000, 512, True)
    positions = sorted({0, n // 2, n - 1} | {p for p in (63, 64, 128, 191, 255, 256) if p < n})
    _compare_with_decode(cfg, _tensors(cfg, 8), n, positions, (0, 1))


@pytest.mark.parametrize("heads, kv_heads", [(4, 2), (8, 8), (8, 2)])
@pytest.mark.parametrize("first, more", [(1, 1), (63, 2), (64, 64), (65, 127), (190, 131), (320, 180)])
def test_prefill_attention_around_its_tiles(heads, kv_heads, first, more):
    """Key tiles of 64, query blocks of 128, key ranges: a second call whose queries start and end beside their edges."""
    cfg = ModelConfig(512, 1280, 2, heads, kv_heads, 1000, 512, True)
    tensors = _tensors(cfg, 9)
    n = first + more
    toks = _inputs(cfg, n)
    dec = _build(cfg, tensors)
    for i in range(n):
        dec.forward(int(toks[i]), i, want_logits=False)
    pre = _build(cfg, tensors)
    pre.prefill(toks[:first], 0)
    pre.prefill(toks[first:], first)
    for pos in sorted({first, (first + n) // 2, n - 1}):
        for which in (5, 6):
            a, b = dec.read_buffer(which, cfg.kv_dim, 1, pos), pre.read_buffer(which, cfg.kv_dim, 1, pos)
            assert float(np.abs(a - b).max()) / float(np.abs(a).max()) < CACHE_TOL, (pos, which)
    assert pre.stats().device_status == 0
    dec.close()
    pre.close()


def _v_behind_attention(cfg, tensors, toks, k, v, rows, pieces=None):
    """float64: V rows of layer 1, from layer 0's embedded tokens, its attention over the cache rows given and what follows."""
    d, h, n_l, kv = cfg.dim, cfg.hidden_dim, cfg.n_layers, cfg.kv_dim
    n, hs, mul = len(toks), cfg.dim // cfg.n_heads, cfg.n_heads // cfg.n_kv_heads
    mat = lambda t, r, c: dequant(tensors[t], n_l * r * c).reshape(n_l, r, c)
    rms = lambda x, w: w * (x / np.sqrt((x * x).mean(-1, keepdims=True) + 1e-5))
    g_att, g_ffn = (dequant(tensors[t], n_l * d).reshape(n_l, d) for t in (L.T_RMS_ATT, L.T_RMS_FFN))
    x = np.asarray(tensors[L.T_TOKEN_EMBEDDING], dtype=np.float64).reshape(cfg.vocab_size, d)[toks]
    q = rms(x, g_att[0]) @ mat(L.T_WQ, d, d)[0].T
    i = np.arange(0, d, 2)
    angle = np.arange(n)[:, None] / 10000.0 ** ((i % hs) / hs)
    q[:, 0::2], q[:, 1::2] = (q[:, 0::2] * np.cos(angle) - q[:, 1::2] * np.sin(angle),
                              q[:, 0::2] * np.sin(angle) + q[:, 1::2] * np.cos(angle))
    x = x[rows]
    out = np.zeros((len(rows), d))
    for head in range(cfg.n_heads):
        cols, kvc = slice(head * hs, (head + 1) * hs), slice(head // mul * hs, (head // mul + 1) * hs)
        s = bf16_pieces(q[rows, cols] / np.sqrt(hs), pieces) @ bf16_pieces(k[:, kvc], pieces).T
        s = np.where(np.arange(n)[None, :] <= np.asarray(rows)[:, None], s, -np.inf)
        p = np.exp(s - s.max(-1, keepdims=True))
        out[:, cols] = bf16_pieces(p, pieces) @ bf16_pieces(v[:, kvc], pieces) / p.sum(-1, keepdims=True)
    x = x + out @ mat(L.T_WO, d, d)[0].T
    xb = rms(x, g_ffn[0])
    h1 = xb @ mat(L.T_W1, h, d)[0].T
    x = x + (h1 / (1 + np.exp(-h1)) * (xb @ mat(L.T_W3, h, d)[0].T)) @ mat(L.T_W2, d, h)[0].T
    return rms(x, g_att[1]) @ mat(L.T_WV, kv, d)[1].T


@pytest.mark.parametrize("heads, kv_heads, cuts", [(4, 2, ()), (8, 4, (200,))])
@pytest.mark.parametrize("scale", [1, 4])
def test_prefill_attention_against_float64(heads, kv_heads, cuts, scale):
    """Operands in three bf16 pieces lose nothing that FP32 holds.  The gate is what the pieces decide: with two of them
    the error against float64 (computed here, on the CPU) would be at least twice what is allowed.  `scale` sharpens the
    softmax: scores of about 1 and 16 times that."""
    cfg = ModelConfig(512, 1280, 2, heads, kv_heads, 1000, 512, True)
    tensors = _tensors(cfg, 12)
    rng = np.random.default_rng(13)
    for t in (L.T_WQ, L.T_WK):
        tensors[t] = syn.quant_encode(rng.normal(0, 0.02 * scale, cfg.tensor_floats(t)).astype(np.float32))
    toks = rng.integers(3, cfg.vocab_size, 330).astype(np.int32)
    m = _build(cfg, tensors)
    for a, b in zip((0, *cuts), (*cuts, len(toks))):
        m.prefill(toks[a:b], a)
    rows = [1, 63, 64, 127, 128, 199, 200, 255, 256, 329]
    got = np.stack([m.read_buffer(6, cfg.kv_dim, 1, p) for p in rows])
    k, v = (np.stack([m.read_buffer(which, cfg.kv_dim, 0, p) for p in range(len(toks))]) for which in (5, 6))
    assert m.stats().device_status == 0
    m.close()
    exact, two = (_v_behind_attention(cfg, tensors, toks, k, v, rows, pieces) for pieces in (None, 2))
    error = lambda x: np.linalg.norm(x - exact) / np.linalg.norm(exact)
    print(f"error {error(got):.2e}, with two pieces {error(two):.2e}")
    assert error(got) < 0.5 * error(two)


def test_a_smaller_shape_does_not_take_the_larger_ones_shared_memory():
    """Two contexts of one device in turn: a long row and a large vocabulary, then short ones, then the first again."""
    toks = np.random.default_rng(4).integers(3, 300, 70).astype(np.int32)
    models = []
    for hidden, vocab in ((5120, 30000), (512, 300)):
        cfg = ModelConfig(512, hidden, 1, 4, 4, vocab, 128, True)
        models.append(_build(cfg, _tensors(cfg, 10)))
    rounds = []
    for _ in range(2):
        got = []
        for m in models:
            m.reset()
            m.prefill(toks, 0)
            got.append(m.forward(7, toks.size)[0].copy())
            m.batch_create(2, 8)
            got.append(m.batch_forward([0, 1], [0, 0], [5, 6])[0])
            m.sampler_seed(1)
            got.append(m.sample(0.9, 0.9))
        rounds.append(got)
    for a, b in zip(*rounds):
        assert np.array_equal(a, b)
    for m in models:
        assert m.stats().device_status == 0
        m.close()


def test_prefill_then_decode_against_the_checker(oracle):
    """A 100-token prompt through l2j_prefill, then greedy decoding: logits of every decoded position within
    the north star's 1e-3 of range of the CPU checker that ran the whole sequence token by token."""
    cfg = ModelConfig(256, 768, 4, 4, 4, 2000, 256, True)
    tensors = _tensors(cfg, 5)
    toks = _inputs(cfg, 100)
    pre = _build(cfg, tensors)
    pre.prefill(toks, 0)
    om = oracle.OracleModel(cfg, tensors, oracle.SILU_EXACT, oracle.SOFTMAX_REFERENCE)
    for i in range(100):
        om.forward(int(toks[i]), i)
    token = 11
    for pos in range(100, 132):
        got = pre.forward(token, pos)[0].copy()
        ref = om.forward(token, pos).copy()
        span = float(ref.max() - ref.min())
        assert float(np.abs(got - ref).max()) / span < ORACLE_TOL, pos
        assert int(got.argmax()) == int(ref.argmax()), pos
        token = int(ref.argmax())
    om.close()
    pre.close()


def test_shapes_outside_the_tensor_core_path_use_the_decode_step():
    """Rows that straddle quantisation groups (15M shape): the prompt goes through the decode step, bitwise."""
    cfg = syn.SHAPES["stories15M"]
    tensors = _tensors(cfg, 6)
    toks = _inputs(cfg, 40)
    dec = _build(cfg, tensors)
    for i in range(40):
        dec.forward(int(toks[i]), i, want_logits=False)
    ref = dec.forward(5, 40)[0].copy()
    dec.close()
    pre = _build(cfg, tensors)
    pre.prefill(toks, 0)
    assert pre.prefill_launches() == 0
    got = pre.forward(5, 40)[0].copy()
    pre.close()
    assert np.array_equal(got, ref)


def test_prefill_argument_checks():
    cfg = ModelConfig(256, 768, 2, 4, 4, 500, 128, True)
    m = _build(cfg, _tensors(cfg, 7))
    with pytest.raises(L.L2jError):
        m.prefill(np.arange(3, 133, dtype=np.int32), 0)          # 130 positions in a sequence of 128
    with pytest.raises(L.L2jError):
        m.prefill(np.array([1, 500], dtype=np.int32), 0)          # token outside the vocabulary
    m.prefill(np.array([], dtype=np.int32), 0)
    m.close()
