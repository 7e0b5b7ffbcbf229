"""The persistent kernel at the edges of its mapping, against the per-step kernels and a float64 model; when it is chosen; and
what it does beside other contexts.

Both kernels form the same products from the same 24-bit activations and add the FP32 group terms of a row in other orders; a row of g groups
is then off by at most about g roundings of 2^-24 of its terms, and two layers of them move a logit by a few 1e-6 of the range
(observed: 1e-6).  The bound is 1e-5."""
import threading

import numpy as np
import pytest

from llama2j_b200 import lib as L
from llama2j_b200 import synthetic as syn
from llama2j_b200.model_files import ModelConfig
from llama2j_b200.transformer import Transformer
from tests.np_model import NumpyModel

pytestmark = pytest.mark.gpu

TOL = 1e-5


def _build(cfg, tensors, flags):
    m = Transformer(cfg, 0, 0, None, flags)
    m.upload_all(tensors)
    m.finalize()
    assert m.launch_mode()["persistent"] == (flags == L.F_PERSISTENT)
    return m


# dim, hidden, heads, kv heads: one group per row and warps without one; groups that fill a warp and one more; head sizes 8 (more lane
# groups than lanes in the merge), 32, 64, 128; shared K/V heads; rows of 56 groups (all consumer warps on one set of rows)
SHAPES = [(256, 512, 32, 32), (512, 1280, 16, 4), (1024, 1280, 8, 8), (1280, 2304, 10, 2), (768, 14336, 12, 12), (4096, 2816, 32, 8)]


@pytest.mark.parametrize("dim,hidden,heads,kv", SHAPES)
def test_against_step_kernels(dim, hidden, heads, kv):
    cfg = ModelConfig(dim=dim, hidden_dim=hidden, n_layers=2, n_heads=heads, n_kv_heads=kv, vocab_size=500, seq_len=800,
                      shared_classifier=True)
    tensors = syn.synthetic_tensors(cfg, 8)
    rng = np.random.default_rng(9)
    for t in (L.T_RMS_ATT, L.T_RMS_FFN, L.T_RMS_FINAL):
        tensors[t] = syn.quant_encode(rng.uniform(0.5, 1.5, cfg.tensor_floats(t)).astype(np.float32))
    a, b = _build(cfg, tensors, L.F_PERSISTENT), _build(cfg, tensors, L.F_STEP_KERNELS)
    # ends of attention units (32 positions), of the short regime (512), positions whose partials come from several blocks
    check = {0, 1, 30, 31, 32, 33, 63, 64, 127, 128, 129, 255, 256, 510, 511, 512, 513, 640, 799}
    for p in range(800):
        tok = int(rng.integers(3, cfg.vocab_size))
        want = p in check
        x, _ = a.forward(tok, p, want_logits=want)
        y, _ = b.forward(tok, p, want_logits=want)
        if want:
            assert float(np.abs(x - y).max()) <= TOL * float(y.max() - y.min()), p
    # what the launch leaves behind for readers
    for which, n in ((0, dim), (1, dim), (2, dim), (3, hidden)):      # x, the attention output, q, the hidden vector
        x, y = a.read_buffer(which, n), b.read_buffer(which, n)
        assert float(np.abs(x - y).max()) <= TOL * float(np.abs(y).max()), which
    assert a.stats().device_status == 0
    a.close()
    b.close()


@pytest.mark.parametrize("dim,hidden,heads,kv", SHAPES[:4])
def test_against_float64(dim, hidden, heads, kv):
    """Every position of two attention units and a bit.  An activation is held to 2^-23 of its group's largest element and a row sum
    adds some ten FP32 terms: a few 1e-7 of the range per matrix, eight of them in a row."""
    cfg = ModelConfig(dim=dim, hidden_dim=hidden, n_layers=2, n_heads=heads, n_kv_heads=kv, vocab_size=500, seq_len=70, shared_classifier=True)
    tensors = syn.synthetic_tensors(cfg, 15)
    m, ref = _build(cfg, tensors, L.F_PERSISTENT), NumpyModel(cfg, tensors)
    for p, tok in enumerate(syn.synthetic_prompt(70, 16, cfg.vocab_size)):
        x, y = m.forward(int(tok), p)[0], ref.forward(int(tok), p)
        assert float(np.abs(x - y).max()) <= TOL * float(y.max() - y.min()), p
    m.close()


@pytest.mark.parametrize("value", [1e-30, 3e37, np.inf, np.nan])
def test_embedding_at_the_ends_of_the_range(value):
    """Tiny and huge activations through the fixed-point conversion: finite where the per-step kernels are, not finite where they are not."""
    cfg = ModelConfig(dim=512, hidden_dim=1280, n_layers=2, n_heads=4, n_kv_heads=4, vocab_size=300, seq_len=16, shared_classifier=False)
    tensors = syn.synthetic_tensors(cfg, 10)
    emb = np.array(tensors[L.T_TOKEN_EMBEDDING], dtype=np.float32).reshape(cfg.vocab_size, cfg.dim)
    emb[5, 7] = value
    tensors[L.T_TOKEN_EMBEDDING] = emb.reshape(-1)
    a, b = _build(cfg, tensors, L.F_PERSISTENT), _build(cfg, tensors, L.F_STEP_KERNELS)
    x, y = a.forward(5, 0)[0].copy(), b.forward(5, 0)[0].copy()
    if np.isfinite(y).all():
        span = max(float(y.max() - y.min()), 1e-30)
        assert float(np.abs(x - y).max()) <= 1e-4 * span      # one element decides the group's scale
    else:
        assert np.array_equal(np.isnan(x), np.isnan(y))
    a.close()
    b.close()


@pytest.mark.parametrize("name,value", [("L2J_CHAIN", "0"), ("L2J_BLOCKS_PER_SM", "2")])
@pytest.mark.parametrize("flags", [0, L.F_PERSISTENT])
def test_switches_that_take_away_what_the_kernel_needs(monkeypatch, name, value, flags):
    """No forward counter, or more blocks than are resident at once: the context runs the per-step kernels, with their bits."""
    cfg = ModelConfig(dim=1280, hidden_dim=2304, n_layers=2, n_heads=10, n_kv_heads=2, vocab_size=500, seq_len=16, shared_classifier=True)
    tensors = syn.synthetic_tensors(cfg, 11)
    monkeypatch.setenv(name, value)
    a, b = (Transformer(cfg, 0, 0, None, f) for f in (flags, L.F_STEP_KERNELS))
    assert not a.launch_mode()["persistent"]
    for m in (a, b):
        m.upload_all(tensors)
        m.finalize()
    for p, t in enumerate((1, 17, 400)):
        assert np.array_equal(a.forward(t, p)[0], b.forward(t, p)[0])
    assert a.stats().device_status == 0
    a.close()
    b.close()


@pytest.mark.parametrize("dim,heads,persistent", [(768, 12, False), (1024, 8, True), (1536, 12, True), (2560, 20, True), (7168, 56, True),
                                                  (7424, 58, False), (8192, 64, False)])
def test_which_kernel_is_the_default(dim, heads, persistent):
    """From dim 1024 on, as long as a row leaves room for two sets of consumer warps (28 groups)."""
    cfg = ModelConfig(dim=dim, hidden_dim=2816, n_layers=1, n_heads=heads, n_kv_heads=heads, vocab_size=256, seq_len=8, shared_classifier=True)
    for flags, want in ((0, persistent), (L.F_PERSISTENT, True), (L.F_STEP_KERNELS, False)):
        m = Transformer(cfg, 0, 0, None, flags)
        assert m.launch_mode()["persistent"] == want
        m.close()


def test_contexts_that_work_at_the_same_time():
    """Two persistent kernels want all SMs, a prompt's kernels some of them: everybody gets what they get alone."""
    cfg = ModelConfig(dim=1280, hidden_dim=2816, n_layers=4, n_heads=10, n_kv_heads=10, vocab_size=2000, seq_len=512, shared_classifier=True)
    tensors = syn.synthetic_tensors(cfg, 12)
    prompt = syn.synthetic_prompt(300, 3, cfg.vocab_size)

    def greedy(m):
        m.reset()
        return m.generate_greedy(prompt[:8], 300)

    def host_loop(m):
        m.reset()
        return np.array([m.forward(int(prompt[p]), p)[0].copy() for p in range(200)])

    def prompts(m):
        m.reset()
        m.prefill(prompt, 0)
        return m.forward(7, prompt.size)[0].copy()

    jobs = [greedy, host_loop, prompts, greedy]
    models = []
    for _ in jobs:
        m = Transformer(cfg, 0)
        m.upload_all(tensors)
        m.finalize()
        models.append(m)
    assert models[0].launch_mode()["persistent"]
    alone = [job(m) for job, m in zip(jobs, models)]
    bad = []

    def work(i):
        try:
            for _ in range(4):
                if not np.array_equal(jobs[i](models[i]), alone[i]):
                    bad.append((i, "other results"))
        except L.L2jError as e:
            bad.append((i, str(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    for m in models:
        assert m.stats().device_status == 0
        m.close()


def test_more_bytes_per_token_than_31_bits_count():
    """Heads that share one K/V head read a long cache 32 times over: a block's ring takes more than 2^31 bytes in one token.  The keys
    and values of the last positions differ from zero; the bound is the prompt path's (305,000 FP32 terms per softmax sum)."""
    last = 305_000
    cfg = ModelConfig(dim=4096, hidden_dim=256, n_layers=32, n_heads=32, n_kv_heads=1, vocab_size=300, seq_len=last + 8, shared_classifier=True)
    assert cfg.n_layers * cfg.n_heads * last * 128 * 8 > 148 << 31
    rng = np.random.default_rng(13)
    data = {t: syn.synth_quant(cfg.tensor_floats(t) // cfg.n_layers, 14, t) for t in (L.T_WQ, L.T_WK, L.T_WV, L.T_WO, L.T_W1, L.T_W2, L.T_W3)}
    emb = syn.synth_f32(cfg.tensor_floats(L.T_TOKEN_EMBEDDING), 14, L.T_TOKEN_EMBEDDING)
    k, v = (rng.normal(0, s, (500, cfg.kv_dim)).astype(np.float32) for s in (1.0, 30.0))
    logits = []
    for flags in (L.F_STEP_KERNELS, 0):
        m = Transformer(cfg, 0, 0, None, flags)
        assert m.launch_mode()["persistent"] == (flags == 0)
        for t in L.QUANT_TENSORS:
            n = cfg.tensor_floats(t)
            if t not in data:
                m.upload_quant(t, syn.quant_encode(np.ones(n, dtype=np.float32)))
                continue
            for layer in range(cfg.n_layers):
                m.upload_quant(t, data[t], n // cfg.n_layers, layer * (n // cfg.n_layers))
        m.upload_f32(L.T_TOKEN_EMBEDDING, emb)
        m.finalize()
        for layer in range(cfg.n_layers):
            m.kv_write(layer, last - 500, k, v)
        logits.append(np.array([m.forward(7, last + i)[0].copy() for i in range(2)]))
        assert m.stats().device_status == 0
        m.close()
    assert float(np.abs(logits[0] - logits[1]).max()) <= 1e-4 * float(logits[0].max() - logits[0].min())
