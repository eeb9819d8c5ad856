"""-m gpu: launches of few rows, whose norms ride in the products' epilogues (Qwen2) and whose feed-forward's first product shares
the mixer's launch (Razesun), at the ends of the token tiles and on both sides of the limit of 64 rows."""
import numpy as np
import pytest

from razesun_cases import LIMIT, Case, error, mixed_config

pytestmark = pytest.mark.gpu
ROWS = [2, 15, 16, 17, 31, 33, 63, 64, 65]


@pytest.mark.parametrize("name,expert", [("mini05", True), ("mini7", True), ("mini7", False), ("tiny128", True)])
def test_rows_of_a_prompt(model_dirs, name, expert):
    """one launch over n rows against the oracle (the bounds of test_parity_gpu.py)"""
    import oracle
    import synth
    import tffn
    d, ep, cfg = model_dirs[name]
    m = tffn.qwen_load(d)
    e = tffn.checkpoint_load(ep, m, 0.1) if expert else None
    s = tffn.Session(m, e, max_batch=1, max_seq=96)
    toks = synth.prompts(1, max(ROWS), 5, cfg["vocab_size"])[0]
    ref = oracle.Oracle(d, 96, ep if expert else None, 0.1).forward(toks)["logits"]
    for n in ROWS:
        s.qwen_reset()
        got = s.qwen_forward(toks[:n])
        scale = np.abs(ref[:n]).max()
        assert np.abs(got - ref[:n]).max() / scale <= 1.5e-2, n
        assert np.abs(got - ref[:n]).mean() / scale <= 2e-3, n


def test_razesun_rows_of_a_prompt(tmp_path):
    c = Case(tmp_path, mixed_config(), seed=3, sharp=1.5)
    t = c.tokens(max(ROWS))
    want = c.expect(t)[0]
    s = c.session("bfloat16", max_seq=96)
    for n in ROWS:
        s.qwen_reset()
        e = error(s.qwen_forward(t[:n]), want[:n])
        assert e.max() <= LIMIT["bfloat16"], (n, float(e.max()))
    s.free()


# 33 to 64 tokens and a long K: row tiles that sixteen 32-wide splits hold at once (9), one more (10), many (17), and a ragged K and N
@pytest.mark.parametrize("T", [33, 48, 64])
@pytest.mark.parametrize("N,K", [(1152, 4096), (1153, 4096), (2100, 4120), (130, 9000)])
def test_long_products_match_numpy(T, N, K):
    import synth
    import tffn
    rng = np.random.default_rng([T, N, K])
    X, W = (synth.f32_to_bf16((rng.standard_normal((n, K), dtype=np.float32) * s).reshape(-1)).reshape(n, K) for n, s in ((T, 1.0), (N, 0.05)))
    out = tffn.op_gemm(X, W)
    ref = synth.bf16_to_f32(X).astype(np.float64) @ synth.bf16_to_f32(W).astype(np.float64).T
    assert np.abs(out - ref).max() / np.abs(ref).max() < 2e-5  # fp32 accumulation of exact bf16 products
