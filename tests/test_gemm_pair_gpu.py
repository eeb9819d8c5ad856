"""-m gpu: the two-CTA GEMM tiles that prompts of more than 64 (gate|up) or 128 tokens run on, at the edges of their tiles:
alone against numpy, and every epilogue inside a model, whole prompts against the same prompts in small portions (which run
on the one-CTA tiles)."""
import numpy as np
import pytest

from rafilix_cases import LIMIT, Case, attention_layer, error, moe_mlp, rafilix_config

pytestmark = pytest.mark.gpu


def _rand_bf16(rng, shape, scale=1.0):
    import synth
    return synth.f32_to_bf16((rng.standard_normal(shape, dtype=np.float32) * scale).reshape(-1)).reshape(shape)


# tokens around 128 and 256, weight rows around 128 and 256 and not a multiple of 4, K not a multiple of 64 and longer than
# the ring, more tiles than pairs of SMs, a router's single row tile
@pytest.mark.parametrize("T,N,K", [(129, 136, 64), (255, 256, 72), (256, 255, 512), (257, 257, 1000), (384, 1030, 904), (1000, 130, 8),
                                   (2048, 60, 136), (4000, 1152, 896), (2500, 3000, 640), (2300, 896, 4864)])
def test_tiles_match_numpy(T, N, K):
    import synth
    import tffn
    rng = np.random.default_rng([T, N, K])
    X, W = _rand_bf16(rng, (T, K)), _rand_bf16(rng, (N, K), 0.05)
    out = tffn.op_gemm(X, W)
    ref = synth.bf16_to_f32(X).astype(np.float64) @ synth.bf16_to_f32(W).astype(np.float64).T
    assert np.abs(out - ref).max() / np.abs(ref).max() < 2e-5  # fp32 accumulation of exact bf16 products
    assert (tffn.op_gemm(X, W) == out).all()


# tiles in parts of K: all 36 in two, all 22 in three, the last six of 80 in four and three, the last eight of 82 in three; K and
# N not multiples of a block or a tile; then few tiles of a long K on both sides of where the one-CTA tiles' clusters end
@pytest.mark.parametrize("T,N,K", [(2300, 896, 4864), (2600, 300, 6000), (5000, 1024, 3000), (4865, 1000, 1800), (10400, 500, 2400),
                                   (129, 2048, 10800), (131, 2048, 10816), (256, 1500, 17920), (400, 896, 9728), (700, 900, 9728)])
def test_split_tiles_match_numpy(T, N, K):
    test_tiles_match_numpy(T, N, K)


def test_split_tiles_of_two_operand_pairs(tmp_path):
    """down projections of base and expert in parts that hold the one pair, the other, or both: a prompt of 4 100 rows (16 tiles of
    128 k-blocks in a launch, four parts each, and one of 4 rows) against the same in small portions"""
    import synth
    import tffn
    shape = dict(hidden_size=256, num_hidden_layers=1, num_attention_heads=4, num_key_value_heads=2, intermediate_size=4096, vocab_size=512,
                 tie_word_embeddings=True)
    cfg = synth.write_model(str(tmp_path), shape, seed=21, norm_jitter=0.1)
    synth.write_expert(str(tmp_path / "expert.bin"), cfg, seed=22)
    m = tffn.qwen_load(str(tmp_path))
    e = tffn.checkpoint_load(str(tmp_path / "expert.bin"), m, 0.5)
    t = synth.prompts(1, 4100, 3, 512)[0]
    got, want = [], []
    for out, cuts in ((got, [4100]), (want, [100] * 41)):
        s = tffn.Session(m, e, max_batch=1, max_seq=4160)
        at = 0
        for n in cuts:
            out.append(s.qwen_forward(t[at:at + n]))
            at += n
        s.free()
    got, want = np.concatenate(got), np.concatenate(want)
    err = np.abs(got - want) / np.abs(want).max()
    assert err.max() <= 1.5e-2 and err.mean() <= 2e-3  # as below


@pytest.mark.parametrize("name", ["mini05", "tiny128", "mini7"])
@pytest.mark.parametrize("expert", [False, True])
def test_prompts_whole_and_in_portions(model_dirs, name, expert):
    """q|k|v with bias, rotation and page writes on 64- and 128-wide heads, residual products of one and two operand pairs,
    SwiGLU of one and two problems. Both runs round at the same points and sum in fp32; what differs is single bf16 flips,
    which move a logit by up to 1.5e-2 of the largest and a row by 2e-3 on average (as against the oracle)."""
    import tffn
    d, ep, cfg = model_dirs[name]
    m = tffn.qwen_load(d)
    e = tffn.checkpoint_load(ep, m, 0.1) if expert else None
    rng = np.random.default_rng(5)
    prompts = [rng.integers(0, cfg["vocab_size"], n).astype(np.int32) for n in (300, 1, 129, 777, 64)]
    whole = tffn.Session(m, e, max_batch=5, max_seq=800)
    parts = tffn.Session(m, e, max_batch=5, max_seq=800)
    got = whole.prefill(prompts, want_logits=True)[1]
    for i, p in enumerate(prompts):
        want = [parts.qwen_forward(p[k:k + 64], slot=i) for k in range(0, len(p), 64)][-1][-1]
        err = np.abs(got[i] - want) / np.abs(want).max()
        assert err.max() <= 1.5e-2 and err.mean() <= 2e-3, (i, err.max(), err.mean())
    a, b = (s.decode_step([3] * 5, want_logits=True)[1] for s in (whole, parts))  # reads every page the prompts wrote
    err = np.abs(a - b) / np.abs(b).max()
    assert err.max() <= 1.5e-2 and err.mean() <= 2e-3
    assert whole.status() == 0
    for x in (whole, parts):
        x.free()


def test_experts_of_many_rows(tmp_path):
    """grouped launches, groups of three 256-row tiles (the last one of 8 rows) and empty ones: squared ReLU and plain epilogues"""
    def edit(name, x):  # corrections that settle the choices: near ties would be decided by rounding
        return np.array([3.0, 2.0, 0.0, 1.0, -1.0]) if name.endswith("correction") else None
    c = Case(tmp_path, rafilix_config(64, 97, [attention_layer(2, 1, 16, 16, chunk=20, mlp=moe_mlp(5, 2, 136))]), edit=edit)
    t = c.tokens(520)
    want, _ = c.expect(t)
    s = c.session("bfloat16", max_seq=544)
    assert error(s.qwen_forward(t), want).max() <= LIMIT["bfloat16"]
    s.qwen_reset()
    last = s.prefill([t], want_logits=True)[1]
    assert error(last, want[-1:]).max() <= LIMIT["bfloat16"]
    assert s.status() == 0
    s.free()
