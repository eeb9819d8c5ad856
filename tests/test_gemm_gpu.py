"""-m gpu: the tcgen05 GEMM of the batched path alone, against numpy on the same bf16 inputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rand_bf16(rng, shape, scale=1.0):
    import synth
    return synth.f32_to_bf16((rng.standard_normal(shape, dtype=np.float32) * scale).reshape(-1)).reshape(shape)


def _ref(X, W):
    import synth
    return synth.bf16_to_f32(X).astype(np.float64) @ synth.bf16_to_f32(W).astype(np.float64).T


@pytest.mark.parametrize("T,N,K", [(1, 128, 64), (5, 256, 128), (16, 384, 448), (17, 1000, 896), (64, 1152, 896),
                                   (100, 640, 256), (200, 448, 608), (300, 896, 4864), (513, 256, 64),
                                   # few wide tiles, short K: split 8 ways into clusters whose rings are then cut back so
                                   # that all of them are resident at once (the parked plane must still fit the ring)
                                   (512, 896, 896), (256, 1152, 896), (130, 896, 896), (32, 2304, 3584),
                                   # long K with more tiles than 16 splits have room for; many tiles of a short K
                                   (64, 2048, 6144), (40, 1536, 8960), (4096, 1344, 384), (777, 2500, 104)])
def test_gemm_matches_numpy(T, N, K):
    import tffn
    rng = np.random.default_rng([T, N, K])
    X, W = _rand_bf16(rng, (T, K)), _rand_bf16(rng, (N, K), 0.05)
    out = tffn.op_gemm(X, W)
    ref = _ref(X, W)
    err = np.abs(out - ref).max() / np.abs(ref).max()
    assert err < 2e-5, err  # fp32 accumulation of exact bf16 products


@pytest.mark.parametrize("splits", [1, 2, 4, 8, 16])
def test_gemm_split_k_is_deterministic(splits):
    import tffn
    rng = np.random.default_rng(99)
    X, W = _rand_bf16(rng, (48, 1024)), _rand_bf16(rng, (256, 1024), 0.05)
    a = tffn.op_gemm(X, W, splits=splits)
    b = tffn.op_gemm(X, W, splits=splits)
    assert (a == b).all()
    ref = _ref(X, W)
    assert np.abs(a - ref).max() / np.abs(ref).max() < 2e-5


def _ffn_ref(h, w, gate, up, down, eps):
    """numpy restatement of one FFN branch input/outputs in float64 with the bf16 rounding points of
    inference/src/model/qwen.cu:422-437 (rmsnorm -> bf16, gate/up -> bf16, act -> bf16, down fp32)"""
    import synth
    f, r = synth.bf16_to_f32, lambda x: synth.bf16_to_f32(synth.f32_to_bf16(np.asarray(x, dtype=np.float32)))
    x = f(h).astype(np.float64)
    xn = r(x * (1.0 / np.sqrt((x * x).mean() + eps)) * f(w))
    g, u = r(f(gate).astype(np.float64) @ xn), r(f(up).astype(np.float64) @ xn)
    act = r((g / (1.0 + np.exp(-g.astype(np.float64)))) * u)
    return f(down).astype(np.float64) @ act


@pytest.mark.parametrize("H,I,expert", [(256, 96, True), (896, 4864, True), (896, 4864, False), (448, 1216, True),
                                        (1536, 8960, True), (2048, 2752, True)])
def test_fused_bs1_ffn_kernel(H, I, expert):
    """the fused batch-1 SwiGLU kernel alone, at sizes where every CTA's ring wraps several times"""
    import synth
    import tffn
    rng = np.random.default_rng([H, I])
    h = _rand_bf16(rng, (H,))
    w = synth.f32_to_bf16(1.0 + 0.1 * rng.standard_normal(H, dtype=np.float32))
    mats = [[_rand_bf16(rng, s, 0.02) for s in ((I, H), (I, H), (H, I))] for _ in range(2)]
    pb, pe = tffn.pack_ffn(*mats[0]), tffn.pack_ffn(*mats[1])
    out = synth.bf16_to_f32(tffn.op_swiglu_bs1(h, w, pb, pe if expert else None, 0.1, 1e-6))
    ref = synth.bf16_to_f32(h).astype(np.float64) + _ffn_ref(h, w, *mats[0], 1e-6)
    if expert:
        ref = ref + 0.1 * _ffn_ref(h, w, *mats[1], 1e-6)
    scale = np.abs(ref).max()
    assert np.abs(out - ref).max() / scale <= 1e-2   # one bf16 ulp of the largest element is 0.8 %
    assert np.abs(out - ref).mean() / scale <= 1.5e-3
    again = synth.bf16_to_f32(tffn.op_swiglu_bs1(h, w, pb, pe if expert else None, 0.1, 1e-6))
    assert (again == out).all()  # fixed reduction order


# widths around what a lane holds (256 columns per piece; 12 warps up to 1 024, then 9), records around a ring's and a warp round's ends
@pytest.mark.parametrize("H,I,expert", [(64, 3, True), (64, 7001, False), (1024, 1730, True), (1088, 1297, False), (1280, 1300, True),
                                        (1792, 1153, False), (1920, 2000, True), (2048, 145, False)])
def test_fused_bs1_ffn_kernel_edges(H, I, expert):
    import synth
    import tffn
    rng = np.random.default_rng([H, I])
    h = _rand_bf16(rng, (H,))
    w = synth.f32_to_bf16(1.0 + 0.1 * rng.standard_normal(H, dtype=np.float32))
    mats = [[_rand_bf16(rng, s, 0.02) for s in ((I, H), (I, H), (H, I))] for _ in range(2)]
    pb, pe = tffn.pack_ffn(*mats[0]), tffn.pack_ffn(*mats[1])
    out = synth.bf16_to_f32(tffn.op_swiglu_bs1(h, w, pb, pe if expert else None, 0.1, 1e-6))
    ref = synth.bf16_to_f32(h).astype(np.float64) + _ffn_ref(h, w, *mats[0], 1e-6)
    if expert:
        ref = ref + 0.1 * _ffn_ref(h, w, *mats[1], 1e-6)
    scale = np.abs(ref).max()
    assert np.abs(out - ref).max() / scale <= 1e-2   # one bf16 ulp of the largest element is 0.8 %
    assert np.abs(out - ref).mean() / scale <= 1.5e-3
    again = synth.bf16_to_f32(tffn.op_swiglu_bs1(h, w, pb, pe if expert else None, 0.1, 1e-6))
    assert (again == out).all()  # fixed reduction order


# The same kernel inside a step, where its weights are requested in two portions (14 336 / H records at once, half as many with the
# expert): the rest of a ring short and long, ring rounds and rest, nothing left for the second portion, 9 and 12 warps
@pytest.mark.parametrize("H,heads,kv,I,expert", [(896, 14, 2, 4864, True), (896, 14, 2, 1160, True), (1024, 16, 4, 4328, False), (1088, 17, 17, 2600, True),
                                                 (1536, 12, 2, 1600, False), (2048, 16, 2, 648, True), (2048, 16, 2, 1184, False), (128, 2, 1, 17000, False)])
def test_bs1_ffn_in_two_portions(tmp_path, H, heads, kv, I, expert):
    """early starts (portions) and full dependencies (everything requested at once) give the same bits"""
    import synth
    import tffn
    shape = dict(hidden_size=H, num_hidden_layers=3, num_attention_heads=heads, num_key_value_heads=kv, intermediate_size=I, vocab_size=512,
                 tie_word_embeddings=True)
    cfg = synth.write_model(str(tmp_path), shape, seed=31, norm_jitter=0.1)
    e = None
    m = tffn.qwen_load(str(tmp_path))
    if expert:
        synth.write_expert(str(tmp_path / "expert.bin"), cfg, seed=32)
        e = tffn.checkpoint_load(str(tmp_path / "expert.bin"), m, 0.5)
    t = synth.prompts(1, 24, 3, 512)[0]
    rows = {}
    for mode in (0, 1, 2):
        s = tffn.Session(m, e, max_batch=1, max_seq=64)
        s.set_launch_mode(mode)
        s.prefill([t[:8]])
        rows[mode] = np.concatenate([s.decode_step(t[i:i + 1], want_logits=True)[1] for i in range(8, 24)])
        assert s.status() == 0
        s.free()
    assert np.isfinite(rows[0]).all()
    assert (rows[1] == rows[0]).all() and (rows[2] == rows[0]).all()
