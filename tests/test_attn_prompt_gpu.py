"""-m gpu: the prompt attention tiles (128 / G tokens x G heads, 64 keys per step) at their edges: chunked, odd and very large
groups of heads against the 64-bit restatement, in two portions, and pages that were used before."""
import numpy as np
import pytest

from rafilix_cases import LIMIT, Case, attention_layer, error, rafilix_config

pytestmark = pytest.mark.gpu


# heads, kv heads, key and value width (padded to 64 or 128 columns; 16-byte and other output rows), chunk (0: all keys)
@pytest.mark.parametrize("heads,kv,dim,vdim,chunk", [(7, 1, 64, 64, 0), (6, 3, 24, 18, 70), (1, 1, 72, 128, 0), (9, 1, 128, 13, 100), (140, 1, 8, 8, 0),
                                                     (128, 2, 16, 40, 33)])
@pytest.mark.parametrize("n", [149, 191, 192, 193, 300])
def test_tiles_match_the_restatement(tmp_path_factory, heads, kv, dim, vdim, chunk, n):
    c = Case(tmp_path_factory.mktemp("m"), rafilix_config(64, 97, [attention_layer(heads, kv, dim, vdim, chunk=chunk or 4096)]), qk_norm=2.0)
    t = c.tokens(n + 150)
    want, _ = c.expect(t)
    s = c.session("bfloat16", max_batch=1, max_seq=480)
    first = s.qwen_forward(t[:n])
    rest = s.qwen_forward(t[n:])  # behind a cached prefix that ends anywhere in a page
    assert error(np.concatenate([first, rest]), want).max() <= LIMIT["bfloat16"]
    assert s.status() == 0
    s.free()


def test_ragged_batch(tmp_path_factory):
    """tiles of one and of a few tokens beside full ones, and the same prompts as a block per token"""
    c = Case(tmp_path_factory.mktemp("m"), rafilix_config(64, 97, [attention_layer(14, 2, 64, 64, chunk=100)]))
    prompts = [c.tokens(k, seed=k) for k in (1, 130, 2, 17, 18, 19, 64)]
    s = c.session("bfloat16", max_batch=7, max_seq=160)
    got = s.prefill(prompts, want_logits=True)[1]
    s.qwen_reset()
    for i, q in enumerate(prompts):
        want = c.expect(q)[0][-1:]
        alone = s.qwen_forward(q[:60], slot=i) if len(q) <= 60 else np.concatenate([s.qwen_forward(q[:60], slot=i), s.qwen_forward(q[60:], slot=i)])
        assert error(got[i:i + 1], want).max() <= LIMIT["bfloat16"] and error(alone[-1:], want).max() <= LIMIT["bfloat16"], i
    assert s.status() == 0
    s.free()


def test_pages_of_an_earlier_request(model_dirs):
    """what an earlier request left in a page, behind the keys of a later one, makes no difference at all"""
    import tffn
    d, _, cfg = model_dirs["mini05"]
    m = tffn.qwen_load(d)
    rng = np.random.default_rng(3)
    a, b = (rng.integers(0, cfg["vocab_size"], n).astype(np.int32) for n in (192, 165))
    used, fresh = (tffn.Session(m, None, max_batch=1, max_seq=192) for _ in range(2))
    used.prefill([a])
    used.qwen_reset()
    got, want = used.prefill([b], want_logits=True)[1], fresh.prefill([b], want_logits=True)[1]
    assert (got == want).all()
    for s in (used, fresh):
        s.free()


# context splits that are a cluster: 2, 4 and 8 of them, sequences that leave most of them empty, chunks that end inside one
@pytest.mark.parametrize("lens,chunk", [((511, 1), 0), ((1030, 1, 517), 0), ((2047, 2100), 700), ((300, 2049), 0)])
@pytest.mark.parametrize("dim,vdim", [(64, 64), (72, 128)])
def test_decode_over_split_contexts(tmp_path_factory, lens, chunk, dim, vdim):
    c = Case(tmp_path_factory.mktemp("m"), rafilix_config(64, 97, [attention_layer(14, 2, dim, vdim, chunk=chunk or 4096)]), qk_norm=2.0)
    rows = [c.tokens(n + 2, seed=n) for n in lens]
    s = c.session("bfloat16", max_batch=len(lens), max_seq=2112)
    s.prefill([r[:-2] for r in rows])
    got = [s.decode_step([r[k] for r in rows], want_logits=True)[1] for k in (-2, -1)]
    for i, r in enumerate(rows):
        want = c.expect(r)[0][-2:]
        assert error(np.stack([g[i] for g in got]), want).max() <= LIMIT["bfloat16"], i
    assert s.status() == 0
    s.free()
