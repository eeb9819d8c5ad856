"""-m gpu: decode attention through every way of merging context splits (none, clusters, the workspace's two forms) at one long
context, against the 64-bit restatement of its last rows."""
import numpy as np
import pytest

import rafilix_plain as plain
from rafilix_cases import LIMIT, Case, attention_layer, error, rafilix_config
from test_attention_cut_cpu import RESIDENT

pytestmark = pytest.mark.gpu
CTX, STEPS = 24000, 6


def last_rows(c, tokens, left_out=None):
    """logits of the last STEPS tokens of a model of one attention layer; left_out: keys (a slice) that no query sees"""
    layer, w, eps = c.plain_cfg["layers"][0], c.w, c.plain_cfg["norm"]["eps"]
    m, p = layer["mixer"], "l0.mix."
    H, G, dim = m["heads"], m["kv_heads"], m["dim"]
    x = w["embed"][tokens].astype(np.float64)
    h = plain.rms_norm(x, w["l0.norm1"], eps)
    k = plain.rms_norm((h @ w[p + "k"].T).reshape(-1, G, dim), w[p + "k.norm"], eps)
    k = np.stack([plain.rotate(k[t], t, m["rot"]) for t in range(len(tokens))])
    v = (h @ w[p + "v"].T).reshape(-1, G, m["vdim"])
    out = []
    for i in range(len(tokens) - STEPS, len(tokens)):
        q = plain.rotate(plain.rms_norm((h[i] @ w[p + "q"].T).reshape(H, dim), w[p + "q.norm"], eps), i, m["rot"])
        s = np.einsum("shd,hd->sh", np.repeat(k[:i + 1], H // G, 1), q) * m["scale"]
        if left_out is not None:
            s[left_out] = -np.inf
        e = np.exp(s - s.max(0))
        out.append(np.einsum("sh,shd->hd", e / e.sum(0), np.repeat(v[:i + 1], H // G, 1)).ravel() @ w[p + "o"].T)
    x = x[-STEPS:] + plain.rms_norm(np.stack(out), w["l0.norm1b"], eps)
    return plain.rms_norm(x, w["final.norm"], eps) @ w["embed"].T


@pytest.fixture(scope="module")
def long_context(tmp_path_factory):
    c = Case(tmp_path_factory.mktemp("m"), rafilix_config(64, 97, [attention_layer(14, 2, 64, 64, chunk=32768)]), qk_norm=2.5)
    t = c.tokens(CTX + STEPS, seed=3)
    want = last_rows(c, t)
    for z in (0, 7, 23):  # a split that is not merged would be seen
        assert error(last_rows(c, t, slice(1000 * z, 1000 * z + 1000)), want).max() > 2 * LIMIT["bfloat16"], z
    return c, t, want


# sequences (all but one are short), splits, whether they are a cluster
@pytest.mark.parametrize("n,splits,cluster", [(1, 24, False), (5, 14, False), (8, 9, False), (12, 5, True), (24, 3, False), (40, 1, False)])
def test_every_way_of_merging(long_context, n, splits, cluster):
    import tffn
    c, t, want = long_context
    assert tffn.attention_cut(n, 14, 2, 64, CTX + 1, 148, RESIDENT) == (splits, cluster)
    s = c.session("bfloat16", max_batch=n, max_seq=CTX + 64)
    s.prefill([t[:CTX]] + [t[i:i + 1] for i in range(1, n)])
    got = [s.decode_step(np.full(n, x), want_logits=True)[1][0] for x in t[CTX:]]
    assert error(np.stack(got), want).max() <= LIMIT["bfloat16"]
    assert s.status() == 0
    s.free()
