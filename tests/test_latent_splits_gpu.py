"""-m gpu: latent attention decode at the context lengths where its splits change: 2, 4, 8 and 16 of a cluster, the short ring of few
tiles and the deep one, one and several sequences; and where they go through the workspace."""
import numpy as np
import pytest

from razesun_cases import LIMIT, Case, error, latent_layer, plant_key, razesun_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [(255,), (257,), (1030,), (2050,), (3500, 300), (2100, 1, 511)])
@pytest.mark.parametrize("rank,rot,heads", [(512, 64, 16), (72, 16, 5), (256, 32, 20)])
def test_decode_over_split_contexts(tmp_path_factory, lens, rank, rot, heads):
    c = Case(tmp_path_factory.mktemp("m"), razesun_config(64, 97, [latent_layer(heads, 16, rot, 16, rank, 32)]), sharp=2.0)
    rows = [c.tokens(n + 2, seed=n) for n in lens]
    s = c.session("bfloat16", max_batch=len(lens), max_seq=3520)
    s.prefill([r[:-2] for r in rows])
    got = [s.decode_step([r[k] for r in rows], want_logits=True)[1] for k in (-2, -1)]
    for i, r in enumerate(rows):
        assert error(np.stack([g[i] for g in got]), c.expect(r, last=2)[0]).max() <= LIMIT["bfloat16"], i
    assert s.status() == 0
    s.free()


# splits through the workspace: more than sixteen of one context, more than eight of four sequences' longest; a cluster of sixteen
@pytest.mark.parametrize("lens,splits,cluster", [((9300,), 18, False), ((4750, 1, 1, 1), 9, False), ((4750,), 16, True)])
def test_one_key_in_any_split(tmp_path, lens, splits, cluster):
    """a key in the first, in a middle and in the last split that the last query alone asks for"""
    import tffn
    c, key, ask, other = plant_key(tmp_path)
    for m in (layer["mixer"] for layer in c.cfg["layers"]):
        assert tffn.latent_attention_cut(len(lens), m["heads"], m["kv_rank"], m["rot_dim"], lens[0], 148)[:2] == (splits, cluster)
    filler = c.tokens(lens[0], seed=6)
    filler[np.isin(filler, [key, ask])] = other
    s = c.session("bfloat16", max_batch=len(lens), max_seq=lens[0] + 20)
    for kpos in (3, lens[0] // 2, lens[0] - 50):
        t = filler.copy()
        t[kpos], t[-1] = key, ask
        want = c.expect(t, last=1)[0]
        s.qwen_reset()
        s.prefill([t[:-1]] + [t[:1]] * (len(lens) - 1))
        got = s.decode_step([t[-1]] + [other] * (len(lens) - 1), want_logits=True)[1][:1]
        assert error(got, want).max() <= LIMIT["bfloat16"], kpos
        t[kpos] = other
        assert error(c.expect(t, last=1)[0], want)[0] > 3 * LIMIT["bfloat16"]  # the plant is seen
    assert s.status() == 0
    s.free()
