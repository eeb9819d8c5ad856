"""-m gpu: latent attention decode at the context lengths where its splits change: 2, 4, 8 and 16 of a cluster, the short ring of few
tiles and the deep one, one and several sequences."""
import numpy as np
import pytest

from razesun_cases import LIMIT, Case, error, latent_layer, razesun_config

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
