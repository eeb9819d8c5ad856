"""-m gpu: the fp32 products at the edges of their two kernels (up to eight tokens; tiles of 64 tokens and 64 weight rows, K split
over a cluster where tiles are few), inside models that compute in fp32, against the 64-bit restatements."""
import numpy as np
import pytest

import rafilix_cases
import razesun_cases
from rafilix_cases import attention_layer, error, moe_mlp, rafilix_config
from razesun_cases import dense_mlp, delta_layer, razesun_config, rglru_layer

pytestmark = pytest.mark.gpu


def run(sess, tokens, sizes):
    out, at = [], 0
    for n in sizes:
        out.append(sess.qwen_forward(tokens[at:at + n]))
        at += n
    return np.concatenate(out)


# token counts around 1, 2, 4, 8 and 64; products of N not a multiple of 8 or 64 (vocabulary 211, 6 heads, 5-column parts),
# K not a multiple of 8 (52, 60) or of 32 (1 100, split over eight CTAs) and shorter than a team of 32 threads' pieces
@pytest.mark.parametrize("sizes", [[1, 2, 3, 4, 5, 7, 8, 9], [63], [64], [65, 1], [128, 8, 2], [200]])
def test_products_match_the_restatement(tmp_path_factory, sizes):
    c = razesun_cases.Case(tmp_path_factory.mktemp("m"), razesun_config(52, 211, [
        rglru_layer(60, 12, conv=2, mlp=dense_mlp(1100)), delta_layer(6, 2, 24, 40, mlp=dense_mlp(2056))]))
    t = c.tokens(sum(sizes))
    s = c.session("float32", max_seq=256)
    assert error(run(s, t, sizes), c.expect(t)[0]).max() <= razesun_cases.LIMIT["float32"]
    assert s.status() == 0
    s.free()


@pytest.mark.parametrize("sizes", [[1, 2, 5, 1], [70, 1]])
def test_grouped_products(tmp_path_factory, sizes):
    """the experts of a mixture: groups without rows, of a few rows and of more than a tile"""
    def edit(name, x):  # corrections that settle the choices
        return np.array([3.0, 2.0, 0.0, 1.0, -1.0]) if name.endswith("correction") else None
    c = rafilix_cases.Case(tmp_path_factory.mktemp("m"), rafilix_config(64, 97, [attention_layer(2, 1, 16, 16, chunk=20, mlp=moe_mlp(5, 2, 136))]), edit=edit)
    t = c.tokens(sum(sizes))
    want, _ = c.expect(t)
    s = c.session("float32", max_seq=128)
    assert error(run(s, t, sizes), want).max() <= rafilix_cases.LIMIT["float32"]
    s.free()
