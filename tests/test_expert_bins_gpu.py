"""-m gpu: launches of few rows with every row at the same experts. In bf16 the rows stand in one bin per expert (full bins of several
tiles, the others empty), at the ends of the tiles and of the bins, and in launches that use no bins; in fp32 the experts' weights are
streamed for a few rows at a time, several times for those with more."""
import numpy as np
import pytest

from rafilix_cases import LIMIT, Case, attention_layer, error, moe_mlp, rafilix_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("compute", ["bfloat16", "float32"])
@pytest.mark.parametrize("experts,top,identity", [(12, 2, 0), (40, 3, 2), (3, 3, 0)])
def test_full_and_empty_bins(tmp_path, experts, top, identity, compute):
    def edit(name, x):  # settles every choice
        if name.endswith("correction"):
            y = np.zeros_like(x)
            for i, e in enumerate([1, experts - 1, 0][:top]):
                y[e] = 8.0 - 2 * i
            return y
    c = Case(tmp_path, rafilix_config(64, 97, [attention_layer(2, 1, 16, 16, chunk=20, mlp=moe_mlp(experts, top, 40, identity=identity))]), edit=edit)
    t = c.tokens(140)
    want, _ = c.expect(t)
    s = c.session(compute, max_seq=160)
    for n in (1, 2, 15, 16, 17, 32, 33, 63, 64, 65, 127, 128, 129, 140):
        s.qwen_reset()
        e = error(s.qwen_forward(t[:n]), want[:n])
        assert e.max() <= LIMIT[compute], (n, float(e.max()))
    assert s.status() == 0
    s.free()


@pytest.mark.parametrize("compute", ["bfloat16", "float32"])
@pytest.mark.parametrize("experts,top,identity,live", [(12, 3, 0, [7]), (3, 3, 0, [2]), (5, 2, 1, []), (40, 4, 2, [5, 39]), (70, 6, 6, [69, 70])])
def test_fewer_live_experts_than_choices(tmp_path, experts, top, identity, live, compute):
    """corrections of -inf (retired experts) leave fewer entries than a token chooses: the first of the others are taken, each once"""
    def edit(name, x):
        if name.endswith("correction"):
            y = np.full_like(x, -np.inf)
            y[live] = x[live]
            return y
    c = Case(tmp_path, rafilix_config(64, 97, [attention_layer(2, 1, 16, 16, chunk=20, mlp=moe_mlp(experts, top, 40, identity=identity))]), edit=edit)
    t = c.tokens(130)
    want, _ = c.expect(t)
    s = c.session(compute, max_seq=160)
    for n in (1, 2, 3, 16, 17, 64, 65, 128, 130):
        s.qwen_reset()
        e = error(s.qwen_forward(t[:n]), want[:n])
        assert e.max() <= LIMIT[compute], (n, float(e.max()))
    assert s.status() == 0
    s.free()
