"""-m gpu: the delta rule's scan with few and many sequences in a launch, which gives a lane one to eight value columns, with one decay
per head and one per channel, on heads of 32 to 256 key channels and of columns that are no multiple of anything."""
import pytest

import rafilix_cases as rafilix
import razesun_cases as razesun
from synth import channel_delta_layer, delta_layer, razesun_config, rafilix_config

pytestmark = pytest.mark.gpu
HEADS = [(2, 2, 32, 32), (2, 1, 64, 64), (3, 3, 90, 58), (2, 2, 128, 128), (1, 1, 200, 36)]


@pytest.mark.parametrize("n", [1, 3, 12, 40])
@pytest.mark.parametrize("heads", HEADS, ids=str)
@pytest.mark.parametrize("family", ["razesun", "rafilix"])
def test_sequences(tmp_path, family, heads, n):
    if family == "razesun":
        c = razesun.Case(tmp_path, razesun_config(48, 97, [delta_layer(*heads, conv=3, mlp=None)]))
    else:
        c = rafilix.Case(tmp_path, rafilix_config(48, 97, [channel_delta_layer(*heads, conv=3, mlp=None)]))
    steps = 2
    lens = [1 + (29 * i + 40) % 70 for i in range(n)]
    seqs = [c.tokens(k + steps, seed=i) for i, k in enumerate(lens)]
    s = c.session("float32", max_batch=n, max_seq=96)
    got = [s.prefill([q[:k] for q, k in zip(seqs, lens)], want_logits=True)[1].copy()]
    for j in range(steps):
        got.append(s.decode_step([q[k + j] for q, k in zip(seqs, lens)], want_logits=True)[1].copy())
    for i in sorted({0, n // 2, n - 1}):
        want = c.expect(seqs[i])
        want = want[0] if isinstance(want, tuple) else want
        for j in range(steps + 1):
            assert razesun.error(got[j][i:i + 1], want[lens[i] - 1 + j:lens[i] + j]).max() <= razesun.LIMIT["float32"], (i, j)
    assert s.status() == 0
    s.free()


# 2 160 rows in a launch: convolutions and unit vectors of eight (or four) tokens at a time, with ends of sequences inside such a run
@pytest.mark.parametrize("family,heads,conv", [("razesun", (10, 5, 32, 24), 4), ("rafilix", (10, 10, 64, 64), 3), ("rafilix", (8, 4, 72, 40), 2),
                                               ("razesun", (12, 6, 16, 128), 1), ("rafilix", (12, 4, 18, 22), 5)])
def test_long_launches(tmp_path, family, heads, conv):
    if family == "razesun":
        c = razesun.Case(tmp_path, razesun_config(48, 97, [delta_layer(*heads, conv=conv, mlp=None)]))
    else:
        c = rafilix.Case(tmp_path, rafilix_config(48, 97, [channel_delta_layer(*heads, conv=conv, mlp=None)]))
    seqs = [c.tokens(n, seed=i) for i, n in enumerate((851, 9, 500, 1, 799))]
    s = c.session("float32", max_batch=5, max_seq=864)
    got = s.prefill(seqs, want_logits=True)[1].copy()
    step = s.decode_step([3] * 5, want_logits=True)[1]
    for i in (1, 2, 4):
        want = c.expect(list(seqs[i]) + [3])
        want = want[0] if isinstance(want, tuple) else want
        assert razesun.error(got[i:i + 1], want[-2:-1]).max() <= razesun.LIMIT["float32"], i
        assert razesun.error(step[i:i + 1], want[-1:]).max() <= razesun.LIMIT["float32"], i
    assert s.status() == 0
    s.free()
