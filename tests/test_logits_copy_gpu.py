"""-m gpu: logits of 16 MB or more for memory that is not pinned are copied in chunks by several threads."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_copies_equal_small_ones(tmp_path):
    import synth
    import tffn
    V = 70001
    synth.write_model(str(tmp_path), dict(hidden_size=128, num_hidden_layers=1, num_attention_heads=2, num_key_value_heads=1, intermediate_size=256,
                                          vocab_size=V, tie_word_embeddings=True), seed=3)
    m = tffn.qwen_load(str(tmp_path))
    t = synth.prompts(1, 60, 3, V)[0]
    problems = []

    def run():
        s = tffn.Session(m, None, max_batch=1, max_seq=96)
        small = s.qwen_forward(t[:58])  # 58 x V x 4 bytes: one plain copy; the same tiles of the same products
        for _ in range(3):
            s.qwen_reset()
            large = s.qwen_forward(t)
            if not (large[:58] == small).all() or not np.isfinite(large).all():
                problems.append("rows differ")
        s.qwen_reset()
        if not (s.qwen_forward(t[:58]) == small).all():
            problems.append("plain copy after a staged one")
        s.free()

    threads = [threading.Thread(target=run) for _ in range(2)]
    for x in threads:
        x.start()
    for x in threads:
        x.join()
    assert not problems, problems


# bytes: 16 MB; 25 MB; 18 MB and 4 bytes; 16 MB and a chunk of 23 KB. Destinations at the start of a page and inside one
@pytest.mark.parametrize("V,rows,offset", [(65536, 64, 0), (65536, 100, 1), (44099, 107, 0), (44099, 107, 777), (70001, 60, 5)])
def test_every_byte(tmp_path, V, rows, offset):
    """the same rows through a plain copy into pinned memory; a poisoned destination with guards around it"""
    import synth
    import tffn
    import torch
    synth.write_model(str(tmp_path), dict(hidden_size=128, num_hidden_layers=1, num_attention_heads=2, num_key_value_heads=1, intermediate_size=256,
                                          vocab_size=V, tie_word_embeddings=True), seed=5)
    m = tffn.qwen_load(str(tmp_path))
    s = tffn.Session(m, None, max_batch=1, max_seq=128)
    t = np.ascontiguousarray(synth.prompts(1, rows, 9, V)[0], dtype=np.int32)
    n, poison, guard = rows * V, np.float32(-12345.5), 1024
    pinned = torch.empty(n, dtype=torch.float32, pin_memory=True).numpy()
    pages = np.full(n + 3 * guard + 1024, poison, dtype=np.float32)
    skip = -pages.ctypes.data % 4096 // 4 + guard + offset  # guard: a page
    out = pages[skip:skip + n]
    for dst in (pinned, out):
        s.qwen_reset()
        tffn._check(tffn._L.tffn_forward(s._h, 0, t.ctypes.data, rows, dst.ctypes.data))
    assert np.isfinite(pinned).all() and not (pinned == poison).any()
    assert (out == pinned).all()
    assert (pages[:skip] == poison).all() and (pages[skip + n:] == poison).all()
    s.free()


PER_THREAD = 2  # the handle of CUDA's per-thread default stream: another stream in every thread that uses it


def test_per_thread_default_stream(tmp_path):
    """the same logits as on a stream of the session's own, of prompts and of steps that are not much shorter than their copy"""
    import synth
    import tffn
    V = 70001
    synth.write_model(str(tmp_path), dict(hidden_size=128, num_hidden_layers=12, num_attention_heads=2, num_key_value_heads=1, intermediate_size=1024,
                                          vocab_size=V, tie_word_embeddings=True), seed=4)
    m = tffn.qwen_load(str(tmp_path))
    prompts = [synth.prompts(1, 20, i, V)[0] for i in range(64)]
    got = []
    for stream in (None, PER_THREAD):
        s = tffn.Session(m, None, max_batch=64, max_seq=64, stream=stream)
        rows = [s.prefill(prompts, want_logits=True)[1].copy()]
        for k in range(6):
            rows.append(s.decode_step([(997 * i + 31 * k) % V for i in range(64)], want_logits=True)[1].copy())
        got.append(rows)
        assert s.status() == 0
        s.free()
    for a, b in zip(*got):
        assert (a == b).all()
