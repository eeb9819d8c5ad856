"""A launch that can fail (a cluster that finds no room, a tensor map that cannot be encoded) must reach its caller: a call that
drops the launcher's result does not compile with the library's flags."""
import subprocess

import pytest

CALLS = {
    "launch_gemm": "launch_gemm(g, w, 0)",
    "launch_gemm_f32": "launch_gemm_f32(g, w, 0)",
    "launch_attention": "launch_attention(nullptr, kv, 0, nullptr, nullptr, nullptr, 1, 1, 1, a, 148, nullptr, 0)",
    "launch_attention_prefill": "launch_attention_prefill(nullptr, kv, 0, nullptr, nullptr, nullptr, nullptr, 1, nullptr, 1, 148, nullptr, nullptr, 0)",
    "launch_attention_latent": "launch_attention_latent(l, 1, 0, 1, a, 148, nullptr, 0, false)",
}


def compiles(tmp_path, statement):
    import build
    src = tmp_path / "call.cu"
    src.write_text('#include "kernels.h"\nnamespace tffn {\nint f(const GemmCall& g, const GemmWorkspace& w, KvView kv, AttnWorkspace a, const LatentAttn& l) {\n'
                   "    %s;\n    return 0;\n}\n}\n" % statement)
    r = subprocess.run([build.NVCC, *build.NVCC_FLAGS, "-I", build.CSRC, "-c", str(src), "-o", str(tmp_path / "call.o")], capture_output=True, text=True)
    return r.returncode == 0, r.stderr


@pytest.mark.parametrize("name", sorted(CALLS))
def test_a_dropped_result_does_not_compile(tmp_path, name):
    ok, messages = compiles(tmp_path, "return " + CALLS[name])
    assert ok, messages
    ok, messages = compiles(tmp_path, CALLS[name])
    assert not ok and "unused-result" in messages and name in messages
