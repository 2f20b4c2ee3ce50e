"""A bounded wait that ran out in any launch of a call makes that call fail.  The failure is the status word such a kernel
leaves, written from the host before the call."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "insignia_decode.hpp"
#include <cstdio>
#include <cstring>
using namespace insignia;
int main(int, char **argv)
{
    ModelFile model(argv[1]);
    Qwen35Weights w(model, 4ull << 30);
    DecodeOptions o;
    o.n_layers = 4;
    o.vocab = 64;
    DecodeWorkspace ws(64, nullptr, o);
    Qwen35Decode dec(w, ws);
    const int prompt[] = {3, 1, 4, 1, 5, 9, 2, 6, 5, 3}, drafts[] = {1, 2, 3, 4, 5, 6};
    auto call = [&](const char *name, auto &&f) {
        ws.reset();
        dec.forward_tokens(prompt, 10);
        dec.logits_argmax();
        for (int failed = 0; failed < 2; failed++) { // as it is; with the status word set
            cudaDeviceSynchronize();
            cudaMemcpy(ws.d_token + 3, &failed, sizeof failed, cudaMemcpyHostToDevice);
            const char *what = "returned";
            try {
                f();
            } catch (const std::exception &e) {
                what = std::strstr(e.what(), "bounded wait") ? "failed" : e.what();
            }
            std::printf("%s %d %s\n", name, failed, what);
        }
    };
    call("decode_token", [&] { dec.decode_token(7); });
    call("prompt", [&] { dec.forward_tokens(prompt, 10); dec.logits_argmax(); });
    call("generate", [&] { dec.generate(7, 3); });
    call("speculative", [&] { dec.generate_speculative(7, 6, nullptr, drafts); });
}
"""


def test_a_failed_wait_fails_the_call(cuda, golden_ckpt, tmp_path):
    src, exe, lib = str(tmp_path / "status.cpp"), str(tmp_path / "status"), os.path.join(ROOT, "insignia_b200", "lib")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.check_call(["nvcc", "-std=c++17", "-I", os.path.join(ROOT, "include"), src, "-L", lib, "-linsignia_b200", "-Xlinker", "-rpath", "-Xlinker", lib, "-o", exe])
    out = subprocess.run([exe, golden_ckpt[1]], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    got = [line.split(" ", 2) for line in out.stdout.strip().splitlines()]
    assert got == [[name, str(f), "failed" if f else "returned"] for name in ("decode_token", "prompt", "generate", "speculative") for f in (0, 1)]
