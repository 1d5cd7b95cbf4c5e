"""CPU: the rule that splits the tensor-core adjoint's time axis into chunks
(blade_b200/csrc/adjoint_chunks.cuh), compiled on its own: every tile belongs to exactly
one non-empty chunk, and a block is never split worse than into one chunk per SM that its
channels leave it (sm_count / F chunks per channel), however few its channels are."""

import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
#include <cstdio>
#include "adjoint_chunks.cuh"
int main() {
    const uint64_t channels[] = {1, 2, 3, 5, 36, 74, 75, 100, 148, 149, 192, 300, 4096, 100000};
    const uint64_t tiles[] = {1, 2, 3, 7, 16, 63, 64, 65, 100, 147, 148, 149, 150, 511, 1024, 8192, 16777215};
    const uint64_t parts[] = {148, 132};
    for (uint64_t sms : parts)
        for (uint64_t F : channels)
            for (uint64_t n : tiles) {
                uint64_t nch = 0, tpc = 0;
                bb::adjoint_chunks(F, n, sms, nch, tpc);
                // one CTA per SM and channel share, as many as there are tiles
                uint64_t each = sms / F;
                if (each < 1) each = 1;
                if (each > n) each = n;
                const uint64_t per = (n + each - 1) / each, chunks = (n + per - 1) / per;
                const bool cover = nch >= 1 && nch * tpc >= n && (nch - 1) * tpc < n;
                if (!cover || bb::adjoint_chunk_cost(F, nch, tpc, sms) > bb::adjoint_chunk_cost(F, chunks, per, sms)) {
                    std::printf("sms %llu F %llu tiles %llu: %llu chunks of %llu\\n", (unsigned long long)sms,
                                (unsigned long long)F, (unsigned long long)n, (unsigned long long)nch,
                                (unsigned long long)tpc);
                    return 1;
                }
            }
    return 0;
}
"""


def test_chunks_use_the_sms(tmp_path):
    src, exe = tmp_path / "chunks.cc", tmp_path / "chunks"
    src.write_text(PROGRAM)
    cxx = shutil.which("g++") or "g++"
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "blade_b200", "csrc"), str(src), "-o",
                        str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
