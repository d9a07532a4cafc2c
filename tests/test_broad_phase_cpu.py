"""Pieces of the body-pair broad phase (colb_b200/csrc/bpair.cu) from their
source on the CPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
EMIT = r"""
#include <cstdio>
#include <vector>
#define DV inline
struct BpArgs { unsigned long long* out; int cap; int* count; };
inline int atomicAdd(int* p, int v) { int o = *p; *p += v; return o; }
#include "emit.inc"
int main() {
    int bad = 0;
    const int caps[] = {1, 2, 31, 4096}, more[] = {-1, 0, 1, 2, 40, 5000};
    for (int cap : caps)
        for (int d : more) {
            const int hits = cap + d;
            std::vector<unsigned long long> out(cap + 1, ~0ull);
            int count = 0;
            BpArgs A{out.data(), cap, &count};
            for (int i = 0; i < hits; i++) bp_emit(A, i & 1, i, i + 7);
            // the host takes the list when the count does not exceed its capacity
            bool ok = (count <= cap) == (hits <= cap) && out[cap] == ~0ull;
            if (hits <= cap) ok = ok && count == hits;
            for (int i = 0; i < hits && i < cap; i++)
                ok = ok && out[i] == (((unsigned long long)(i & 1) << 62) | ((unsigned long long)i << 31) | (unsigned long long)(i + 7));
            if (!ok) { std::printf("capacity %d, %d hits: count %d\n", cap, hits, count); bad++; }
        }
    return bad;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_a_list_that_lacks_a_hit_is_seen_to_overflow(tmp_path):
    d = str(tmp_path)
    src = open(os.path.join(ROOT, "colb_b200", "csrc", "bpair.cu")).read()
    at = src.index("DV void bp_emit(")
    open(os.path.join(d, "emit.inc"), "w").write(src[at:src.index("\n}\n", at) + 3])
    open(os.path.join(d, "emit.cpp"), "w").write(EMIT)
    exe = os.path.join(d, "emit")
    subprocess.check_call(["g++", "-std=c++17", "-O1", os.path.join(d, "emit.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
