"""The handle's growing arrays (eng_grow_blocks, eng_grow_contacts and
eng_grow_swept in colb_b200/csrc/capi.cu, bp_reserve in bpair.cu) from their source
on the CPU, with an allocator that fails at any one call: the handle keeps
arrays of the capacity it states, nothing is freed twice and nothing is lost;
and lists near the largest count."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
DRIVER = r"""
#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <map>
#include <string>
#include <vector>
#define DV inline
struct int2 { int x, y; }; struct int4 { int x, y, z, w; }; struct float4 { float x, y, z, w; };
enum { ABD_OK = 0, ABD_ERR_CUDA = -2, ABD_ERR_CONTACT_OVERFLOW = -3 };
typedef int cudaError_t;
enum { cudaSuccess = 0, cudaErrorMemoryAllocation = 2 };
// fake allocations: addresses are never used again, sizes up to `most` bytes in all
static std::map<void*, size_t> live;
static size_t total, most = ~(size_t)0;
static uintptr_t next_addr = 4096;
static long calls, fail_at = -1, double_frees;
static cudaError_t fake_malloc(void** p, size_t n) {
    if (calls++ == fail_at || n > most || total + n > most) return cudaErrorMemoryAllocation;
    *p = (void*)next_addr; next_addr += 4096; live[*p] = n; total += n;
    return cudaSuccess;
}
template <class T> static cudaError_t cudaMalloc(T** p, size_t n) { return fake_malloc((void**)p, n); }
static cudaError_t cudaFree(void* p) {
    auto it = live.find(p);
    if (it == live.end()) { double_frees++; return 1; }
    total -= it->second; live.erase(it);
    return cudaSuccess;
}
static cudaError_t cudaGetLastError() { return cudaSuccess; }
static cudaError_t cudaStreamSynchronize(int) { return cudaSuccess; }
namespace cub { struct DeviceRadixSort { template <class... A> static int SortKeys(void*, size_t& b, A...) { b = 64; return 0; } }; }
struct Engine {
    int nb = 10, nv = 1000, ne = 3000, nt = 2000, stream = 0; bool mixed = false;
    int* bcol = nullptr; void* vals = nullptr; int blk_cap = 0;
    int4 *contacts = nullptr, *cst = nullptr; int* ctype = nullptr; double* cxb = nullptr; int2* cbody = nullptr;
    unsigned long long *keys = nullptr, *keys_s = nullptr, *ukeys = nullptr; int cap = 0;
    int4* sw = nullptr; int *sw_flag = nullptr, *sw_off = nullptr; int sw_cap = 0; bool sw_valid = true;
    void* cub_tmp = nullptr; size_t cub_bytes = 0;
    void* bp_state = nullptr;
    int fail(int rc, const std::string&) { return rc; }
};
static int eng_stream_sync(Engine*) { return 0; }
static size_t cub_need(Engine*, int sw_cap, int nkeys) { return (size_t)sw_cap / 64 + (size_t)nkeys / 16 + 64; }
#include "growth.inc"

static long wrong;
static void holds(const char* what, const void* p, size_t bytes) {
    auto it = live.find((void*)p);
    if (it == live.end() || it->second < bytes) { std::printf("%s: fewer than %zu bytes\n", what, bytes); wrong++; }
}
// every array is allocated and as large as the handle says; none is lost
static void check(Engine& E) {
    size_t n = 0;
    auto one = [&](const char* w, const void* p, size_t bytes, bool used) { if (used) { holds(w, p, bytes); n++; } };
    const size_t c = E.cap, k = E.nb + 2 * c, s = E.sw_cap;
    one("bcol", E.bcol, 4 * (size_t)E.blk_cap, E.blk_cap > 0); one("vals", E.vals, 1152 * (size_t)E.blk_cap, E.blk_cap > 0);
    one("contacts", E.contacts, 16 * c, c > 0); one("cst", E.cst, 16 * c, c > 0); one("ctype", E.ctype, 4 * c, c > 0);
    one("cxb", E.cxb, 8 * c, c > 0); one("cbody", E.cbody, 8 * c, c > 0);
    one("keys", E.keys, 8 * k, c > 0); one("keys_s", E.keys_s, 8 * k, c > 0); one("ukeys", E.ukeys, 8 * k, c > 0);
    one("sw", E.sw, 16 * s, s > 0); one("sw_flag", E.sw_flag, 4 * (s + 1), s > 0); one("sw_off", E.sw_off, 4 * (s + 1), s > 0);
    one("cub_tmp", E.cub_tmp, E.cub_bytes, E.cub_bytes > 0);
    if (E.bp_state) {
        BpScratch* S = bps(&E);
        one("slab", S->slab, 1, true); one("bpairs", S->bpairs, 8 * (size_t)S->bp_cap, S->bp_cap > 0);
        one("items", S->items, 16 * (size_t)S->item_cap, S->item_cap > 0);
        one("keys", S->keys, 16 * (size_t)S->key_cap, S->key_cap > 0); one("tmp", S->tmp, S->tmp_bytes, S->key_cap > 0);
        if (S->key_cap > 0 && S->keys_s != S->keys + S->key_cap) { std::printf("keys_s\n"); wrong++; }
    }
    if (n != live.size()) { std::printf("%zu arrays live, %zu held\n", live.size(), n); wrong++; }
}
static int grow(Engine& E, int what, int need) {
    switch (what) {
        case 0: return eng_grow_blocks(&E, need);
        case 1: return eng_grow_contacts(&E, need);
        case 2: return eng_grow_swept(&E, need);
        default: return bp_reserve(&E, need, 8LL * need, need);
    }
}
int main() {
    // each growth of a handle that holds small arrays, failing at every one of its allocations
    for (int what = 0; what < 4; what++)
        for (int k = 0; k < 12; k++) {
            live.clear(); total = 0; fail_at = -1;
            Engine E;
            for (int w = 0; w < 4; w++) if (grow(E, w, 2000) != ABD_OK) wrong++;
            check(E);
            calls = 0; fail_at = k;
            const int rc = grow(E, what, 100000), ran = (int)calls;
            fail_at = -1;
            if (rc == ABD_OK && ran > k) { std::printf("growth %d: failure %d not reported\n", what, k); wrong++; }
            check(E);
            if (grow(E, what, 100000) != ABD_OK) { std::printf("growth %d: cannot grow after a failure\n", what); wrong++; }
            check(E);
        }
    // lists up to the largest count, with and without the memory for them
    for (int need : {1 << 28, 1000000000, 1600000000, 1717986919, 1800000000, INT_MAX - (1 << 20), INT_MAX})
        for (size_t memory : {~(size_t)0, (size_t)180 << 30})
            for (int what = 1; what < 4; what++) {
                live.clear(); total = 0; most = memory;
                Engine E;
                for (int w = 0; w < 3; w++) if (grow(E, w, 2000) != ABD_OK) wrong++;
                const int rc = grow(E, what, need);
                check(E);
                const int cap = what == 1 ? E.cap : what == 2 ? E.sw_cap : E.bp_state ? bps(&E)->key_cap : 0;
                if (rc == ABD_OK && cap < need) { std::printf("growth %d to %d: capacity %d\n", what, need, cap); wrong++; }
                if (rc != ABD_OK && rc != ABD_ERR_CONTACT_OVERFLOW) { std::printf("growth %d to %d: code %d\n", what, need, rc); wrong++; }
            }
    std::printf("wrong %ld, double frees %ld\n", wrong, double_frees);
    return wrong || double_frees ? 1 : 0;
}
"""


def _cut(name, first, last):
    src = open(os.path.join(ROOT, "colb_b200", "csrc", name)).read()
    return src[src.index(first):src.index(last, src.index(first))]


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_arrays_grow_wholly_or_not_at_all(tmp_path):
    d = str(tmp_path)
    text = _cut("engine.cuh", "constexpr int LIST_MAX", "// index of block (r, c)")
    text += _cut("capi.cu", "int eng_grow_blocks(", "bool eng_use_bp(")
    text += _cut("bpair.cu", "struct BpBoxes {", "struct BpDisp {") + _cut("bpair.cu", "struct BpScratch {", "void eng_step_boxes(")
    text += _cut("bpair.cu", "static int bp_reserve(", "// the counts to pinned host memory")
    open(os.path.join(d, "growth.inc"), "w").write(text)
    open(os.path.join(d, "growth.cpp"), "w").write(DRIVER)
    exe = os.path.join(d, "growth")
    subprocess.check_call(["g++", "-std=c++17", "-O1", os.path.join(d, "growth.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
