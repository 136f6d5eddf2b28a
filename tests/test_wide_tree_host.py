"""The host side of the four-wide tree in a program of its own (g++, no GPU): a
tree of 2^17 triangles is packed to the same bytes whether or not the system
has threads to give; pthread_create is the test's, and refuses after a count."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "noor_b200" / "csrc"

THREADS = r"""
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>
#include "wide_bvh.h"
#include "noor_b200.h"
int set_error(int code, const std::string&) { return code; }
void clear_error() {}
static int g_left = 1 << 30;
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) noexcept {
    if (g_left-- <= 0) return EAGAIN;
    using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    static Fn real = (Fn)dlsym(RTLD_NEXT, "pthread_create");
    return real(t, a, f, x);
}
static std::vector<uint32_t> w;
static uint32_t put(uint32_t first, uint32_t count) {
    const uint32_t n = (uint32_t)(w.size() / 8);
    w.resize(w.size() + 8);
    float lo[3] = {(float)first, 0.0f, 0.0f}, hi[3] = {(float)(first + count), 1.0f, 1.0f};
    uint32_t w0 = first, w1 = NOOR_TRI_LEAF_MASK | count;
    if (count > 1) {
        put(first, count / 2);
        w0 = put(first + count / 2, count - count / 2);
        w1 = 0;
    }
    std::memcpy(&w[8 * n], lo, 12);
    w[8 * n + 3] = w0;
    std::memcpy(&w[8 * n + 4], hi, 12);
    w[8 * n + 7] = w1;
    return n;
}
static nb::WideTreeDev pack(int threads) {
    nb::WideTree t;
    nb::WideTreeDev d;
    g_left = threads;
    std::string why;
    if (!nb::build_wide_tree(w.data(), w.size() / 8, 0, nb::kWideMaxStack, t, &why) ||
        !nb::pack_wide_tree(w.data(), t, 1 << 17, std::vector<uint32_t>(1, 1u), d))
        printf("no tree: %s\n", why.c_str());
    g_left = 1 << 30;
    return d;
}
int main() {
    put(0, 1 << 17);
    const nb::WideTreeDev a = pack(1 << 30);
    if (a.nodes.size() < 1 << 15) return 2;
    for (int threads : {0, 1, 3}) {
        const nb::WideTreeDev b = pack(threads);
        if (a.nodes.size() != b.nodes.size() || a.root_word != b.root_word || a.leaf_of != b.leaf_of ||
            std::memcmp(a.nodes.data(), b.nodes.data(), a.nodes.size() * sizeof(a.nodes[0])))
            return 3;
    }
    puts("same");
}
"""


def _program(tmp_path, text, name):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    src, exe = tmp_path / (name + ".cpp"), tmp_path / name
    src.write_text(text)
    cmd = [gxx, "-std=c++17", "-O1", "-D_GNU_SOURCE", "-pthread", "-I", str(CSRC), "-I", str(ROOT / "include"),
           str(src), str(CSRC / "wide_bvh.cpp"), "-o", str(exe), "-ldl"]
    out = subprocess.run(cmd, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-3000:]
    return subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)


def test_packing_without_threads(tmp_path):
    out = _program(tmp_path, THREADS, "threads")
    assert out.returncode == 0 and out.stdout.split() == ["same"], (out.returncode, out.stdout, out.stderr)


WORDS = r"""
#include <cstdio>
#include <string>
#include "wide_bvh.h"
int set_error(int code, const std::string&) { return code; }
void clear_error() {}
int main() {
    using namespace nb;
    // how the walks read a kWRef word: a leaf, an instance, else a node
    auto node = [](uint32_t w) { return (w & (kWUntested | kWLeaf)) != kWLeaf && !(w & kWUntested) ? w & kWIndex : kWNone; };
    for (size_t n : {(size_t)1, (size_t)2, (size_t)kWIndex - 1, (size_t)kWIndex, (size_t)kWIndex + 1, (size_t)kWLeaf + 6,
                     (size_t)kWUntested + 1, (size_t)1 << 31, (size_t)0xFFFFFFFFu}) {
        const uint32_t last = (uint32_t)(n - 1);
        if (ref_words_fit(n) && node(kWRef | last) != last) return 2;
        WideTree tree;
        if (!ref_words_fit(n) && build_wide_tree(nullptr, n, 0, kWideMaxStack, tree, nullptr)) return 3;
    }
    if (!ref_words_fit((size_t)kWIndex - 1)) return 4;
    puts("same");
}
"""


def test_words_of_large_trees(tmp_path):
    """node indices beyond a word's 29 bits are kept out of the walks that go by words"""
    out = _program(tmp_path, WORDS, "words")
    assert out.returncode == 0 and out.stdout.split() == ["same"], (out.returncode, out.stdout, out.stderr)
