"""The pool that hands every operator-API weight its own error word (`csrc/word_pool.hpp`), compiled for the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include "word_pool.hpp"
#define CHECK(c) if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; }
int live = 0;
bool full = false;
int main() {
    auto get = [](uint32_t n) -> uint32_t* { if (full) return nullptr; live++; return (uint32_t*)std::calloc(n, 4); };
    auto put = [](uint32_t* p) { live--; std::free(p); };
    wick::WordPool<decltype(get), decltype(put), 1024> pool(get, put);
    std::vector<uint32_t*> w;
    for (int i = 0; i < 3000; i++) w.push_back(pool.take());
    CHECK(std::set<uint32_t*>(w.begin(), w.end()).size() == 3000 && live == 3);   // no two takers share a word
    *w[1500] = 7;
    for (int i = 0; i < 3000; i++) CHECK(i == 1500 || *w[i] == 0);
    pool.give_back(nullptr);
    for (int i = 0; i < 2999; i++) pool.give_back(w[i]);
    CHECK(live == 1);                                                             // pages go back, the last one stays
    pool.give_back(w[2999]);
    CHECK(live == 1);
    for (int i = 0; i < 1024; i++) { w[i] = pool.take(); CHECK(w[i] && *w[i] == 0); }
    full = true;
    CHECK(pool.take() == nullptr);
    pool.give_back(w[3]);
    CHECK(pool.take() == w[3]);
    return 0;
}
"""


def test_every_taker_has_a_word_of_its_own(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "wick_b200", "csrc"), "-o", str(tmp_path / "t"), str(src)])
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
