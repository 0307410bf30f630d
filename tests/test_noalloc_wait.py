"""The wait at the allocation-free frame's grid barrier, as the kernel compiles it
(csrc/noalloc_wait.h), with threads for blocks (CPU): whatever block gives up at
whatever moment, all blocks pass the last barrier or none does, and a frame in
which no wait runs out always ends."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <atomic>
#include <cstdio>
#include <random>
#include <thread>
#include <vector>
#include "noalloc_wait.h"

struct Word {
    std::atomic<unsigned>* p;
    std::mt19937* rng;
    unsigned patience;      // looks before the wait is over, 0: never
    unsigned waited = 0;
    void pause() { if ((*rng)() & 1) std::this_thread::yield(); }
    void arrive() { pause(); p->fetch_add(1, std::memory_order_release); }
    unsigned look() { pause(); return p->load(std::memory_order_acquire); }
    void start() { waited = 0; }
    bool late() { return patience && ++waited > patience; }
    void replace(unsigned v, unsigned to) { pause(); p->compare_exchange_strong(v, to); }
};

int main()
{
    const int phases = 3;
    std::mt19937 seeds(1);
    int whole = 0, given_up = 0;
    for (int run = 0; run < 6000; ++run) {
        const int blocks = 2 + run % 3;
        std::atomic<unsigned> word{0};
        std::vector<int> passed(blocks, 0);
        std::vector<std::thread> t;
        const bool patient = run % 4 == 0;
        for (int b = 0; b < blocks; ++b) {
            const unsigned seed = seeds();
            t.emplace_back([&, b, seed] {
                std::mt19937 rng(seed);
                for (int ph = 1; ph <= phases; ++ph) {
                    for (unsigned n = rng() % 4; n; --n) std::this_thread::yield();   // the block's work
                    Word w{&word, &rng, patient ? 0u : 1u + (unsigned)(rng() % 6u)};
                    if (!pdg::na_wait_on(w, (unsigned)(ph * blocks))) return;
                }
                passed[b] = 1;
            });
        }
        for (auto& q : t) q.join();
        int n = 0;
        for (int b = 0; b < blocks; ++b) n += passed[b];
        if (n != 0 && n != blocks) { std::printf("run %d: %d of %d blocks passed\n", run, n, blocks); return 1; }
        if (patient && n == 0) { std::printf("run %d: given up although no wait ran out\n", run); return 1; }
        if ((word.load() & pdg::kNaGaveUp) ? n != 0 : n == 0) { std::printf("run %d: the mark says otherwise\n", run); return 1; }
        (n ? whole : given_up) += 1;
    }
    std::printf("%d %d\n", whole, given_up);
    return whole > 100 && given_up > 100 ? 0 : 2;   // both ends were met
}
"""


def test_all_blocks_pass_or_none(tmp_path):
    src = tmp_path / "wait.cpp"
    src.write_text(SOURCE)
    exe = str(tmp_path / "wait")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "cloth-cuda_gb300", "csrc"), str(src),
                    "-o", exe], check=True)
    p = subprocess.run([exe], stdout=subprocess.PIPE, text=True, timeout=300)
    assert p.returncode == 0, p.stdout
