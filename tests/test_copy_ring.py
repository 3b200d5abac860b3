"""The bookkeeping of the tensor-core kernels' copy rings (csrc/copy_ring.h) against a model of the barriers on the CPU: no copy is
asked for into a slot whose copy before has not landed and been read, and none is under way when the block may end, also
where readers stop, go on without waiting, or copies are late."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

MODEL = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "copy_ring.h"

constexpr int SLOTS = %d;
constexpr long LIMIT = 200;   // a wait gives up after this many steps

struct Model {
    std::mt19937 rng;
    long now = 0;
    unsigned full[SLOTS] = {}, empty[SLOTS] = {};   // phases completed
    long lands[SLOTS];                              // when the slot's copy lands, -1: none under way
    std::vector<long> delay, read;                  // of copy k: steps until it lands; steps its readers take
    unsigned stop, wild;                            // readers stop before copy `stop`; from `wild` on they wait for nothing
    unsigned next_read = 0;
    long read_at = -1;
    long stuck = 0, bad = 0;
    unsigned asked = 0;
    Model() { for (auto& l : lands) l = -1; }

    void step() {
        ++now;
        for (int s = 0; s < SLOTS; ++s)
            if (lands[s] >= 0 && now >= lands[s]) lands[s] = -1, ++full[s];
        if (next_read >= delay.size() || next_read >= stop) return;
        const unsigned s = next_read %% SLOTS;
        if (read_at < 0) {
            if (next_read < wild && full[s] <= next_read / SLOTS) return;   // not landed yet
            read_at = now + read[next_read];
        }
        if (now >= read_at) ++empty[s], ++next_read, read_at = -1;
    }
    bool wait(const unsigned* phases, unsigned s, unsigned parity) {
        for (long i = 0; i < LIMIT; ++i, step())
            if ((phases[s] & 1u) != parity) return true;
        return (phases[s] & 1u) != parity;
    }
    void ask() {
        const unsigned s = asked %% SLOTS;
        if (lands[s] >= 0) ++bad;                                                  // two copies of one slot under way
        if (asked >= SLOTS && empty[s] < asked / SLOTS && next_read < wild) ++bad;   // over contents that are still to be read
        lands[s] = now + delay[asked];
        ++asked;
    }
};

int main() {
    for (unsigned seed = 0; seed < 4000; ++seed) {
        Model m;
        m.rng.seed(seed);
        auto pick = [&](long lo, long hi) { return lo + (long) (m.rng() %% (unsigned long) (hi - lo + 1)); };
        const unsigned n = (unsigned) pick(0, 40);
        for (unsigned k = 0; k < n; ++k) {
            m.delay.push_back(pick(0, 1) ? pick(1, 5) : pick(1, seed %% 3 ? 150 : LIMIT + 150));   // a third of the runs: copies later than a wait
            m.read.push_back(pick(1, 20));
        }
        m.stop = seed %% 2 ? n : (unsigned) pick(0, n);
        m.wild = seed %% 5 ? n : (unsigned) pick(0, n);
        auto empty = [&](unsigned s, unsigned p) { return m.wait(m.empty, s, p); };
        auto full = [&](unsigned s, unsigned p) { return m.wait(m.full, s, p); };
        fnxk::CopyRing<SLOTS> ring;
        for (unsigned k = 0; k < n && ring.acquire(empty, full); ++k) m.ask(), ring.asked();
        ring.drain(full);
        ring.drain(full);   // (a copy later than one wait: what is checked is that the ring waits for the right phases)
        for (int s = 0; s < SLOTS; ++s) m.bad += m.lands[s] >= 0;
        if (m.stop == n && m.wild == n && seed %% 3 && ring.round * SLOTS + ring.slot != n) ++m.bad;   // nothing went wrong: every copy was asked for
        if (m.bad) return std::printf("seed %%u: %%ld\n", seed, m.bad), 1;
    }
    return 0;
}
"""


@pytest.mark.parametrize("slots", [1, 2, 3, 4, 6])
def test_ring_leaves_no_copy_under_way(tmp_path, slots):
    src, exe = tmp_path / "model.cpp", tmp_path / "model"
    src.write_text(MODEL % slots)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "sfnx_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
