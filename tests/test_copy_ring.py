"""The order in which the partition swap drives its ring of bulk copies (ge-2_b200/csrc/copy_ring.cuh), followed on the host: a program
around the same header plays the copy engine, and lets the wait for one piece run out."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <set>
#include "copy_ring.cuh"
constexpr int S = 6;
struct Engine {
    int fail;                                  // the piece whose wait runs out (-1: none)
    std::set<int> loading, settled;            // loads in flight; those that were given a chance to land
    std::set<int> reading;                     // stores that may still read their stage
    int stored = 0, finished = 0;
    void need(bool ok, const char* what) { if (!ok) { printf("%s\n", what); exit(1); } }
    void load(int i) {
        for (int k : loading) need(k % S != i % S, "a stage is loaded while a load into it is in flight");
        for (int k : reading) need(k % S != i % S, "a stage is loaded while a store may still read it");
        loading.insert(i);
    }
    bool wait(int i) {
        need(loading.count(i) == 1, "waits for a piece that is not on its way");
        if (i == fail) return false;
        loading.erase(i);
        return true;
    }
    void store(int i) {
        need(i == stored, "stores out of order");
        stored++;
        reading.insert(i);
    }
    void stores_read() { while (reading.size() > 1) reading.erase(reading.begin()); }
    void settle(int i) { need(loading.erase(i) == 1, "settles what is not in flight"); settled.insert(i); }
    void finish() { reading.clear(); finished++; }
};
int main() {
    for (int n = 0; n < 20; n++)
        for (int fail = -1; fail < n; fail++) {
            Engine e{fail};
            const bool ok = ge2::copy_ring<S>(n, e);
            e.need(ok == (fail < 0), "the result does not say whether a wait ran out");
            e.need(e.loading.empty(), "returns with a load in flight that nobody waited for");
            e.need(e.finished == 1 && e.reading.empty(), "returns with a store in flight");
            e.need(e.stored == (fail < 0 ? n : fail), "a piece is missing");
            const int ahead = fail < 0 ? 0 : (n - fail < S - 1 ? n - fail : S - 1);
            e.need((int)e.settled.size() == ahead, "not every load ahead was given its chance");
        }
    return 0;
}
"""


def test_every_load_in_flight_is_waited_for_when_one_wait_runs_out(tmp_path):
    src = tmp_path / "ring.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "ring"
    r = subprocess.run(["g++", "-std=c++17", "-I", str(ROOT / "ge-2_b200" / "csrc"), "-x", "c++", str(src), "-o", str(exe)], capture_output=True, text=True)
    if r.returncode != 0 and "not found" in r.stderr:
        pytest.skip("no C++ compiler: " + r.stderr[:80])
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
