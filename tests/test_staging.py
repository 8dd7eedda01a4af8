"""Buffers kept between calls: as many as calls were in flight at once, none
made or freed again by the same number of threads (host code only), and calls
of more threads than that agree with one thread's (GPU)."""
import os
import subprocess
import threading

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <atomic>
#include <barrier>
#include <cstdio>
#include <thread>
#include <vector>
#include "qoa_staging.h"
std::atomic<int> made{0}, freed{0};
struct Fake {
    static void* get() { ++made; return new int(0); }
    static void put(void* p) { ++freed; delete static_cast<int*>(p); }
};
qoa::KeptBuffers<Fake, 64> pool;
void round(int threads, int calls) {
    std::barrier all(threads);
    std::vector<std::thread> t;
    for (int k = 0; k < threads; ++k)
        t.emplace_back([&] {
            for (int c = 0; c < calls; ++c) {
                int* p = static_cast<int*>(pool.take());
                if (++*p != 1) std::printf("shared buffer\n");
                all.arrive_and_wait();  // every thread holds one
                --*p;
                pool.give(p);
                all.arrive_and_wait();
            }
        });
    for (auto& x : t) x.join();
}
int main() {
    round(32, 20); std::printf("%d %d\n", made.load(), freed.load());
    round(16, 20); std::printf("%d %d\n", made.load(), freed.load());
    round(70, 1);  std::printf("%d %d\n", made.load(), freed.load());
    pool.trim(8);  std::printf("%d %d\n", made.load(), freed.load());
}
"""


def test_as_many_as_calls_in_flight(tmp_path):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++20", "-O1", "-pthread", "-I", os.path.join(ROOT, "qoa_b200", "csrc"), str(src), "-o",
                    str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=60).stdout.split("\n")
    assert out[:4] == ["32 0", "32 0", "70 6", "70 62"]


@pytest.mark.gpu
def test_sixteen_threads_read_their_own_results():
    import qoa_b200 as qb

    n, shots, threads = 10, 24, 16
    u = np.random.default_rng(3).random((threads, shots * n))
    states = [qb.QuantumState(n) for _ in range(threads)]
    for k, st in enumerate(states):
        st.set_random_state(100 + k)
    want = [(st.sample(shots, u[k]), st.get_probabilities(), st.get_state_vector()) for k, st in enumerate(states)]
    bad = []

    def work(k):
        for _ in range(30):
            got = (states[k].sample(shots, u[k]), states[k].get_probabilities(), states[k].get_state_vector())
            if not (np.array_equal(got[0], want[k][0]) and np.allclose(got[1], want[k][1], rtol=1e-13, atol=0)
                    and np.allclose(got[2], want[k][2], rtol=1e-13, atol=1e-16)):
                bad.append(k)

    ts = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for st in states:
        st.close()
    assert not bad
