"""The tensor-core ring's control flow (csrc/mma_ring.h) under host threads: work that ends in time, and work that does not."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "adock_b200" / "csrc"
HARNESS = r"""
#include "mma_ring.h"
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>
using Clock = std::chrono::steady_clock;
static const int STAGES = 3, THREADS = 6;

struct Cta {
    std::mutex m;
    std::condition_variable cv;
    int arrived = 0, generation = 0;
    bool vote = false, result = false, stray = false;
    std::vector<Clock::time_point> done;   // when each commit completes, in issue order
    std::atomic<int> refilled{0};          // fills of a stage whose work was still running
    int steps, slow, slow_ms;

    bool complete(int commit) {            // lock held
        return commit < (int)done.size() && Clock::now() >= done[commit];
    }
    // a barrier per stage: phase p completes with commit p * STAGES + stage
    bool try_wait(int stage, unsigned parity) {
        std::lock_guard<std::mutex> g(m);
        int phase = 0;
        while (complete(phase * STAGES + stage)) ++phase;
        return (unsigned)(phase & 1) != parity;
    }
    bool any(bool flag) {
        std::unique_lock<std::mutex> g(m);
        vote |= flag;
        const int gen = generation;
        if (++arrived == THREADS) {
            result = vote;
            vote = false;
            arrived = 0;
            ++generation;
            cv.notify_all();
        } else if (!cv.wait_for(g, std::chrono::seconds(5), [&] { return generation != gen; })) {
            stray = true;                  // the others never came: the threads parted ways
        }
        return result;
    }
};

int main(int argc, char** argv) {
    Cta c;
    c.steps = atoi(argv[1]);
    c.slow = atoi(argv[2]);      // this commit takes slow_ms, the others nothing; -1: none
    c.slow_ms = atoi(argv[3]);
    std::vector<int> ok(THREADS), votes(THREADS);
    std::vector<std::thread> threads;
    std::atomic<int> running{0};
    for (int t = 0; t < THREADS; ++t)
        threads.emplace_back([&, t] {
            const auto limit = std::chrono::milliseconds(20 + 3 * t);   // threads give up at different times
            auto wait = [&](int s, unsigned parity) {
                const auto t0 = Clock::now();
                while (!c.try_wait(s, parity)) {
                    if (Clock::now() - t0 > limit) return false;
                    std::this_thread::yield();
                }
                return true;
            };
            auto fill = [&](int it, int s) {
                std::lock_guard<std::mutex> g(c.m);
                if (it >= STAGES && !c.complete(it - STAGES)) ++c.refilled;
            };
            auto any = [&](bool f) {
                ++votes[t];
                return c.any(f);
            };
            auto issue = [&](int it, int) {
                if (t) return;
                std::lock_guard<std::mutex> g(c.m);
                auto end = Clock::now() + std::chrono::milliseconds(it == c.slow ? c.slow_ms : 0);
                if (!c.done.empty()) end = std::max(end, c.done.back());   // work completes in order
                c.done.push_back(end);
            };
            ok[t] = adock::run_ring<STAGES>(c.steps, wait, fill, any, issue);
            std::lock_guard<std::mutex> g(c.m);
            if (!c.done.empty() && !c.complete((int)c.done.size() - 1)) ++running;
        });
    for (auto& t : threads) t.join();
    bool same = !c.stray;
    for (int t = 1; t < THREADS; ++t) same = same && ok[t] == ok[0] && votes[t] == votes[0];
    printf("%d %d %d %d %d\n", (int)same, ok[0], (int)c.done.size(), (int)running, (int)c.refilled);
}
"""


@pytest.fixture(scope="module")
def ring(tmp_path_factory):
    d = tmp_path_factory.mktemp("ring")
    (d / "ring.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(CSRC), str(d / "ring.cpp"), "-o", str(d / "ring")],
                   check=True)

    def run(steps, slow=-1, ms=0):
        """(threads agreed, completed, commits issued, threads that returned with work running, early refills)"""
        out = subprocess.run([str(d / "ring"), str(steps), str(slow), str(ms)], capture_output=True, text=True, check=True,
                             timeout=60)
        return [int(v) for v in out.stdout.split()]
    return run


@pytest.mark.parametrize("steps", [0, 1, 2, 3, 4, 7, 20])
def test_work_in_time(ring, steps):
    assert ring(steps) == [1, 1, steps, 0, 0]


@pytest.mark.parametrize("steps,slow", [(1, 0), (4, 0), (5, 1), (8, 2), (8, 7), (13, 5), (13, 12)])
def test_threads_stay_together_after_a_late_wait(ring, steps, slow):
    same, ok, issued = ring(steps, slow, 5000)[:3]   # longer than every wait (nothing sleeps that long)
    assert (same, ok) == (1, 0) and issued <= steps


@pytest.mark.parametrize("steps,slow", [(1, 0), (4, 0), (5, 1), (5, 2), (8, 2), (8, 4), (8, 7), (13, 5), (13, 12)])
def test_late_work_has_ended_when_the_threads_return(ring, steps, slow):
    """Work later than one wait (20-35 ms) but not than the second one."""
    same, ok, issued, running, refilled = ring(steps, slow, 45)
    assert same and issued >= slow + 1 and running == 0 and refilled == 0
