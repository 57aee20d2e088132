"""The host's wait for a step's report (csrc/step_wait.hpp) with a device that is a script: reports that come, steps that give up, a stream that fails."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quintrit_b200", "csrc")

SOURCE = r"""
#include <chrono>
#include <cstdio>
#include <initializer_list>

#include "step_wait.hpp"
using namespace qtb;

struct Device {
    uint32_t done = 0, told = 0, count = 0;  // steps the device has counted, steps it has told of, steps launched
    int until_told = 0, until_dry = 1 << 30, looks = 0, recounts = 0;
    bool fails = false;
    uint32_t reported() { if (until_told > 0 && --until_told == 0) told = done; return told; }
    uint32_t launched() const { return count; }
    StepStream stream() { ++looks; return fails ? StepStream::kFailed : looks > until_dry ? StepStream::kDry : StepStream::kBusy; }
    void recount() { ++recounts, count = done; }
    void launch(bool gives_up, int polls) { ++count, looks = 0, until_dry = 1 << 30; if (gives_up) until_dry = 3; else ++done, until_told = polls; }
};
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    Device d;
    CHECK(wait_for_steps(d) == StepOutcome::kReported);  // nothing launched
    for (int polls : {1, 5, 127, 128, 129, 4096, 20000}) {
        d.launch(false, polls);
        CHECK(wait_for_steps(d) == StepOutcome::kReported && d.told == d.count && d.recounts == 0);
    }
    // a step that gives up, whatever its status says: found when the stream is dry, counted out, and the steps behind it are waited for as ever
    for (int turn = 1; turn <= 3; ++turn) {
        d.launch(true, 0);
        CHECK(wait_for_steps(d) == StepOutcome::kNoReport && d.recounts == turn && d.count == d.told && d.looks == 4);
        d.launch(false, 300);
        CHECK(wait_for_steps(d) == StepOutcome::kReported && d.recounts == turn && d.told == d.count);
    }
    // the report comes with the stream's end, seen between the two looks
    d.launch(false, 4097), d.until_dry = 0;
    CHECK(wait_for_steps(d) == StepOutcome::kReported && d.recounts == 3);
    // the counter passes zero
    d.done = d.told = d.count = 0xFFFFFFFFu;
    d.launch(false, 10);
    CHECK(wait_for_steps(d) == StepOutcome::kReported && d.count == 0);
    d.launch(true, 0), d.fails = true;
    CHECK(wait_for_steps(d) == StepOutcome::kStreamFailed);
    // more waiting threads than cores, on one core: each gives the core away, or the last would come to its turn after all the others' time slices
    std::atomic<uint32_t> turn{0};
    std::atomic<bool> late{false};
    struct Turns {
        std::atomic<uint32_t>& now;
        uint32_t want;
        uint32_t reported() const { return now.load(std::memory_order_relaxed) >= want ? want : want - 1; }
        uint32_t launched() const { return want; }
        StepStream stream() const { return StepStream::kBusy; }
        void recount() {}
    };
    constexpr uint32_t kThreads = 8, kTurns = 25;
    const auto start = std::chrono::steady_clock::now();
    std::thread all[kThreads];
    for (uint32_t t = 0; t < kThreads; ++t)
        all[t] = std::thread([&, t] {
            for (uint32_t k = 0; k < kTurns; ++k) {
                Turns mine{turn, k * kThreads + t};
                if (mine.want > 0 && wait_for_steps(mine) != StepOutcome::kReported) late = true;
                while (turn.load() != mine.want) std::this_thread::yield();
                turn.store(mine.want + 1);
            }
        });
    for (std::thread& t : all) t.join();
    const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - start).count();
    std::printf("%.1f\n", ms);
    return late ? 1 : 0;
}
"""


def test_waiting_for_steps(tmp_path):
    (tmp_path / "wait.cpp").write_text(SOURCE)
    exe = str(tmp_path / "wait")
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Werror", "-pthread", "-I", CSRC, "-o", exe, str(tmp_path / "wait.cpp")], check=True)
    core = str(min(os.sched_getaffinity(0)))
    r = subprocess.run(["taskset", "-c", core, exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    # 200 turns on one core: without yielding most of them cost a time slice of a scheduler (milliseconds) each
    assert float(r.stdout.split()[-1]) < 400, r.stdout
