// The host's wait for a step's report, apart from CUDA, so that it can be followed without a device.
#pragma once
#include <atomic>
#include <cstdint>
#include <thread>

namespace qtb {

enum class StepStream { kBusy, kDry, kFailed };
enum class StepOutcome { kReported, kNoReport, kStreamFailed };

// Polls of a wait (a pause of the processor each, about 40 ns) between two offers of the core to other threads, and between two looks at the stream.
constexpr unsigned int kStepYieldPolls = 128, kStepStreamPolls = 4096;

// Waits until every step launched has reported. `s` has
//   reported()  steps that the device has told of (memory that it writes);   launched()  steps that were launched;
//   stream()    whether the steps' stream is still busy;                     recount()   makes launched() the number of steps that the device has counted.
// A step that gives up reports nothing and is not counted: its stream runs dry, and without the recount every later wait would look for its report as well.
template <typename Steps>
StepOutcome wait_for_steps(Steps& s) {
    for (unsigned int polls = 1; s.reported() != s.launched(); ++polls) {
#if defined(__x86_64__)
        __builtin_ia32_pause();
#endif
        if (polls % kStepYieldPolls != 0) continue;
        if (polls % kStepStreamPolls == 0) {
            const StepStream state = s.stream();
            if (state == StepStream::kFailed) return StepOutcome::kStreamFailed;
            if (state == StepStream::kDry) {
                if (s.reported() == s.launched()) break;  // (it came between the two looks)
                s.recount();
                return StepOutcome::kNoReport;
            }
        }
        std::this_thread::yield();
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    return StepOutcome::kReported;
}

}  // namespace qtb
