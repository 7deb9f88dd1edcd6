// The host's wait for a flag that a kernel raises in page-locked memory.
#pragma once

#include <atomic>
#include <chrono>

#if defined(__x86_64__) || defined(__i386__)
#include <immintrin.h>
#endif

namespace b200 {

// How the process wants its host threads to wait for the device
// (cudaSetDeviceFlags): reading the flag without leaving the core, offering the
// core to other threads between reads, or asleep in the driver.  (Yielding after
// 50 us of reads in every process, on a shared 16-core host with four waiting
// threads: the served bench's median latency 1.24 -> 1.55 ms at 80 % load.)
enum class WaitSchedule { kSpin, kYield, kBlock };
enum class WaitEnd { kRaised, kFailed, kNotRaised };

// Time between queries of the stream while the flag is not raised: a query takes
// driver locks that other threads' launches need, and only an error needs it.
// (A query every 4,096 reads came every few microseconds.)
constexpr std::chrono::microseconds kWaitQuery{200};
constexpr unsigned kWaitReads = 32;  // reads of the flag between looks at the clock

inline void wait_pause() {
#if defined(__x86_64__) || defined(__i386__)
    _mm_pause();
#endif
}

// Waits until *flag == seq.  query() says whether the stream is still running
// (0), done (1) or failed (-1); block() waits for the stream and answers 1 or -1;
// yield() offers the core.  kNotRaised: the stream ended without the flag.
template<typename Query, typename Block, typename Yield>
WaitEnd wait_for_flag(const volatile unsigned long long* flag, unsigned long long seq,
                      WaitSchedule how, Query&& query, Block&& block, Yield&& yield) {
    using Clock = std::chrono::steady_clock;
    int state = 1;
    if (how == WaitSchedule::kBlock) {
        state = block();
    } else {
        Clock::time_point asked = Clock::now();
        for (unsigned reads = 1; *flag != seq; reads++) {
            if (how == WaitSchedule::kYield) yield();
            else wait_pause();
            if (reads % kWaitReads != 0) continue;
            const Clock::time_point now = Clock::now();
            if (now - asked < kWaitQuery) continue;
            asked = now;
            state = query();
            if (state != 0) break;
            state = 1;
        }
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    if (state < 0) return WaitEnd::kFailed;
    return *flag == seq ? WaitEnd::kRaised : WaitEnd::kNotRaised;
}

}  // namespace b200
