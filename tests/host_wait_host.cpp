// Host driver of gpuspgemm_b200/csrc/host_wait.hpp for tests/test_host_wait.py: the
// flag is raised by another thread, the stream is a word that says how it stands.
//
// Usage: host_wait_host SCHEDULE RAISE_MS END   (SCHEDULE spin|yield|block; END 0
// running, 1 done, -1 failed: what the stream answers after RAISE_MS; RAISE 0|1)
// Prints one JSON object.
#include <cstdio>
#include <cstdlib>
#include <string>
#include <thread>

#include "../gpuspgemm_b200/csrc/host_wait.hpp"

int main(int argc, char** argv) {
    using namespace b200;
    if (argc != 5) return 2;
    const std::string how = argv[1];
    const int ms = std::atoi(argv[2]);
    const int end = std::atoi(argv[3]);
    const bool raise = std::atoi(argv[4]) != 0;
    volatile unsigned long long flag = 6;
    std::atomic<int> stream{0};
    long queries = 0, blocks = 0, yields = 0;
    std::thread device([&] {
        std::this_thread::sleep_for(std::chrono::milliseconds(ms));
        if (raise) flag = 7;
        stream = end;
    });
    const auto t0 = std::chrono::steady_clock::now();
    const WaitEnd w = wait_for_flag(
        &flag, 7,
        how == "block" ? WaitSchedule::kBlock
        : how == "yield" ? WaitSchedule::kYield : WaitSchedule::kSpin,
        [&] { queries++; return stream.load(); },
        [&] {
            blocks++;
            while (stream == 0) std::this_thread::sleep_for(std::chrono::microseconds(100));
            return stream.load();
        },
        [&] { yields++; std::this_thread::yield(); });
    const double us = std::chrono::duration<double, std::micro>(
        std::chrono::steady_clock::now() - t0).count();
    device.join();
    std::printf("{\"end\": \"%s\", \"queries\": %ld, \"blocks\": %ld, \"yields\": %ld, \"us\": %.1f, "
                "\"query_us\": %lld}\n",
                w == WaitEnd::kRaised ? "raised" : w == WaitEnd::kFailed ? "failed" : "not raised",
                queries, blocks, yields, us, static_cast<long long>(kWaitQuery.count()));
    return 0;
}
