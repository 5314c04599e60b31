// Turns of a solve service's lanes on the GPU (serve.cpp). An on-chip linear
// solve in its grid form holds up to all SMs until it ends, and nothing
// preempts it; with several lanes at work the GPU's order of the waiting
// launches let the two oldest requests alternate, whole linear solves of 10 ms
// and more at a time, while requests of a few ms waited for seconds. So a
// grid's solve takes turns of a bounded number of iterations, in the order in
// which the lanes ask for them.
#pragma once

#include <atomic>
#include <condition_variable>
#include <mutex>

namespace cp {

class LaneGate {
public:
    // Two launches at a time: one that runs and one that follows on the GPU
    // while the first one's lane wakes up.
    static constexpr unsigned long long kAtOnce = 2;

    // Requests at work, the batch as one; turns are taken while there are others.
    std::atomic<int> busy{0};
    bool shared() const { return busy.load(std::memory_order_relaxed) > 1; }

    class Turn {
    public:
        explicit Turn(LaneGate& gate) : g(gate) {
            std::unique_lock<std::mutex> lock(g.mu);
            const unsigned long long ticket = g.next++;
            g.cv.wait(lock, [&] { return ticket < g.left + kAtOnce; });
        }
        ~Turn() {
            {
                std::lock_guard<std::mutex> lock(g.mu);
                ++g.left;
            }
            g.cv.notify_all();
        }
        Turn(const Turn&) = delete;
        Turn& operator=(const Turn&) = delete;

    private:
        LaneGate& g;
    };

private:
    std::mutex mu;
    std::condition_variable cv;
    unsigned long long next = 0, left = 0;  // tickets given out, turns ended
};

}  // namespace cp
