// Host-side waiting shared by the C-ABI entry points.
//
// A wait polls, so that a stuck device surfaces as a timeout status instead of
// a hang. It polls without sleeping at first (a sleep of a few microseconds
// takes 55-60 with the kernel's timer slack, longer than most of the work that
// is waited for), and later sleeps for a small share of the time already
// waited, which bounds both the overshoot and the polling. Measured on a B200
// box: forces, statistics, a probe and a slice after 10 steps of 512x256x256,
// 6.98 ms with sleeps that doubled from 5 to 500
// us, 6.70 ms so.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <thread>

namespace fc {

// Polled without sleeping up to here: the first sleep adds some 50 us, which a
// wait of half a millisecond (the voxelizer's second) would feel.
constexpr long long kSpinNs = 1'000'000;

// Polls done() (a cudaError_t: cudaErrorNotReady to go on) until it returns
// something else or `timeout_ms` (negative: none) have passed; then
// cudaErrorNotReady is returned.
template <class F>
cudaError_t poll_until(F&& done, long long timeout_ms) {
    const auto t0 = std::chrono::steady_clock::now();
    for (;;) {
        const cudaError_t e = done();
        if (e != cudaErrorNotReady) return e;
        const long long ns =
            std::chrono::duration_cast<std::chrono::nanoseconds>(std::chrono::steady_clock::now() - t0).count();
        if (timeout_ms >= 0 && ns >= timeout_ms * 1'000'000) return cudaErrorNotReady;
        if (ns < kSpinNs)
            std::this_thread::yield();
        else
            std::this_thread::sleep_for(std::chrono::nanoseconds(std::clamp<long long>(ns / 64, 20'000, 500'000)));
    }
}

// The same for a condition that another host thread makes true, and which is
// sure to become true.
template <class P>
void wait_until(P&& ready) {
    poll_until([&] { return ready() ? cudaSuccess : cudaErrorNotReady; }, -1);
}

}  // namespace fc
