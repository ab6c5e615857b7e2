// device_share.h -- who of this process holds a device's SMs for long: scan
// streams, whose kernel keeps every SM but a few until it is drained, and batch
// scans while they run.
//
// The window network's row kernel (mlp.cu) has a form in clusters of four CTAs,
// which needs four whole SMs of one GPC at a time, and a form of single CTAs,
// which makes progress on any one SM.  The first is the faster one on a free
// device; beside a scan stream it would wait until the stream is drained, which
// the thread that waits may be the one to do.  So a network call takes the
// single form while a holder is counted here, and a stream that is about to
// launch its kernel waits for the network calls that run in the other form.
// That wait is bounded: a network call may itself be queued behind work of the
// caller's that only ends after the stream has been fed.
//
// Team launches (team.cuh) ask for streams too: few trajectories are spread over
// as many blocks as a free device has room for, but beside a stream those blocks
// would take turns on the reserved SMs.
#pragma once

#include <chrono>
#include <condition_variable>
#include <mutex>

namespace cor {

struct DeviceShare {
    std::mutex mu;
    std::condition_variable none;   // no network call in clusters
    int holders = 0;                // scan streams launched, batch scans running
    int streams = 0;                // of these, the streams
    int clusters = 0;               // network calls running in clusters
};

constexpr int kShareDevices = 64;   // (devices beyond share an entry: the single form a little more often)

// Never destroyed: a call may still end in another thread while the program exits.
__attribute__((visibility("hidden"))) inline DeviceShare& device_share(int device) {
    static DeviceShare* const all = new DeviceShare[kShareDevices];
    return all[(unsigned)device % kShareDevices];
}

// A stream that is about to launch its kernel, and one whose launch has ended.
inline void share_stream_begin(int device) {
    DeviceShare& d = device_share(device);
    std::unique_lock<std::mutex> l(d.mu);
    d.holders++;
    d.streams++;
    d.none.wait_for(l, std::chrono::seconds(2), [&] { return d.clusters == 0; });
}

inline void share_stream_end(int device) {
    DeviceShare& d = device_share(device);
    std::lock_guard<std::mutex> l(d.mu);
    d.holders--;
    d.streams--;
}

inline bool share_has_stream(int device) {
    DeviceShare& d = device_share(device);
    std::lock_guard<std::mutex> l(d.mu);
    return d.streams > 0;
}

// A batch scan, for as long as the object lives.  (It ends by itself: it waits for nobody.)
struct ShareHold {
    DeviceShare& d;
    explicit ShareHold(int device) : d(device_share(device)) {
        std::lock_guard<std::mutex> l(d.mu);
        d.holders++;
    }
    ~ShareHold() {
        std::lock_guard<std::mutex> l(d.mu);
        d.holders--;
    }
    ShareHold(const ShareHold&) = delete;
    ShareHold& operator=(const ShareHold&) = delete;
};

// A network call: in clusters if it can be and nobody holds the device.
struct NetworkTurn {
    DeviceShare& d;
    bool clusters = false;
    NetworkTurn(int device, bool can_cluster) : d(device_share(device)) {
        std::lock_guard<std::mutex> l(d.mu);
        clusters = can_cluster && d.holders == 0;
        if (clusters) d.clusters++;
    }
    ~NetworkTurn() {
        if (!clusters) return;
        std::lock_guard<std::mutex> l(d.mu);
        if (--d.clusters == 0) d.none.notify_all();
    }
    NetworkTurn(const NetworkTurn&) = delete;
    NetworkTurn& operator=(const NetworkTurn&) = delete;
};

}  // namespace cor
