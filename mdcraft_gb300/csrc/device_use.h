// device_use.h — which host threads have work on a device.
#pragma once

#include <atomic>

namespace mdg {

// A call or a served request that has work on a device, for as long as the
// object lives. A team of blocks (solo.cu) holds the GPU for its steps, so it
// takes a run only where nothing else is there, a few milliseconds at a time
// (kTeamLaunchUs); a mixed or FP64 step gives the same bits either way. Eight
// threads with an LJ argon system of 4,000 atoms each, us per step and system:
// teams in turn 12.5, graphs side by side 4.4.
class DeviceHold {
public:
    explicit DeviceHold(int device) : n_(count(device)) { n_.fetch_add(1); }
    ~DeviceHold() { n_.fetch_sub(1); }
    DeviceHold(const DeviceHold&) = delete;
    DeviceHold& operator=(const DeviceHold&) = delete;
    static int in_flight(int device) { return count(device).load(); }

protected:
    static std::atomic<int>& count(int device) {
        static std::atomic<int> in_flight[64];
        return in_flight[device & 63];
    }
    std::atomic<int>& n_;
};

// The same for a thread inside one of the C entry points that work on a
// device, counted once however the entry points call one another.
class DeviceUse {
public:
    explicit DeviceUse(int device) : device_(device & 63) {
        if (depth(device_)++ > 0) return;
        hold().fetch_add(1);
        inside(device_).fetch_add(1);
    }
    ~DeviceUse() {
        if (--depth(device_) > 0) return;
        hold().fetch_sub(1);
        inside(device_).fetch_sub(1);
    }
    DeviceUse(const DeviceUse&) = delete;
    DeviceUse& operator=(const DeviceUse&) = delete;
    // No other thread and no request has work on the device.
    bool alone() const { return DeviceHold::in_flight(device_) == 1; }
    // Threads inside such calls.
    static int threads(int device) { return inside(device & 63).load(); }

private:
    struct Counts : DeviceHold {
        using DeviceHold::count;
    };
    std::atomic<int>& hold() const { return Counts::count(device_); }
    static std::atomic<int>& inside(int device) {
        static std::atomic<int> n[64];
        return n[device];
    }
    static int& depth(int device) {
        static thread_local int d[64] = {};
        return d[device];
    }
    int device_;
};

}  // namespace mdg
