// Admission of cooperative kernels to a device.
//
// The blocks of a cooperative kernel (resident.cu, persist.cu) wait for one
// another, so all of them have to be resident. Two such kernels that start
// together could each hold a part of the SMs and wait for the other's. A
// device's SMs are therefore dealt into four lanes. A kernel takes as many lanes
// as have an SM for each of its blocks, all of them where it has more blocks
// than that, and starts after the kernels that took these lanes before it. So
// the kernels that run at one time have no more blocks than there are SMs (or
// one of them has the device), a block that waits for a place finds an SM that
// holds none of the others, and the other kernels' blocks there end by themselves.
//
// Four lanes, because four step graphs is what the device runs at a time (N
// carriers of 16^3 by per-pass kernels, without any order between them, step in
// 3.1, 3.4 and 6.3 ms for N = 1, 4 and 8). N plain carriers stepped together on
// a B200, ms, one after another / by lanes: 16^3 (one lane) N = 4 3.6 / 1.0,
// N = 8 7.1 / 1.9; 32^3 (two lanes) N = 4 7.1 / 3.6, N = 8 14.1 / 7.1. The
// per-pass kernels that the resident one replaced took 3.4, 6.3, 7.0 and 13.6.
#include "coop.hpp"

#include "internal.hpp"

namespace rb200 {

uint64_t coop_user() {
    static std::atomic<uint64_t> last{0};
    return ++last;
}

std::atomic<int>& coop_active(int device) {
    static std::atomic<int> active[64] = {};
    return active[device & 63];
}

struct CoopDevice {
    std::mutex mu;
    int sms = 0;  // 0: not set up
    uint64_t turns = 0;
    // the ends of the lanes' last launches: one event more than lanes, so that
    // one is free for the next launch
    cudaEvent_t done[kCoopLanes + 1] = {};
    struct {
        int done = -1;  // -1: nothing to wait for
        uint64_t user = 0, turn = 0;
    } lane[kCoopLanes];
};

int CoopTurn::begin(cudaStream_t s, int blocks, uint64_t user) {
    if (blocks < 1) return RB200_OK;
    static CoopDevice devices[64];
    int id = 0;
    RB200_CUDA(cudaGetDevice(&id));
    if (id < 0 || id >= 64) {
        set_error("cooperative launch: device index out of range");
        return RB200_EXECUTION;
    }
    CoopDevice& d = devices[id];
    lock_ = std::unique_lock<std::mutex>(d.mu);
    if (!d.sms) {
        for (auto& e : d.done)
            if (!e) RB200_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        RB200_CUDA(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, id));
    }
    const int width = d.sms / kCoopLanes;
    int want = kCoopLanes;
    while (want > 1 && blocks <= (want - 1) * width) --want;
    // the user's own lanes first (no other launch is held up by them), then the
    // ones taken longest ago
    taken_ = 0;
    unsigned waited = 0;  // bit per event
    for (int q = 0; q < want; ++q) {
        int best = -1;
        for (int l = 0; l < kCoopLanes; ++l) {
            if (taken_ & (1u << l)) continue;
            const bool own = d.lane[l].user == user, best_own = best >= 0 && d.lane[best].user == user;
            if (best < 0 || own > best_own || (own == best_own && d.lane[l].turn < d.lane[best].turn)) best = l;
        }
        taken_ |= 1u << best;
        const auto& lane = d.lane[best];
        if (lane.user == user || lane.done < 0 || (waited & (1u << lane.done))) continue;
        waited |= 1u << lane.done;
        RB200_CUDA(cudaStreamWaitEvent(s, d.done[lane.done], 0));
    }
    dev_ = &d;
    stream_ = s;
    user_ = user;
    return RB200_OK;
}

int CoopTurn::end() {
    if (!dev_) return RB200_OK;
    CoopDevice& d = *dev_;
    dev_ = nullptr;
    unsigned used = 0;
    for (int l = 0; l < kCoopLanes; ++l)
        if (!(taken_ & (1u << l)) && d.lane[l].done >= 0) used |= 1u << d.lane[l].done;
    int event = 0;
    while (used & (1u << event)) ++event;
    RB200_CUDA(cudaEventRecord(d.done[event], stream_));
    ++d.turns;
    for (int l = 0; l < kCoopLanes; ++l) {
        if (!(taken_ & (1u << l))) continue;
        d.lane[l].done = event;
        d.lane[l].user = user_;
        d.lane[l].turn = d.turns;
    }
    lock_.unlock();
    return RB200_OK;
}

}  // namespace rb200
