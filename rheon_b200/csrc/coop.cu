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

#include <cstdint>

#include "internal.hpp"

namespace rb200 {

namespace {
constexpr int kLanes = 4;
}

struct CoopDevice {
    std::mutex mu;
    int sms = 0;  // 0: not set up
    uint64_t turns = 0;
    struct {
        cudaEvent_t done = nullptr;  // the end of the last launch that took the lane
        cudaStream_t last = nullptr;
        uint64_t turn = 0;
    } lane[kLanes];
};

int CoopTurn::begin(cudaStream_t s, int blocks) {
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
        for (auto& l : d.lane)
            if (!l.done) RB200_CUDA(cudaEventCreateWithFlags(&l.done, cudaEventDisableTiming));
        RB200_CUDA(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, id));
    }
    const int width = d.sms / kLanes;
    int want = kLanes;
    while (want > 1 && blocks <= (want - 1) * width) --want;
    // the stream's own lanes first (no other launch is held up by them), then
    // the ones taken longest ago
    taken_ = 0;
    for (int q = 0; q < want; ++q) {
        int best = -1;
        for (int l = 0; l < kLanes; ++l) {
            if (taken_ & (1u << l)) continue;
            const bool own = d.lane[l].last == s;
            if (best < 0 || own > (d.lane[best].last == s) ||
                (own == (d.lane[best].last == s) && d.lane[l].turn < d.lane[best].turn))
                best = l;
        }
        taken_ |= 1u << best;
        // its own lane too: a stream's handle may come back for a new stream
        RB200_CUDA(cudaStreamWaitEvent(s, d.lane[best].done, 0));
    }
    dev_ = &d;
    stream_ = s;
    return RB200_OK;
}

int CoopTurn::end() {
    if (!dev_) return RB200_OK;
    CoopDevice& d = *dev_;
    dev_ = nullptr;
    ++d.turns;
    for (int l = 0; l < kLanes; ++l) {
        if (!(taken_ & (1u << l))) continue;
        RB200_CUDA(cudaEventRecord(d.lane[l].done, stream_));
        d.lane[l].last = stream_;
        d.lane[l].turn = d.turns;
    }
    lock_.unlock();
    return RB200_OK;
}

}  // namespace rb200
