// Admission of cooperative kernels to a device (coop.cu).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <mutex>

namespace rb200 {

// One launch (or graph launch) that holds a cooperative kernel:
//
//     CoopTurn turn;
//     if ((rc = turn.begin(stream, blocks, user))) return rc;
//     ... the launch on `stream` ...
//     if ((rc = turn.end())) return rc;
//
// begin makes the stream wait for the launches whose lanes this one takes; end
// records its own end on them. The device's lanes stay locked in between, so
// that no other thread's launch comes between the wait and the record. Nothing
// here waits on the host for the device. blocks = 0 (no cooperative kernel)
// takes no lane. `user` is the launching solver's number (coop_user); a solver
// launches on one stream all its life, so its own launches need no wait.
constexpr int kCoopLanes = 4;  // of a device's SMs

uint64_t coop_user();  // a number that no other solver has
// Cooperative solves in flight on a device: carriers' steps and host-driven solves.
std::atomic<int>& coop_active(int device);

class CoopTurn {
public:
    CoopTurn() = default;
    CoopTurn(const CoopTurn&) = delete;
    CoopTurn& operator=(const CoopTurn&) = delete;
    int begin(cudaStream_t s, int blocks, uint64_t user);
    int end();

private:
    std::unique_lock<std::mutex> lock_;
    struct CoopDevice* dev_ = nullptr;
    cudaStream_t stream_ = nullptr;
    uint64_t user_ = 0;
    unsigned taken_ = 0;  // bit per lane
};

}  // namespace rb200
