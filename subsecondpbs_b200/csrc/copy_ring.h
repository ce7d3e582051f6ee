// Page-locked slots through which pageable host memory is copied.
#pragma once

#include <cuda_runtime.h>

#include "copy_threads.h"

namespace pbs {

// Two slots, an event per slot behind its last transfer, and the threads that fill and
// empty them.
struct CopyRing {
    static constexpr size_t kSlots = 2, kSlotBytes = size_t(4) << 20, kPieces = 2;
    float* mem = nullptr;
    cudaEvent_t done[kSlots] = {};
    CopyThreads threads;
    cudaStream_t last = nullptr;  // stream of the last transfers
    bool taken = false;
};

// Page-locking a ring takes 3 to 6 ms, so the contexts of a device share at most
// kMaxRings of them; one is lent for one copy, and all are freed with the last context
// that used them (CopyRingUser). A ring goes to a copy if its transfers are through, or
// lie in the copy's own stream: no context waits for another one's kernels.
constexpr size_t kMaxRings = 4;

// Counts a context among the users of its device's rings, from its first copy on.
class CopyRingUser {
public:
    CopyRingUser() = default;
    CopyRingUser(const CopyRingUser&) = delete;
    CopyRingUser& operator=(const CopyRingUser&) = delete;
    void begin(int device);
    void end();  // the context's streams are idle

private:
    int device_ = -1;
};

// A ring on loan to one copy on stream `s`; null if none is to be had. `volume`: a copy
// that gains too little (0.13 ms for 5 MB) to pay for a new ring by itself: one is made for the
// 32nd of them.
class CopyRingLoan {
public:
    CopyRingLoan(int device, cudaStream_t s, bool volume);
    ~CopyRingLoan();
    CopyRingLoan(const CopyRingLoan&) = delete;
    CopyRingLoan& operator=(const CopyRingLoan&) = delete;
    CopyRing* operator->() const { return ring_; }
    explicit operator bool() const { return ring_ != nullptr; }

private:
    CopyRing* ring_ = nullptr;
    cudaStream_t stream_;
};

}  // namespace pbs
