// Copies between pageable host memory and the device through page-locked
// slots, by several host threads: the driver's own pageable copy runs on one
// thread, which for a fresh destination also takes every page fault (94 MB of
// decoded horizons: 18 ms of a 23 ms decode).
#pragma once

#include "internal.cuh"

namespace ls200 {

// Owned by a context (its calls are serialised); slots and streams are made
// on first use and released with it.  A host that will not page-lock the slots
// (10 MB; a small locked-memory limit) or a driver without a stream to spare
// gets the driver's own copy, one that has some streams as many threads.
class StagedCopies {
public:
    ~StagedCopies();
    // Return when the bytes have arrived (page-locked host memory by the driver's
    // copy).  `after`: the stream whose work the
    // copy follows.  Throws Error on a failed copy.
    void to_host(int device, void *host, const void *src, size_t bytes, cudaStream_t after);
    void to_device(int device, void *dst, const void *host, size_t bytes, cudaStream_t after);

private:
    static constexpr int kThreads = 10;  // at most; never more than the host has cores
    static constexpr size_t kSlot = size_t(1) << 20;
    int open();  // the streams there are; 0: no slots, no event or no stream
    void run(int device, bool to_host, char *host, char *gpu, size_t bytes, cudaStream_t after);
    char *slots_ = nullptr;  // kThreads x kSlot, page-locked
    cudaStream_t streams_[kThreads] = {};
    cudaEvent_t ready_ = nullptr;
};

}  // namespace ls200
