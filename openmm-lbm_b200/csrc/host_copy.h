// Copies of large device arrays into the caller's (pageable) host memory.
//
// cudaMemcpy into pageable memory stages through the driver's buffers on one thread, which also takes the page faults of
// a freshly allocated destination: 226 MB of fields (192^3) took 145 ms with the conversion around it.  Here several
// threads each copy chunks through two pinned buffers of their own on a stream of their own, so that the transfer, the
// copy into place and the page faults overlap: 15 ms.
#pragma once

#include "lbm_internal.h"
#include <cuda_runtime.h>
#include <memory>
#include <mutex>
#include <vector>

namespace lbm {

class HostCopy {
public:
    struct Piece {
        void* host;
        const void* device;
        size_t bytes;
    };
    explicit HostCopy(int device) : device(device) {}
    ~HostCopy();
    // The copier of a device, shared by the kernels on it (pinned memory takes milliseconds to get): at most 8 MB of
    // pinned memory, given back with the last kernel that holds it.
    static std::shared_ptr<HostCopy> forDevice(int device);
    HostCopy(const HostCopy&) = delete;
    HostCopy& operator=(const HostCopy&) = delete;
    // Copies the pieces once the work on `stream` is done; returns when they are in place.  The copies themselves take
    // turns (they would share the same link); a caller waits for its own stream before its turn.  Without pinned memory,
    // streams or events for two threads the copy is a plain one.
    void download(const std::vector<Piece>& pieces, cudaStream_t stream);
private:
    struct Worker {
        cudaStream_t stream = nullptr;
        cudaEvent_t landed[2] = {nullptr, nullptr};
        char* pinned = nullptr;    // two chunks
    };
    static bool create(Worker& worker);
    static void release(Worker& worker);
    int prepare(int threads);
    const int device;
    std::mutex busy;
    std::vector<Worker> workers;
};

} // namespace lbm
