// Copies of large device arrays into pageable host memory (see host_copy.h).
#include "host_copy.h"
#include <algorithm>
#include <atomic>
#include <cstring>
#include <map>
#include <thread>

namespace lbm {

namespace {

const size_t kChunk = 1 << 19;
const size_t kBytesPerThread = 4 << 20;   // a thread for every 4 MB (starting one costs less than copying that much)
const int kMaxThreads = 8;

void check(cudaError_t e, const char* what) {
    if (e != cudaSuccess)
        throw Error(LBM_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

} // namespace

std::shared_ptr<HostCopy> HostCopy::forDevice(int device) {
    static std::mutex mutex;
    static std::map<int, std::weak_ptr<HostCopy>> copiers;
    std::lock_guard<std::mutex> lock(mutex);
    std::shared_ptr<HostCopy> copier = copiers[device].lock();
    if (!copier) {
        copier = std::make_shared<HostCopy>(device);
        copiers[device] = copier;
    }
    return copier;
}

HostCopy::~HostCopy() {
    for (Worker& w : workers) {
        if (w.stream != nullptr)
            cudaStreamDestroy(w.stream);
        for (cudaEvent_t e : w.landed)
            if (e != nullptr)
                cudaEventDestroy(e);
    }
    cudaFreeHost(pinned);
}

void HostCopy::prepare(int threads) {
    while ((int) workers.size() < threads) {
        workers.emplace_back();
        Worker& w = workers.back();
        check(cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking), "cudaStreamCreate");
        for (cudaEvent_t& e : w.landed)
            check(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "cudaEventCreate");
    }
    if (pinnedWorkers < threads) {
        cudaFreeHost(pinned);
        pinned = nullptr;
        pinnedWorkers = 0;
        check(cudaHostAlloc((void**) &pinned, 2*kChunk*threads, cudaHostAllocDefault), "cudaHostAlloc");
        pinnedWorkers = threads;
    }
}

void HostCopy::download(const std::vector<Piece>& pieces, cudaStream_t stream) {
    size_t total = 0;
    for (const Piece& p : pieces)
        total += p.bytes;
    const int cores = std::max(1, (int) std::thread::hardware_concurrency());
    const int threads = std::min({kMaxThreads, cores, (int) std::min<size_t>(kMaxThreads, total/kBytesPerThread)});
    if (threads < 2) {
        for (const Piece& p : pieces)
            check(cudaMemcpyAsync(p.host, p.device, p.bytes, cudaMemcpyDeviceToHost, stream), "cudaMemcpyAsync");
        check(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
        return;
    }
    // The caller's own steps first: others shall not wait for them.
    check(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
    std::lock_guard<std::mutex> lock(busy);
    prepare(threads);
    std::vector<Piece> chunks;
    for (const Piece& p : pieces)
        for (size_t at = 0; at < p.bytes; at += kChunk)
            chunks.push_back({(char*) p.host + at, (const char*) p.device + at, std::min(kChunk, p.bytes - at)});
    std::atomic<size_t> next(0);
    std::atomic<int> failed((int) cudaSuccess);
    auto run = [&](int t) {
        cudaError_t e = cudaSetDevice(device);
        const Worker& w = workers[t];
        // A chunk lands in one buffer while the one before it is copied out of the other.
        Piece held[2] = {{nullptr, nullptr, 0}, {nullptr, nullptr, 0}};
        for (int b = 0; e == cudaSuccess && failed.load() == (int) cudaSuccess; b ^= 1) {
            const size_t i = next.fetch_add(1);
            char* buffer = pinned + (2*(size_t) t + b)*kChunk;
            held[b].host = nullptr;
            if (i < chunks.size()) {
                held[b] = chunks[i];
                e = cudaMemcpyAsync(buffer, held[b].device, held[b].bytes, cudaMemcpyDeviceToHost, w.stream);
                if (e == cudaSuccess)
                    e = cudaEventRecord(w.landed[b], w.stream);
            }
            Piece& before = held[b ^ 1];
            if (e == cudaSuccess && before.host != nullptr) {
                e = cudaEventSynchronize(w.landed[b ^ 1]);
                if (e == cudaSuccess)
                    std::memcpy(before.host, pinned + (2*(size_t) t + (b ^ 1))*kChunk, before.bytes);
                before.host = nullptr;
            }
            if (held[b].host == nullptr)
                break;
        }
        cudaError_t end = cudaStreamSynchronize(w.stream);
        if (e == cudaSuccess)
            e = end;
        if (e != cudaSuccess)
            failed.store((int) e);
    };
    std::vector<std::thread> pool;
    try {
        for (int t = 1; t < threads; t++)
            pool.emplace_back(run, t);
    }
    catch (...) {
        // No more threads to be had: those that run (at least this one) take all chunks.
    }
    run(0);
    for (std::thread& t : pool)
        t.join();
    check((cudaError_t) failed.load(), "copy to the host");
}

} // namespace lbm
