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
    for (Worker& w : workers)
        release(w);
}

bool HostCopy::create(Worker& w) {
    bool ok = cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking) == cudaSuccess;
    for (cudaEvent_t& e : w.landed)
        ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    ok = ok && cudaHostAlloc((void**) &w.pinned, 2*kChunk, cudaHostAllocDefault) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();        // the copy goes another way: later calls shall not find this error
        release(w);
    }
    return ok;
}

void HostCopy::release(Worker& w) {
    if (w.stream != nullptr)
        cudaStreamDestroy(w.stream);
    for (cudaEvent_t e : w.landed)
        if (e != nullptr)
            cudaEventDestroy(e);
    if (w.pinned != nullptr)
        cudaFreeHost(w.pinned);
    w = Worker();
}

// The workers there are, `threads` of them if they can be had.
int HostCopy::prepare(int threads) {
    while ((int) workers.size() < threads) {
        Worker w;
        workers.reserve(workers.size() + 1);
        if (!create(w))
            break;
        workers.push_back(w);
    }
    return std::min(threads, (int) workers.size());
}

void HostCopy::download(const std::vector<Piece>& pieces, cudaStream_t stream) {
    size_t total = 0;
    for (const Piece& p : pieces)
        total += p.bytes;
    const int cores = std::max(1, (int) std::thread::hardware_concurrency());
    int threads = std::min({kMaxThreads, cores, (int) std::min<size_t>(kMaxThreads, total/kBytesPerThread)});
    std::unique_lock<std::mutex> lock(busy, std::defer_lock);
    if (threads >= 2) {
        // The caller's own steps first: others shall not wait for them.
        check(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
        lock.lock();
        threads = prepare(threads);
    }
    if (threads < 2) {
        if (lock.owns_lock())
            lock.unlock();
        for (const Piece& p : pieces)
            check(cudaMemcpyAsync(p.host, p.device, p.bytes, cudaMemcpyDeviceToHost, stream), "cudaMemcpyAsync");
        check(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
        return;
    }
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
            char* buffer = w.pinned + b*kChunk;
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
                    std::memcpy(before.host, w.pinned + (b ^ 1)*kChunk, before.bytes);
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
