// csrc/host_copy.cpp against stand-ins for the CUDA calls that it makes, so that its threads, its lock and its failures can
// be tested without a GPU (tests/test_host_copy.py builds and runs this).  A stream is a flag that holds its waiters back;
// copies are made at once; the calls of one kind fail from a chosen one on.  Exits with 0, or prints what went wrong.
#include "host_copy.h"
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <thread>

struct CUstream_st {
    std::atomic<bool> held{false};
    std::atomic<CUstream_st*> after{nullptr};
};
struct CUevent_st {
    CUstream_st* stream = nullptr;
};

static std::atomic<int> hostAllocs(0), failFrom(1 << 30), streams(0), failStream(-1), copies(0), failCopy(-1);
static std::atomic<int> live(0);

static cudaError_t wait(CUstream_st* s) {
    for (int i = 0; i < 20000 && s != nullptr; i++) {
        CUstream_st* other = s->after.load();
        if (!s->held && (other == nullptr || !other->held))
            return cudaSuccess;
        std::this_thread::sleep_for(std::chrono::milliseconds(1));
    }
    return s == nullptr ? cudaSuccess : cudaErrorUnknown;
}

extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "made up"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    if (streams++ == failStream)
        return cudaErrorMemoryAllocation;
    live++;
    *s = new CUstream_st;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { live--; delete s; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { live++; *e = new CUevent_st; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { live--; delete e; return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
    const int i = hostAllocs++;
    if (i >= failFrom)
        return cudaErrorMemoryAllocation;
    live++;
    *p = std::malloc(bytes);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    if (p != nullptr)
        live--;
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t bytes, cudaMemcpyKind, cudaStream_t s) {
    if (s == nullptr)
        return cudaErrorInvalidValue;
    if (copies++ == failCopy)
        return cudaErrorUnknown;
    std::memcpy(to, from, bytes);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { e->stream = s; return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { s->after = e->stream; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return wait(e->stream); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return wait(s); }
}

static void fail(const char* what) {
    std::printf("%s\n", what);
    std::fflush(stdout);
    std::_Exit(1);
}

static const size_t kMB = 1 << 20;

// The copies of two pieces (the second not a multiple of a chunk), whose bytes all differ from what was there.
static void copyTwo(lbm::HostCopy& copier, CUstream_st& stream, size_t bytes, const char* what) {
    std::vector<char> a(bytes), b(bytes + 12345), x(a.size(), 0), y(b.size(), 0);
    for (size_t i = 0; i < b.size(); i++) {
        b[i] = (char) (1 + i*7919%250);
        if (i < a.size())
            a[i] = (char) (1 + (i/4096 + i)%251);
    }
    copier.download({{x.data(), a.data(), a.size()}, {y.data(), b.data(), b.size()}}, &stream);
    if (x != a || y != b)
        fail(what);
}

int main() {
    CUstream_st stream, slow;
    for (size_t bytes : {(size_t) 1, 2*kMB, 4*kMB, 9*kMB, 40*kMB}) {
        lbm::HostCopy copier(0);
        copyTwo(copier, stream, bytes, "a copy went wrong");
        copyTwo(copier, stream, bytes, "a second copy went wrong");
    }
    {
        // Steps queued on one kernel's stream hold up that kernel's read-out only.
        lbm::HostCopy copier(0);
        slow.held = true;
        std::atomic<bool> slowDone(false);
        std::thread other([&] {
            copyTwo(copier, slow, 12*kMB, "the copy of the busy stream went wrong");
            slowDone = true;
        });
        std::this_thread::sleep_for(std::chrono::milliseconds(200));
        std::atomic<bool> done(false);
        std::thread mine([&] {
            copyTwo(copier, stream, 12*kMB, "the copy beside a busy stream went wrong");
            done = true;
        });
        for (int i = 0; i < 5000 && !done; i++)
            std::this_thread::sleep_for(std::chrono::milliseconds(1));
        if (!done)
            fail("a read-out waited for another kernel's steps");
        if (slowDone)
            fail("a read-out did not wait for its own steps");
        slow.held = false;
        other.join();
        mine.join();
    }
    // Without pinned memory, with some of it, and once there is some again.
    for (int some : {0, 1, 3}) {
        lbm::HostCopy copier(0);
        failFrom = hostAllocs + some;
        copyTwo(copier, stream, 40*kMB, "a copy without pinned memory went wrong");
        failFrom = 1 << 30;
        copyTwo(copier, stream, 40*kMB, "a copy after the pinned memory ran out went wrong");
    }
    {
        lbm::HostCopy copier(0);
        failStream = streams + 1;
        try {
            copyTwo(copier, stream, 40*kMB, "a copy with too few streams went wrong");
        }
        catch (const lbm::Error&) {
        }
        copyTwo(copier, stream, 40*kMB, "a copy after a stream failed went wrong");
    }
    {
        // A copy that fails is reported, and the next one works.
        lbm::HostCopy copier(0);
        failCopy = copies + 5;
        bool reported = false;
        try {
            copyTwo(copier, stream, 40*kMB, "a copy that failed was taken for a good one");
        }
        catch (const lbm::Error& e) {
            reported = e.status == LBM_ERR_CUDA;
        }
        if (!reported)
            fail("a copy that failed was not reported");
        copyTwo(copier, stream, 40*kMB, "the copy after one that failed went wrong");
    }
    if (live != 0)
        fail("streams, events or pinned memory were not given back");
    return 0;
}
