// Tensor-core 3x3x3 convolutions of the learned warm start (include/lbm_b200_warmstart.h), written for sm_100a:
//
//  convSliceKernel      y[voxel][cout] = sum_k A[voxel][k] W[cout][k], k = tap*cin + ci, A the implicit im2col of x
//                       (zero padding), read in place from slices of x in shared memory
//  convForwardKernel    the same for the channel counts that the slices do not serve: A gathered per 128 voxels, all
//                       cout in one N tile (<= 256)
//  convSliceGradKernel  dW[cout][k] = sum_voxels dy[voxel][cout] A[voxel][k], the K dimension of the GEMMs being the
//                       voxels, from slices of x and shifted copies of dy; results added with FP32 atomics
//
// The GEMM core of the gathering kernel: 128 x N tiles, K in stages of 64 BF16 (one 128-byte row).  All 128 threads gather
// a stage into shared memory in the canonical K-major layout with the 128-byte swizzle (8-row atoms of 128-byte rows, the
// 16-byte chunk index XOR the row within the atom), make it visible to the tensor core's proxy, and one thread issues four
// tcgen05.mma (K = 16 each, BF16 x BF16 -> FP32 in tensor memory) and commits them to an mbarrier that every
// thread waits on (bounded: a wait that gives up sets the status flag and the CTA leaves after freeing its tensor
// memory).  The epilogue reads the accumulators with tcgen05.ld (warp w owns lanes 32w..32w+31 = rows of the tile).
// Descriptor layouts: the shared-memory matrix descriptor (start >> 4, leading offset, stride offset 1024 B >> 4,
// version 1, swizzle mode 2 = 128 B) and the instruction descriptor (F32 accumulator, BF16 A and B, both K-major,
// N >> 3, M >> 4) of the PTX ISA's tcgen05 matrix and instruction descriptor formats.
#include "lbm_b200_warmstart.h"
#include "lbm_internal.h"
#include <cuda_bf16.h>
#include <algorithm>
#include <cstdint>
#include <string>
#include <type_traits>

namespace {

constexpr int kThreads = 128;
constexpr int kTileM = 128;
constexpr int kChunk = 64;                     // BF16 per stage row
constexpr long long kSpinLimit = 1LL << 24;    // polls of an mbarrier before giving up

__device__ int convStatus;
// Polls of the waits for the tensor cores (kSpinLimit unless lbm_conv3d_set_wait_limit lowered it).  The drain of a
// stage whose wait gave up always uses kSpinLimit.
__device__ long long convWaitPolls = kSpinLimit;

__device__ __forceinline__ uint32_t smemAddr(const void* p) {
    return (uint32_t) __cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor of a K-major operand tile with the 128-byte swizzle.
__device__ __forceinline__ uint64_t smemDescriptor(uint32_t addr) {
    return (uint64_t) ((addr >> 4) & 0x3FFFu)
         | ((uint64_t) 1 << 16)                    // leading byte offset (16 B; unused for swizzled K-major)
         | ((uint64_t) (1024 >> 4) << 32)          // stride byte offset: 8-row atoms 1024 B apart
         | ((uint64_t) 1 << 46)                    // descriptor version of sm_100
         | ((uint64_t) 2 << 61);                   // 128-byte swizzle
}

// Instruction descriptor: FP32 accumulator, BF16 A and B, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t instrDescriptor(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t) (n >> 3) << 17) | ((uint32_t) (kTileM >> 4) << 24);
}

// Byte offset of 16-byte chunk `chunk` (0..7) of row `row` in a swizzled tile.
__device__ __forceinline__ uint32_t swizzled(int row, int chunk) {
    return (uint32_t) (row*128 + ((chunk ^ (row & 7)) << 4));
}

__device__ __forceinline__ void mmaBf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 :: "r"(tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void commitTo(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(mbar) : "memory");
}

__device__ __forceinline__ bool waitParity(uint32_t mbar, uint32_t parity, long long limit) {
    for (long long i = 0; i < limit; i++) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
                     "selp.b32 %0, 1, 0, P1;\n\t}" : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
        if (done)
            return true;
    }
    return false;
}

__device__ __forceinline__ void fenceAfterSync() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fenceBeforeSync() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

// 8 consecutive FP32 accumulator columns of this thread's row (lane) from tensor memory.
__device__ __forceinline__ void tmemLoad8(uint32_t addr, float v[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    for (int i = 0; i < 8; i++)
        v[i] = __uint_as_float(r[i]);
}

// 16 consecutive FP32 accumulator columns of this thread's row (lane) from tensor memory.
__device__ __forceinline__ void tmemLoad16(uint32_t addr, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                 "%14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                   "=r"(v[15]) : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__host__ __device__ inline uint32_t tmemColumns(int n) {
    return n <= 32 ? 32u : (n <= 64 ? 64u : (n <= 128 ? 128u : (n <= 256 ? 256u : 512u)));
}

// Setup common to both kernels: 1024-byte aligned tiles, tensor memory of `ncols` columns (warp 0), the mbarrier.
struct Stage {
    uint8_t* tileA;
    uint8_t* tileB;
    uint32_t mbar;
    uint32_t tmem;
};

__device__ __forceinline__ Stage setupStage(uint8_t* raw, int rowsB, uint32_t ncols) {
    uint32_t s = smemAddr(raw);
    uint8_t* base = raw + ((1024 - (s & 1023)) & 1023);
    Stage st;
    st.tileA = base;
    st.tileB = base + kTileM*128;
    uint64_t* bar = reinterpret_cast<uint64_t*>(st.tileB + rowsB*128);
    uint32_t* slot = reinterpret_cast<uint32_t*>(bar + 1);
    st.mbar = smemAddr(bar);
    if (threadIdx.x/32 == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smemAddr(slot)), "r"(ncols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(st.mbar), "r"(1) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fenceBeforeSync();
    __syncthreads();
    fenceAfterSync();
    st.tmem = *slot;
    return st;
}

__device__ __forceinline__ void releaseStage(const Stage& st, uint32_t ncols) {
    fenceBeforeSync();
    __syncthreads();
    if (threadIdx.x/32 == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(st.tmem), "r"(ncols) : "memory");
}

// One stage: the tiles are in shared memory; thread 0 issues the four K = 16 MMAs and commits; all threads wait.
// Returns false (for every thread) if the wait gave up; the caller then drains the stage (drainStage) before it
// frees the tensor memory that the MMAs may still be writing.
__device__ __forceinline__ bool runStage(const Stage& st, uint32_t idesc, int stage, long long limit) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
        fenceAfterSync();
        uint32_t a = smemAddr(st.tileA), b = smemAddr(st.tileB);
        for (int j = 0; j < 4; j++)
            mmaBf16(st.tmem, smemDescriptor(a + 32*j), smemDescriptor(b + 32*j), idesc, (stage > 0 || j > 0) ? 1u : 0u);
        commitTo(st.mbar);
    }
    bool ok = waitParity(st.mbar, (uint32_t) (stage & 1), limit);
    return __syncthreads_and(ok) != 0;
}

// After a wait that gave up: wait once more, with the full limit, for the MMAs of that stage (the only ones in flight),
// so that the tensor memory and the shared-memory tiles are released only when the tensor cores are done with them.
__device__ __forceinline__ void drainStage(const Stage& st, int stage) {
    waitParity(st.mbar, (uint32_t) (stage & 1), kSpinLimit);
    __syncthreads();
}

// ---------------------------------------------------------------------------------------------------------------
// The forward convolution from slices of the input held in shared memory.
//
// A CTA owns a column of 8 x 16 voxels (x, y) of one volume and `nTile` output channels, and marches over `zLen`
// planes: plane z of the output is one M = 128 tile (row = 8 y + x) with an accumulator of its own in tensor memory.
// Each input slice (10 x 18 voxels with the halo, zero outside the volume) is copied once into a ring of slots, laid
// out as [8-channel group][voxel] x 16 bytes: 8 x-neighbours are a core matrix of the unswizzled K-major layout, the
// y rows are 160 bytes apart (stride offset), the channel groups kPlane bytes (leading offset), and a tap is nothing
// but another start address in the slot.  Slice s takes part in the planes s - 1 (taps dz = +1), s and s + 1
// (dz = -1), so every plane receives its products in the order (tap, channel), 16 channels per tcgen05.mma: the order
// of the gathering kernel below, and its results bit for bit.
//
// Warps 0-3 read the accumulators (bias, ReLU, BF16 stores), warp 4 issues the MMAs, warps 5-8 copy slices and
// weight tiles with cp.async and hand them over through mbarriers.  The weights of one tap are a tile of
// [8-channel group][output channel] x 16 bytes.  Where all 27 fit they stay resident, those of the three dz of a (dy, dx)
// one below the other, and one MMA serves the three planes of a slice (their accumulators are neighbours, N = 3 nTile):
// A is read once for three taps.  Otherwise they stream through a ring of wSlots tiles, a tap per MMA.
//
// Bound: an MMA of M = 128 and N <= 64 reads 4 KB of A (36 wavefronts of shared memory with 16 channels of B) and holds
// the tensor core for 52 cycles: 41 us for 16 -> 16 channels on two 64 x 64 x 128 volumes with an MMA per tap, 15 us with
// one for three.  Measured there: 40 us, 47 us with an MMA per tap (the copies of the slices, 1.4 times the volume in
// pieces of 16 bytes, are what remains), 229 us with the gathering kernel, whose threads fetch every voxel 27 times and
// wait for each stage's MMAs; 48 -> 16 channels 89 us (124, 880), 32 -> 32 at 32 x 32 x 64 20 us (30, 84), 160 -> 160 at
// 8 x 8 x 16, streamed, 34 us (38, 307).  With one thread issuing from divergent code 16 -> 16 took 82 us (its operands
// went through general registers, 140-200 cycles per MMA), and with the planes' MMAs interleaved tap by tap 111 us (a
// branch per MMA).
// ---------------------------------------------------------------------------------------------------------------

constexpr int kTileX = 8, kTileY = 16, kHaloX = kTileX + 2, kHaloY = kTileY + 2;
constexpr int kSliceVoxels = kHaloX*kHaloY;
constexpr int kPlane = kSliceVoxels*16 + 16;   // bytes per channel group; + 16 spreads the groups over the banks
constexpr int kMaxSlots = 24, kMaxAcc = 8, kTaps = 27;
constexpr int kEpilogueThreads = 128, kProducersResident = 128, kProducersStreamed = 256;
constexpr int kZeroZone = 15*kHaloX*16 + 128;  // 16 core matrices at the stride of the y rows, all zero (cin = 8)

struct SliceParams {
    const __nv_bfloat16* x;
    const __nv_bfloat16* w;
    const float* bias;
    __nv_bfloat16* y;
    int batch, D, H, W, cin, cout, relu;
    int nTile, zLen, slots, wSlots, accSlots;
    int colsX, colsY, zBlocks, nBlocks, items;
};

struct SliceBarriers {
    uint64_t full[kMaxSlots], empty[kMaxSlots], wFull[kTaps], wEmpty[kTaps], accFull[kMaxAcc], accEmpty[kMaxAcc], drain;
    uint32_t tmem;
    int stop;
};

__host__ __device__ inline int sliceBytes(int cin) { return (cin/8)*kPlane; }
// A weight tile of `rows` rows: each group's at 16 bytes, + 16 per group to spread the groups over the banks.
__host__ __device__ inline int weightGroupBytes(int rows) { return rows*16 + 16; }
__host__ __device__ inline int weightTileBytes(int cin, int rows) { return (cin/8)*weightGroupBytes(rows); }
__host__ __device__ inline size_t sliceSmemBytes(int cin, int nTile, int slots, int wSlots) {
    // The single-group layout pairs taps: a 28th tile of zeros and a zero slice stand in for the tap after the last.
    // Resident weights are 9 tiles of the three dz; streamed ones wSlots tiles of a tap.
    const size_t weights = cin == 8 ? (size_t) (kTaps + 1)*weightTileBytes(cin, nTile) + kZeroZone
                         : wSlots == kTaps ? (size_t) 9*weightTileBytes(cin, 3*nTile) : (size_t) wSlots*weightTileBytes(cin, nTile);
    return sizeof(SliceBarriers) + 128 + (size_t) slots*sliceBytes(cin) + weights;
}

struct SliceItem {
    int n, x0, y0, z0, zc, co0;    // volume, origin of the column, first plane, planes, first output channel
};

__device__ __forceinline__ SliceItem sliceItem(const SliceParams& p, int item) {
    SliceItem t;
    int r = item;
    const int cx = r%p.colsX; r /= p.colsX;
    const int cy = r%p.colsY; r /= p.colsY;
    const int zb = r%p.zBlocks;
    t.n = r/p.zBlocks;
    t.x0 = cx*kTileX;
    t.y0 = cy*kTileY;
    t.z0 = zb*p.zLen;
    t.zc = min(p.zLen, p.D - t.z0);
    t.co0 = blockIdx.y*p.nTile;
    return t;
}

__device__ __forceinline__ void arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(mbar) : "memory");
}

// A bounded wait that also ends when another role of the CTA has given up; a wait that runs out makes all give up.
__device__ __forceinline__ bool waitOrStop(uint32_t mbar, uint32_t parity, long long limit, volatile int* stop) {
    for (long long i = 0; i < limit; i++) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
                     "selp.b32 %0, 1, 0, P1;\n\t}" : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
        if (done)
            return true;
        if (*stop)
            return false;
    }
    *stop = 1;
    return false;
}

__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// The 16-byte pieces of a copy that thread `first` of `step` threads takes, channel group fastest, without divisions in
// the loop: (g, v) is group g of voxel (or output channel) v.
struct Pieces {
    int g, v, groups, stepG, stepV;
    __device__ __forceinline__ Pieces(int first, int step, int groups)
            : g(first%groups), v(first/groups), groups(groups), stepG(step%groups), stepV(step/groups) {}
    __device__ __forceinline__ void next(int& pg, int& pv) const {
        pg += stepG;
        const bool carry = pg >= groups;
        pg -= carry ? groups : 0;
        pv += stepV + (carry ? 1 : 0);
    }
};

// The copies of one producer thread: groups are handed over (proxy fence, arrive) when they have landed, at most kLag
// of them in flight; a producer that has to wait for a free slot hands over all of them first, since the consumer may
// be waiting for exactly those.
struct CopyQueue {
    static constexpr int kLag = 3;
    uint32_t bars[kLag];
    int count = 0;
    __device__ __forceinline__ void pop() {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        arrive(bars[0]);
        for (int i = 1; i < kLag; i++)
            bars[i-1] = bars[i];
        count--;
    }
    __device__ __forceinline__ void push(uint32_t bar) {
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (int i = 0; i < kLag; i++)
            if (i == count)
                bars[i] = bar;
        count++;
        if (count == kLag) {
            asm volatile("cp.async.wait_group %0;" :: "n"(kLag - 1) : "memory");
            pop();
        }
    }
    __device__ __forceinline__ void flush() {
        asm volatile("cp.async.wait_all;" ::: "memory");
        while (count > 0)
            pop();
    }
    // Waits until `bar` has completed the phase `parity`.
    __device__ __forceinline__ bool waitFree(uint32_t bar, uint32_t parity, long long limit, volatile int* stop) {
        if (count > 0) {
            uint32_t done;
            asm volatile("{\n\t.reg .pred P1;\n\tmbarrier.test_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
                         "selp.b32 %0, 1, 0, P1;\n\t}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
            if (!done)
                flush();
        }
        return waitOrStop(bar, parity, limit, stop);
    }
};

// The MMA and the commit as a converged warp issues them: the whole warp computes the (uniform) operands, which keeps
// them in uniform registers, and one elected lane issues.
__device__ __forceinline__ void mmaElected(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\telect.sync _|q, 0xffffffff;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 :: "r"(tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void commitElected(uint32_t mbar) {
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" :: "r"(mbar) : "memory");
}
// waitOrStop by a whole warp, with one answer for all lanes.
__device__ __forceinline__ bool warpWait(uint32_t mbar, uint32_t parity, long long limit, volatile int* stop) {
    return __all_sync(0xffffffffu, waitOrStop(mbar, parity, limit, stop));
}

// A matrix descriptor from its words: the low one holds the start address and the leading offset, the high one the
// stride offset and the version (unswizzled layouts).
__device__ __forceinline__ uint64_t join(uint32_t low, uint32_t high) {
    return (uint64_t) high << 32 | low;
}

// How a CTA holds its weights: all 27 taps resident, streamed tap by tap, or resident with one channel group per tap
// (cin = 8), where an MMA takes two taps.
enum { kResident, kStreamed, kSingleGroup };

template <int MODE>
constexpr int sliceThreads = kEpilogueThreads + 32 + (MODE == kStreamed ? kProducersStreamed : kProducersResident);

template <int MODE>
__global__ void __launch_bounds__(sliceThreads<MODE>)
convSliceKernel(const SliceParams p) {
    extern __shared__ __align__(128) uint8_t smemRaw[];
    SliceBarriers* bars = reinterpret_cast<SliceBarriers*>(smemRaw);
    // Rows of a weight tile: a tap's output channels, or those of the three dz of a (dy, dx), dz = 2 first.
    const int tileRows = MODE == kResident ? 3*p.nTile : p.nTile;
    const int slotBytes = sliceBytes(p.cin), tileBytes = weightTileBytes(p.cin, tileRows);
    const uint32_t ring = (smemAddr(smemRaw) + (uint32_t) sizeof(SliceBarriers) + 127u) & ~127u;
    const uint32_t zeroZone = ring + (uint32_t) (p.slots*slotBytes);
    const uint32_t weights = zeroZone + (p.cin == 8 ? kZeroZone : 0);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid/32, 0), lane = tid%32;
    const uint32_t ncols = tmemColumns(p.accSlots*p.nTile);
    volatile int* stop = &bars->stop;
    constexpr bool resident = MODE != kStreamed;
    constexpr int producerThreads = sliceThreads<MODE> - kEpilogueThreads - 32;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smemAddr(&bars->tmem)), "r"(ncols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 32) {
        auto init = [](uint64_t* b, int count) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smemAddr(b)), "r"(count) : "memory");
        };
        for (int i = 0; i < p.slots; i++) {
            init(&bars->full[i], producerThreads);
            init(&bars->empty[i], 1);
        }
        for (int i = 0; i < p.wSlots; i++) {
            init(&bars->wFull[i], producerThreads);
            init(&bars->wEmpty[i], 1);
        }
        for (int i = 0; i < p.accSlots; i++) {
            init(&bars->accFull[i], 1);
            init(&bars->accEmpty[i], kEpilogueThreads);
        }
        init(&bars->drain, 1);
        bars->stop = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (p.cin == 8) {
        for (int i = tid; i < kZeroZone/16; i += sliceThreads<MODE>)
            *reinterpret_cast<uint4*>(smemRaw + (zeroZone - smemAddr(smemRaw)) + 16*i) = make_uint4(0, 0, 0, 0);
        for (int i = tid; i < tileBytes/16; i += sliceThreads<MODE>)
            *reinterpret_cast<uint4*>(smemRaw + (weights - smemAddr(smemRaw)) + kTaps*tileBytes + 16*i) = make_uint4(0, 0, 0, 0);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    fenceBeforeSync();
    __syncthreads();
    fenceAfterSync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, bars->tmem, 0);
    const long long limit = convWaitPolls;
    const int groups = p.cin/8;

    if (warp >= 5) {
        // ---- producers: slices in the order of the planes and the weight tiles in the order of their use, each shared by
        // all threads (a streamed tile by one warp: 224 -> 64 channels at 16x16x32 x 2 in 74 us instead of 59) ----
        const int t = tid - (kEpilogueThreads + 32), producers = producerThreads;
        CopyQueue queue;
        const Pieces bySlice(t, producers, groups), byAll(t, producers, groups);
        const int groupW = weightGroupBytes(tileRows);
        int slot = 0, wSlot = 0;
        uint32_t slotPhase = 1, wPhase = 1;        // a free slot's barrier has completed the phase before its first
        bool ok = true;
        auto copyTile = [&](const Pieces& pieces, int at, int row, int tap, int co0) {
            const uint32_t base = weights + (uint32_t) (at*tileBytes + row*16);
            const __nv_bfloat16* src = p.w + ((size_t) co0*kTaps + tap)*p.cin;
            for (int g = pieces.g, n = pieces.v; n < p.nTile; ) {
                copy16(base + (uint32_t) (g*groupW + n*16), src + (size_t) n*kTaps*p.cin + 8*g, true);
                pieces.next(g, n);
            }
        };
        for (int item = blockIdx.x; item < p.items && ok; item += gridDim.x) {
            const SliceItem it = sliceItem(p, item);
            for (int s = 0; s < it.zc + 2 && ok; s++) {
                const int z = it.z0 + s - 1;
                ok = queue.waitFree(smemAddr(&bars->empty[slot]), slotPhase, limit, stop);
                if (!ok)
                    break;
                const uint32_t base = ring + (uint32_t) (slot*slotBytes);
                const bool inside = z >= 0 && z < p.D;
                const __nv_bfloat16* plane = p.x + ((size_t) it.n*p.D + (inside ? z : 0))*p.H*p.W*p.cin;
                for (int g = bySlice.g, v = bySlice.v; v < kSliceVoxels; ) {
                    const int vy = v/kHaloX, yy = it.y0 + vy - 1, xx = it.x0 + (v - vy*kHaloX) - 1;
                    const bool valid = inside && (unsigned) yy < (unsigned) p.H && (unsigned) xx < (unsigned) p.W;
                    copy16(base + (uint32_t) (g*kPlane + v*16), plane + (valid ? (yy*p.W + xx)*p.cin + 8*g : 0), valid);
                    bySlice.next(g, v);
                }
                queue.push(smemAddr(&bars->full[slot]));
                if (++slot == p.slots) {
                    slot = 0;
                    slotPhase ^= 1;
                }
                for (int dz = 2; dz >= 0 && ok; dz--) {
                    // Plane z0 + s - dz takes the taps 9 dz .. 9 dz + 8 from this slice; resident tiles come with the
                    // CTA's first plane.
                    if (s - dz < 0 || s - dz >= it.zc || (resident && (item != blockIdx.x || s != dz)))
                        continue;
                    for (int k = 0; k < 9 && ok; k++) {
                        if (resident) {
                            MODE == kResident ? copyTile(byAll, k, (2 - dz)*p.nTile, 9*dz + k, it.co0)
                                              : copyTile(byAll, 9*dz + k, 0, 9*dz + k, it.co0);
                            continue;
                        }
                        ok = queue.waitFree(smemAddr(&bars->wEmpty[wSlot]), wPhase, limit, stop);
                        if (!ok)
                            break;
                        copyTile(byAll, wSlot, 0, 9*dz + k, it.co0);
                        queue.push(smemAddr(&bars->wFull[wSlot]));
                        if (++wSlot == p.wSlots) {
                            wSlot = 0;
                            wPhase ^= 1;
                        }
                    }
                    if (resident)
                        queue.push(smemAddr(&bars->wFull[dz]));
                }
            }
        }
        queue.flush();
    }
    else if (warp == 4) {
        // ---- the MMAs: the instructions between two of them are what a narrow layer waits for, so the taps are
        // unrolled, a descriptor is its low word plus a constant, and the warp stays converged (uniform registers) ----
        {
            const uint32_t idesc = instrDescriptor(p.nTile), idesc2 = instrDescriptor(2*p.nTile), idesc3 = instrDescriptor(3*p.nTile);
            const uint32_t groupW = (uint32_t) weightGroupBytes(tileRows), tileUnits = (uint32_t) tileBytes/16;
            const uint32_t aHigh = (kHaloX*16 >> 4) | (1u << 14), bHigh = (128 >> 4) | (1u << 14);
            const uint32_t wLow = (weights >> 4) | ((MODE == kSingleGroup ? (uint32_t) tileBytes : groupW) >> 4 << 16);
            int plane0 = 0, slot = 0, wSlot = 0;
            uint32_t slotPhase = 0, wPhase = 0;
            bool ok = true, issued = false;
            for (int item = blockIdx.x; item < p.items && ok; item += gridDim.x) {
                const SliceItem it = sliceItem(p, item);
                for (int s = 0; s < it.zc + 2 && ok; s++) {
                    ok = warpWait(smemAddr(&bars->full[slot]), slotPhase, limit, stop);
                    if (!ok)
                        break;
                    const uint32_t base = ring + (uint32_t) (slot*slotBytes);
                    if constexpr (MODE == kResident) {
                        // The slice's planes s - 2, s - 1 and s take the taps dz = 2, 1 and 0 of every (dy, dx) from the
                        // same rows of A: one MMA with their accumulators side by side (two where the ring of
                        // accumulators wraps around between them).
                        const int lo = max(0, s - 2), hi = min(it.zc - 1, s), count = hi - lo + 1;
                        if (hi == s && plane0 + s >= p.accSlots) {
                            const int plane = plane0 + s;
                            ok = warpWait(smemAddr(&bars->accEmpty[plane%p.accSlots]), (uint32_t) ((plane/p.accSlots - 1) & 1), limit, stop);
                            fenceAfterSync();
                        }
                        if (item == blockIdx.x && s <= 2)
                            ok = ok && warpWait(smemAddr(&bars->wFull[s]), 0, limit, stop);
                        if (!ok)
                            break;
                        issued = true;
                        const uint32_t aLow = (base >> 4) | (uint32_t) (kPlane/16) << 16;
                        // The MMAs of (dy, dx) = r for `n` planes from accumulator `acc` on, rows of the tile from `row` on.
                        auto multiply = [&](int r, int acc, uint32_t row, int n, uint32_t accumulate) {
                            const uint32_t d = tmem + (uint32_t) (acc*p.nTile), id = n == 3 ? idesc3 : (n == 2 ? idesc2 : idesc);
                            uint32_t a = aLow + (uint32_t) ((r/3)*kHaloX + r%3), b = wLow + (uint32_t) r*tileUnits + row;
                            mmaElected(d, join(a, aHigh), join(b, bHigh), id, accumulate);
                            for (int g = 2; g < groups; g += 2) {
                                a += 2*kPlane/16;
                                b += groupW/8;
                                mmaElected(d, join(a, aHigh), join(b, bHigh), id, 1u);
                            }
                        };
                        const int acc = (plane0 + lo)%p.accSlots, head = min(count, p.accSlots - acc), tail = count - head;
                        const uint32_t row = (uint32_t) ((2 - s + lo)*p.nTile), rowTail = row + (uint32_t) (head*p.nTile);
                        // A plane that starts here overwrites its accumulator in its first MMA.
                        if (hi == s) {
                            const int older = count - 1, olderHead = min(older, head), olderTail = older - olderHead;
                            if (olderHead > 0)
                                multiply(0, acc, row, olderHead, 1u);
                            if (olderTail > 0)
                                multiply(0, 0, rowTail, olderTail, 1u);
                            multiply(0, (plane0 + s)%p.accSlots, 2u*(uint32_t) p.nTile, 1, 0u);
                        }
                        else {
                            multiply(0, acc, row, head, 1u);
                            if (tail > 0)
                                multiply(0, 0, rowTail, tail, 1u);
                        }
                        if (tail == 0) {
#pragma unroll
                            for (int r = 1; r < 9; r++)
                                multiply(r, acc, row, head, 1u);
                        }
                        else {
#pragma unroll
                            for (int r = 1; r < 9; r++) {
                                multiply(r, acc, row, head, 1u);
                                multiply(r, 0, rowTail, tail, 1u);
                            }
                        }
                        if (s >= 2)
                            commitElected(smemAddr(&bars->accFull[(plane0 + s - 2)%p.accSlots]));
                    }
                    auto stage = [&](auto dzc) {
                        constexpr int dz = decltype(dzc)::value;
                        const int k0 = s - dz;
                        if (k0 < 0 || k0 >= it.zc || !ok)
                            return;
                        const int plane = plane0 + k0, acc = plane%p.accSlots;
                        const uint32_t d = tmem + (uint32_t) (acc*p.nTile);
                        if (dz == 0 && plane >= p.accSlots) {
                            ok = warpWait(smemAddr(&bars->accEmpty[acc]), (uint32_t) ((plane/p.accSlots - 1) & 1), limit, stop);
                            if (!ok)
                                return;
                            fenceAfterSync();
                        }
                        if (MODE != kStreamed && item == blockIdx.x && k0 == 0)
                            ok = warpWait(smemAddr(&bars->wFull[dz]), 0, limit, stop);
                        if (!ok)
                            return;
                        issued = true;
                        if constexpr (MODE == kSingleGroup) {
                            // Two taps per MMA, (0,1) (2,3) ... (26, zero): K = 16 is two groups a leading offset apart.
                            constexpr int first = dz == 0 ? 0 : (dz == 1 ? 8 : 18), count = dz == 0 ? 4 : 5;
#pragma unroll
                            for (int i = 0; i < count; i++) {
                                const int tap = first + 2*i, r = tap%9, r1 = (tap + 1)%9;
                                const uint32_t here = base - (tap == 8 ? (uint32_t) slotBytes : 0u);
                                const uint32_t from = here + (uint32_t) ((r/3)*kHaloX + r%3)*16;
                                const uint32_t to = tap == 26 ? zeroZone : base + (uint32_t) ((r1/3)*kHaloX + r1%3)*16;
                                mmaElected(d, join((from >> 4) | ((to - from) >> 4 << 16), aHigh),
                                        join(wLow + (uint32_t) tap*tileUnits, bHigh), idesc, tap > 0 ? 1u : 0u);
                            }
                        }
                        else {
                            const uint32_t aLow = (base >> 4) | (uint32_t) (kPlane/16) << 16;
                            uint32_t bLow = wLow + 9*dz*tileUnits;
#pragma unroll
                            for (int r = 0; r < 9; r++) {
                                if constexpr (MODE == kStreamed) {
                                    ok = ok && warpWait(smemAddr(&bars->wFull[wSlot]), wPhase, limit, stop);
                                    if (!ok)
                                        return;
                                    bLow = wLow + (uint32_t) wSlot*tileUnits;
                                }
                                uint32_t a = aLow + (uint32_t) ((r/3)*kHaloX + r%3), b = bLow;
                                mmaElected(d, join(a, aHigh), join(b, bHigh), idesc, dz > 0 || r > 0 ? 1u : 0u);
                                for (int g = 2; g < groups; g += 2) {
                                    a += 2*kPlane/16;
                                    b += groupW/8;
                                    mmaElected(d, join(a, aHigh), join(b, bHigh), idesc, 1u);
                                }
                                if constexpr (MODE == kStreamed) {
                                    commitElected(smemAddr(&bars->wEmpty[wSlot]));
                                    if (++wSlot == p.wSlots) {
                                        wSlot = 0;
                                        wPhase ^= 1;
                                    }
                                }
                                else
                                    bLow += tileUnits;
                            }
                        }
                        if (dz == 2)
                            commitElected(smemAddr(&bars->accFull[acc]));
                    };
                    if constexpr (MODE != kResident) {
                        stage(std::integral_constant<int, 2>());
                        stage(std::integral_constant<int, 1>());
                        stage(std::integral_constant<int, 0>());
                    }
                    if (!ok)
                        break;
                    // The slice is free once its MMAs are done; with one group the next slice's first pair still reads
                    // it, so each slice is freed one slice later, the last two of a column together.
                    if (MODE != kSingleGroup)
                        commitElected(smemAddr(&bars->empty[slot]));
                    else {
                        if (s > 0)
                            commitElected(smemAddr(&bars->empty[slot - 1]));
                        if (s == it.zc + 1)
                            commitElected(smemAddr(&bars->empty[slot]));
                    }
                    if (++slot == p.slots) {
                        slot = 0;
                        slotPhase ^= 1;
                    }
                }
                plane0 += it.zc;
            }
            // The MMAs and arrivals in flight end before the CTA leaves (a role may have given up).
            if (issued) {
                commitElected(smemAddr(&bars->drain));
                waitParity(smemAddr(&bars->drain), 0, kSpinLimit);
                __syncwarp();
            }
        }
    }
    else {
        // ---- epilogue: warp w owns the lanes 32 w .. 32 w + 31 of the accumulators, rows of the tile.  A load from tensor
        // memory needs the whole warp: all lanes take one answer of the wait, and come together again after the stores of
        // those whose voxel lies in the volume ----
        const int row = warp*32 + lane, vx = row%kTileX, vy = row/kTileX;
        int plane0 = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < p.items && ok; item += gridDim.x) {
            const SliceItem it = sliceItem(p, item);
            const int xx = it.x0 + vx, yy = it.y0 + vy;
            const bool store = xx < p.W && yy < p.H;
            for (int k = 0; k < it.zc; k++) {
                const int plane = plane0 + k, acc = plane%p.accSlots;
                ok = warpWait(smemAddr(&bars->accFull[acc]), (uint32_t) ((plane/p.accSlots) & 1), limit, stop);
                if (!ok)
                    break;
                fenceAfterSync();
                const uint32_t d = tmem + ((uint32_t) (warp*32) << 16) + (uint32_t) (acc*p.nTile);
                __nv_bfloat16* out = p.y + ((((size_t) it.n*p.D + it.z0 + k)*p.H + yy)*p.W + xx)*p.cout + it.co0;
                for (int col = 0; col < p.nTile; col += 16) {
                    uint32_t v[16];
                    tmemLoad16(d + (uint32_t) col, v);
                    if (store) {
                        __align__(16) __nv_bfloat16 o[16];
#pragma unroll
                        for (int i = 0; i < 16; i++) {
                            const float f = __uint_as_float(v[i]) + (p.bias ? __ldg(p.bias + it.co0 + col + i) : 0.0f);
                            o[i] = __float2bfloat16_rn(p.relu ? fmaxf(f, 0.0f) : f);
                        }
                        reinterpret_cast<uint4*>(out + col)[0] = reinterpret_cast<const uint4*>(o)[0];
                        reinterpret_cast<uint4*>(out + col)[1] = reinterpret_cast<const uint4*>(o)[1];
                    }
                    __syncwarp();
                }
                fenceBeforeSync();
                arrive(smemAddr(&bars->accEmpty[acc]));
            }
            plane0 += it.zc;
        }
    }
    fenceBeforeSync();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(ncols) : "memory");
    if (tid == 0 && bars->stop)
        atomicExch(&convStatus, (int) LBM_ERR_DEVICE_TIMEOUT);
}

__global__ void __launch_bounds__(kThreads)
convForwardKernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, const float* __restrict__ bias,
                  __nv_bfloat16* __restrict__ y, int batch, int D, int H, int W, int cin, int cout, int relu) {
    extern __shared__ uint8_t smemRaw[];
    const uint32_t ncols = tmemColumns(cout);
    Stage st = setupStage(smemRaw, cout, ncols);
    const int tid = threadIdx.x, warp = tid/32, lane = tid%32;
    const long long M = (long long) batch*D*H*W;
    const int K = 27*cin, stages = (K + kChunk - 1)/kChunk;
    const uint32_t idesc = instrDescriptor(cout);
    // The voxel of this thread's row of A.
    const long long m = (long long) blockIdx.x*kTileM + tid;
    const bool valid = m < M;
    int vx = 0, vy = 0, vz = 0, vn = 0;
    if (valid) {
        long long r = m;
        vx = (int) (r%W); r /= W;
        vy = (int) (r%H); r /= H;
        vz = (int) (r%D); vn = (int) (r/D);
    }
    const long long limit = convWaitPolls;
    bool ok = true;
    int failedStage = -1;
    for (int c = 0; c < stages && ok; c++) {
        for (int kv = 0; kv < 8; kv++) {
            int k = c*kChunk + kv*8;
            uint4 val = make_uint4(0, 0, 0, 0);
            if (valid && k < K) {
                int tap = k/cin, ci = k - tap*cin;
                int zz = vz + tap/9 - 1, yy = vy + (tap/3)%3 - 1, xx = vx + tap%3 - 1;
                if (zz >= 0 && zz < D && yy >= 0 && yy < H && xx >= 0 && xx < W)
                    val = __ldg(reinterpret_cast<const uint4*>(x + ((((long long) vn*D + zz)*H + yy)*W + xx)*cin + ci));
            }
            *reinterpret_cast<uint4*>(st.tileA + swizzled(tid, kv)) = val;
        }
        for (int i = tid; i < cout*8; i += kThreads) {
            int row = i >> 3, kv = i & 7, k = c*kChunk + kv*8;
            uint4 val = make_uint4(0, 0, 0, 0);
            if (k < K)
                val = __ldg(reinterpret_cast<const uint4*>(w + (long long) row*K + k));
            *reinterpret_cast<uint4*>(st.tileB + swizzled(row, kv)) = val;
        }
        ok = runStage(st, idesc, c, limit);
        if (!ok)
            failedStage = c;
    }
    if (!ok)
        drainStage(st, failedStage);
    fenceAfterSync();
    if (ok) {
        const int row = warp*32 + lane;
        const long long mo = (long long) blockIdx.x*kTileM + row;
        for (int col = 0; col < cout; col += 8) {
            float v[8];
            tmemLoad8(st.tmem + ((uint32_t) (warp*32) << 16) + (uint32_t) col, v);
            if (mo < M) {
                __align__(16) __nv_bfloat16 out[8];
                for (int i = 0; i < 8; i++) {
                    float t = v[i] + (bias ? bias[col + i] : 0.0f);
                    out[i] = __float2bfloat16_rn(relu ? fmaxf(t, 0.0f) : t);
                }
                *reinterpret_cast<uint4*>(y + mo*cout + col) = *reinterpret_cast<const uint4*>(out);
            }
            __syncwarp();
        }
    }
    else if (tid == 0)
        atomicExch(&convStatus, (int) LBM_ERR_DEVICE_TIMEOUT);
    releaseStage(st, ncols);
}

// ---------------------------------------------------------------------------------------------------------------
// The weight gradient dw[co][tap][ci] += sum_v dy[v][co] x[v + tap][ci]: GEMMs whose K are the voxels, with both
// operands in the unswizzled MN-major layout, 8 channels x 8 voxels of 16 bytes a core matrix, 16 x-neighbours (two
// core matrices) per tcgen05.mma.  One MMA serves many taps at once:
//   M (128 rows)  the channels of x on the rows y - 1, y, y + 1: [row][8-channel group] is one sequence of groups at
//                 one stride, so 3 `groupsX` groups (at most 15 of the tile's 16) cover the taps' dy; what the other
//                 rows of the tile read is never looked at
//   N             the channels of dy in three copies, each shifted by one voxel in x: [dz][dx][8-channel group], again
//                 at one stride: N = 3 coTile, or 9 coTile where all three planes fit into 256 columns
// A CTA takes `groupsX` groups of input channels, coTile output channels and all dz (dzCount = 3), or one (more than 48
// output channels: the accumulators of all would not fit into tensor memory).  It walks over its share of the items, columns
// of 16 x 8 voxels (x, y) over zLen planes; warps 0-7 copy slices of x into a ring and the shifted copies of dy into two
// buffers, warp 8 issues the MMAs, and warps 9-16 add finished sums to dw with FP32 atomics.
//
// The tensor core truncates its running sums: their relative error grows by about 2^-25 per MMA.  So a sum is handed to the
// atomics (rounded to nearest) after `chain` MMAs at most (8 to 48, planGradient), and the accumulators are a ring of units
// (all dz of an MMA, or one) that are read and cleared while the next unit fills.
//
// Bound: 16 -> 16 channels read 4 KB of x and 4.6 KB of dy (68 wavefronts of shared memory) per MMA and 16 voxels, 19 us
// on two 64 x 64 x 128 volumes.  Measured there: 76 us, what remains being the copies (dy three times) and the atomics of
// the finished sums (a quarter less, with an error of 4e-6 instead of 9e-7, when a CTA adds its sums once); 1150 us with
// the kernel before it, which gathered both operands transposed element by element and waited for each stage.  48 -> 16:
// 160 us (4000), 32 -> 32 at 32 x 32 x 64 29 us (314), 160 -> 160 at 8 x 8 x 16 25 us (116).
// ---------------------------------------------------------------------------------------------------------------

constexpr int kRunX = 16, kRowsY = 8;
constexpr int kGroupPitch = kRunX*16 + 16;     // bytes of a group's 16 voxels; + 16 spreads the groups over the banks
constexpr int kGradSlots = 4;
constexpr int kGradProducers = 256, kGradReaders = 256;
constexpr int kGradThreads = kGradProducers + 32 + kGradReaders, kMaxUnits = 5;
constexpr int kGradPiecesX = 4;                // (kRowsY + 2) kRunX 5 groups / kGradProducers
constexpr int kGradPieces = 6;                 // up to 32 output channels; more are placed piece by piece

struct GradParams {
    const __nv_bfloat16* x;
    const __nv_bfloat16* dy;
    float* dw;
    int batch, D, H, W, cin, cout;
    int groupsX, chunks, coTile, coBlocks, dzCount, zLen, chain;
    int colsX, colsY, zBlocks, items;
};

struct GradBarriers {
    uint64_t full[kGradSlots], empty[kGradSlots], dyEmpty[2], unitFull[kMaxUnits], unitEmpty[kMaxUnits], drain;
    uint32_t tmem;
    int stop;
};

__host__ __device__ inline int gradSliceBytes(int groupsX) { return (kRowsY + 2)*groupsX*kGroupPitch; }
__host__ __device__ inline int gradDyBytes(int coTile, int zLen) { return kRowsY*zLen*3*(coTile/8)*kGroupPitch; }
__host__ __device__ inline size_t gradSmemBytes(int groupsX, int coTile, int zLen) {
    // The last row's tile reads 16 groups, 3 groupsX of which are its own.
    return sizeof(GradBarriers) + 128 + (size_t) kGradSlots*gradSliceBytes(groupsX) + 16*kGroupPitch
         + 2*(size_t) gradDyBytes(coTile, zLen);
}

__global__ void __launch_bounds__(kGradThreads)
convSliceGradKernel(const GradParams p) {
    extern __shared__ __align__(128) uint8_t smemRaw[];
    GradBarriers* bars = reinterpret_cast<GradBarriers*>(smemRaw);
    const int slotBytes = gradSliceBytes(p.groupsX), dyBytes = gradDyBytes(p.coTile, p.zLen);
    const uint32_t ring = (smemAddr(smemRaw) + (uint32_t) sizeof(GradBarriers) + 127u) & ~127u;
    const uint32_t dyBase = ring + (uint32_t) (kGradSlots*slotBytes + 16*kGroupPitch);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid/32, 0), lane = tid%32;
    const int width = 3*p.coTile;                     // columns per dz
    // Accumulators: units of all dz (one MMA serves them) or of one.
    const bool merged = p.dzCount*width <= 256;
    const int unitsPerSum = merged ? 1 : p.dzCount, unitWidth = merged ? p.dzCount*width : width;
    const int units = min(kMaxUnits, 512/unitWidth);
    const uint32_t ncols = tmemColumns(units*unitWidth);
    volatile int* stop = &bars->stop;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smemAddr(&bars->tmem)), "r"(ncols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 32) {
        auto init = [](uint64_t* b, int count) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smemAddr(b)), "r"(count) : "memory");
        };
        for (int i = 0; i < kGradSlots; i++) {
            init(&bars->full[i], kGradProducers);
            init(&bars->empty[i], 1);
        }
        init(&bars->dyEmpty[0], 1);
        init(&bars->dyEmpty[1], 1);
        for (int i = 0; i < units; i++) {
            init(&bars->unitFull[i], 1);
            init(&bars->unitEmpty[i], kGradReaders);
        }
        init(&bars->drain, 1);
        bars->stop = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    fenceBeforeSync();
    __syncthreads();
    fenceAfterSync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, bars->tmem, 0);
    // The accumulators start at zero, so that every MMA adds.  Warps 9-16 own the lanes 32 (warp % 4) and on, every other
    // 16 columns each.
    const uint32_t laneBase = tmem + ((uint32_t) (warp%4*32) << 16);
    const int share = warp > kGradProducers/32 + 4 ? 16 : 0;
    auto clear = [&](int from, int count) {
        for (int c = from + share; c < from + count; c += 32)
            for (int h = 0; h < 16; h += 8)
                asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};"
                             :: "r"(laneBase + (uint32_t) (c + h)), "r"(0) : "memory");
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    };
    if (warp > kGradProducers/32)
        clear(0, units*unitWidth);
    fenceBeforeSync();
    __syncthreads();
    fenceAfterSync();
    const long long limit = convWaitPolls;
    int block = blockIdx.y;
    const int chunk = block%p.chunks; block /= p.chunks;
    const int co0 = block%p.coBlocks*p.coTile;
    const int dzOnly = p.dzCount == 3 ? 0 : block/p.coBlocks;
    const int group0 = chunk*p.groupsX, groupsX = min(p.groupsX, p.cin/8 - group0), groupsY = p.coTile/8;
    // Slices of an item: every plane's three with all dz, else the one that its dz reads.
    const int halo = p.dzCount - 1;
    auto item = [&](int i, int& n, int& z0, int& zc, int& y0, int& x0) {
        x0 = i%p.colsX*kRunX; i /= p.colsX;
        y0 = i%p.colsY*kRowsY; i /= p.colsY;
        z0 = i%p.zBlocks*p.zLen;
        n = i/p.zBlocks;
        zc = min(p.zLen, p.D - z0);
    };
    // A sum of `chain` MMAs ends with item i where this is the CTA's last or a whole item more could be too much.
    const int room = p.chain - kRowsY*p.zLen;

    if (warp < kGradProducers/32) {
        CopyQueue queue;
        const Pieces byX(tid, kGradProducers, groupsX), byY(tid, kGradProducers, groupsY);
        int slot = 0, buffer = 0;
        uint32_t slotPhase = 1, dyPhase = 1;         // a free slot's barrier has completed the phase before its first
        bool ok = true;
        // A thread's pieces have the same place in a slice, or in a plane of dy, and the same distance in memory from the
        // item's origin, for every item: both are formed once, an item adds which of them lie in the volume, and a copy is
        // a few instructions (16 -> 16 channels on two 64 x 64 x 128 volumes: 78 us, 87 with them formed for every copy).
        const int totalX = (kRowsY + 2)*kRunX*groupsX, totalY = kRowsY*3*kRunX*groupsY;
        const int mineX = (totalX - tid + kGradProducers - 1)/kGradProducers;
        const bool fewY = totalY <= kGradPieces*kGradProducers;
        const int mineY = fewY ? (totalY - tid + kGradProducers - 1)/kGradProducers : 0;
        uint32_t placeX[kGradPiecesX], placeY[kGradPieces], whereX[kGradPiecesX], whereY[kGradPieces];
        ptrdiff_t fromX[kGradPiecesX], fromY[kGradPieces];
        {
            int g = byX.g, v = byX.v;
#pragma unroll
            for (int j = 0; j < kGradPiecesX; j++) {
                const int k = v%kRunX, y = v/kRunX;
                placeX[j] = (uint32_t) ((y*groupsX + g)*kGroupPitch + k*16);
                fromX[j] = ((ptrdiff_t) (y - 1)*p.W + k)*p.cin + 8*g;
                whereX[j] = (uint32_t) (y | k << 16);
                byX.next(g, v);
            }
            g = byY.g;
            v = byY.v;
#pragma unroll
            for (int j = 0; j < kGradPieces; j++) {
                const int k = v%kRunX, r = v/kRunX, y = r/3, dx = r - 3*y;
                placeY[j] = (uint32_t) (((y*p.zLen*3 + dx)*groupsY + g)*kGroupPitch + k*16);
                fromY[j] = ((ptrdiff_t) y*p.W + k + 1 - dx)*p.cout + 8*g;
                whereY[j] = (uint32_t) (y | (k + 2 - dx) << 16);
                byY.next(g, v);
            }
        }
        for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
            int n, z0, zc, y0, x0;
            item(i, n, z0, zc, y0, x0);
            const size_t origin = (size_t) y0*p.W + x0;
            uint32_t inX = 0, inY = 0;
#pragma unroll
            for (int j = 0; j < kGradPiecesX; j++)
                if ((unsigned) (y0 - 1 + (int) (whereX[j] & 0xFFFFu)) < (unsigned) p.H && x0 + (int) (whereX[j] >> 16) < p.W)
                    inX |= 1u << j;
#pragma unroll
            for (int j = 0; j < kGradPieces; j++)
                if (y0 + (int) (whereY[j] & 0xFFFFu) < p.H && (unsigned) (x0 - 1 + (int) (whereY[j] >> 16)) < (unsigned) p.W)
                    inY |= 1u << j;
            ok = queue.waitFree(smemAddr(&bars->dyEmpty[buffer]), dyPhase, limit, stop);
            for (int j = 0; j < zc + halo && ok; j++) {
                if (j < zc) {
                    // Plane z0 + j of dy: copy dx holds dy at x - (dx - 1).
                    const __nv_bfloat16* plane = p.dy + ((size_t) n*p.D + z0 + j)*p.H*p.W*p.cout + co0;
                    const uint32_t base = dyBase + (uint32_t) (buffer*dyBytes);
                    if (fewY) {
                        const uint32_t at = base + (uint32_t) (j*3*groupsY*kGroupPitch);
                        const __nv_bfloat16* from = plane + origin*p.cout;
#pragma unroll
                        for (int k = 0; k < kGradPieces; k++)
                            if (k < mineY) {
                                const bool valid = (inY >> k) & 1u;
                                copy16(at + placeY[k], valid ? from + fromY[k] : p.dy, valid);
                            }
                    }
                    else for (int g = byY.g, v = byY.v; v < kRowsY*3*kRunX; ) {
                        const int k = v%kRunX, r = v/kRunX, y = r/3, dx = r%3;
                        const int yy = y0 + y, xx = x0 + k + 1 - dx;
                        const bool valid = yy < p.H && (unsigned) xx < (unsigned) p.W;
                        copy16(base + (uint32_t) ((((y*p.zLen + j)*3 + dx)*groupsY + g)*kGroupPitch + k*16),
                               plane + (valid ? ((size_t) yy*p.W + xx)*p.cout + 8*g : 0), valid);
                        byY.next(g, v);
                    }
                }
                ok = queue.waitFree(smemAddr(&bars->empty[slot]), slotPhase, limit, stop);
                if (!ok)
                    break;
                const int z = p.dzCount == 3 ? z0 + j - 1 : z0 + j + dzOnly - 1;
                const bool inside = z >= 0 && z < p.D;
                const __nv_bfloat16* plane = p.x + ((size_t) n*p.D + (inside ? z : 0))*p.H*p.W*p.cin + 8*group0;
                const uint32_t base = ring + (uint32_t) (slot*slotBytes);
                const __nv_bfloat16* from = plane + origin*p.cin;
#pragma unroll
                for (int k = 0; k < kGradPiecesX; k++)
                    if (k < mineX) {
                        const bool valid = inside && ((inX >> k) & 1u);
                        copy16(base + placeX[k], valid ? from + fromX[k] : p.x, valid);
                    }
                queue.push(smemAddr(&bars->full[slot]));
                if (++slot == kGradSlots) {
                    slot = 0;
                    slotPhase ^= 1;
                }
            }
            buffer ^= 1;
            dyPhase ^= buffer == 0 ? 1 : 0;
        }
        queue.flush();
    }
    else if (warp == kGradProducers/32) {
        // Both operands MN-major (bits 15 and 16 of the instruction descriptor).
        const uint32_t high = (kGroupPitch >> 4) | (1u << 14), low = (128u >> 4) << 16;
        const uint32_t rowX = (uint32_t) (groupsX*kGroupPitch) >> 4;
        const uint32_t planeY = (uint32_t) (3*groupsY*kGroupPitch) >> 4, rowY = planeY*(uint32_t) p.zLen;
        int slot = 0, buffer = 0, unit = 0, chain = 0;
        uint32_t slotPhase = 0, unitPhase = 1;       // of the sum's first unit
        bool ok = true, issued = false;
        for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
            int n, z0, zc, y0, x0;
            item(i, n, z0, zc, y0, x0);
            const int rows = min(kRowsY, p.H - y0);
            // A new sum waits for its units to have been read and cleared.
            for (int k = 0; k < unitsPerSum && ok && chain == 0; k++) {
                const int at = unit + k;
                ok = warpWait(smemAddr(&bars->unitEmpty[at%units]), unitPhase ^ (at >= units ? 1u : 0u), limit, stop);
                fenceAfterSync();
            }
            for (int j = 0; j < zc + halo && ok; j++) {
                ok = warpWait(smemAddr(&bars->full[slot]), slotPhase, limit, stop);
                if (!ok)
                    break;
                // Slice j meets the planes k of dy with dz = j - k (all dz), in columns of their own, dz = 2 first.
                const int first = max(0, j - halo), last = min(zc - 1, j);
                const int count = last - first + 1, step = merged ? count : 1;
                const uint32_t idesc = instrDescriptor(step*width) | (1u << 15) | (1u << 16);
                const uint32_t a = low | ((ring + (uint32_t) (slot*slotBytes)) >> 4);
                const uint32_t b = low | (((dyBase + (uint32_t) (buffer*dyBytes)) >> 4) + (uint32_t) first*planeY);
                // The rows of an accumulator one after another: an MMA is two additions and its issue (90 -> 87 us).
                for (int k = 0; k < count; k += step) {
                    const int column = halo - j + first + k, at = unit + column;
                    const uint32_t d = tmem + (uint32_t) (merged ? unit*unitWidth + column*width : (at >= units ? at - units : at)*width);
                    const uint32_t bk = b + (uint32_t) k*planeY;
                    if (rows == kRowsY) {
#pragma unroll
                        for (int y = 0; y < kRowsY; y++)
                            mmaElected(d, join(a + (uint32_t) y*rowX, high), join(bk + (uint32_t) y*rowY, high), idesc, 1u);
                    }
                    else
                        for (int y = 0; y < rows; y++)
                            mmaElected(d, join(a + (uint32_t) y*rowX, high), join(bk + (uint32_t) y*rowY, high), idesc, 1u);
                }
                issued = true;
                commitElected(smemAddr(&bars->empty[slot]));
                if (++slot == kGradSlots) {
                    slot = 0;
                    slotPhase ^= 1;
                }
            }
            if (!ok)
                break;
            commitElected(smemAddr(&bars->dyEmpty[buffer]));
            buffer ^= 1;
            chain += rows*zc;
            if (chain > room || i + (int) gridDim.x >= p.items) {
                for (int k = 0; k < unitsPerSum; k++)
                    commitElected(smemAddr(&bars->unitFull[(unit + k)%units]));
                unit += unitsPerSum;
                if (unit >= units) {
                    unit -= units;
                    unitPhase ^= 1;
                }
                chain = 0;
            }
        }
        // The MMAs and arrivals in flight end before the CTA leaves.
        if (issued) {
            commitElected(smemAddr(&bars->drain));
            waitParity(smemAddr(&bars->drain), 0, kSpinLimit);
            __syncwarp();
        }
    }
    else {
        // Row 32 (warp % 4) + lane is (dy tap, channel group, channel), column ((2 - dz) 3 + dx) coTile + co.
        const int row = warp%4*32 + lane, group = row/8;
        const int ty = group/groupsX, ci = 8*(group0 + group%groupsX) + row%8;
        int unit = 0, chain = 0;
        uint32_t unitPhase = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < p.items && ok; i += gridDim.x) {
            int n, z0, zc, y0, x0;
            item(i, n, z0, zc, y0, x0);
            chain += min(kRowsY, p.H - y0)*zc;
            if (chain <= room && i + (int) gridDim.x < p.items)
                continue;
            chain = 0;
            for (int k = 0; k < unitsPerSum && ok; k++) {
                ok = warpWait(smemAddr(&bars->unitFull[unit]), unitPhase, limit, stop);
                if (!ok)
                    break;
                fenceAfterSync();
                for (int c = share; c < unitWidth; c += 32) {
                    uint32_t v[16];
                    tmemLoad16(laneBase + (uint32_t) (unit*unitWidth + c), v);
                    const int co = c%p.coTile, r = c/p.coTile + 3*k, dx = r%3, dz = p.dzCount == 3 ? 2 - r/3 : dzOnly;
                    if (ty < 3) {
                        float* out = p.dw + ((size_t) (co0 + co)*kTaps + 9*dz + 3*ty + dx)*p.cin + ci;
#pragma unroll
                        for (int q = 0; q < 16; q++)
                            atomicAdd(out + (size_t) q*kTaps*p.cin, __uint_as_float(v[q]));
                    }
                    __syncwarp();
                }
                clear(unit*unitWidth, unitWidth);
                fenceBeforeSync();
                arrive(smemAddr(&bars->unitEmpty[unit]));
                if (++unit == units) {
                    unit = 0;
                    unitPhase ^= 1;
                }
            }
        }
    }
    fenceBeforeSync();
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(ncols) : "memory");
    if (tid == 0 && bars->stop)
        atomicExch(&convStatus, (int) LBM_ERR_DEVICE_TIMEOUT);
}

size_t stageBytes(int rowsB) {
    return 1024 + (size_t) kTileM*128 + (size_t) rowsB*128 + 64;
}

// The slice kernel's division of a layer: which channels, planes and slots a CTA takes.  false where it does not apply
// (cin of an odd number of 8-channel groups other than one, whose 16-channel steps straddle taps; slices too wide for
// two slots in shared memory, above 224-240 channels): the gathering kernel takes those.  Where both apply the slices
// are faster from the smallest volumes on (one voxel, 16 -> 16: 8 against 15 us).
constexpr size_t kSmemLimit = 227*1024, kSmemHalf = 113*1024;

bool planSlices(SliceParams& p, int sms, size_t& smem, dim3& grid) {
    if (p.cin != 8 && p.cin%16 != 0)
        return false;
    p.colsX = (p.W + kTileX - 1)/kTileX;
    p.colsY = (p.H + kTileY - 1)/kTileY;
    const long long columns = (long long) p.colsX*p.colsY*p.batch;
    if (columns*p.D > (1LL << 28) || (long long) p.H*p.W*p.cin >= (1LL << 31))
        return false;
    // The output channels and planes per item and the place of the weights, by an estimate of the time in cycles: the
    // rounds of items over the SMs times the slower of an item's MMAs and its copies, and the copies before the first
    // MMA.  An MMA of 16 channels takes the 52 cycles that were measured for N = 16, more as N grows (36 + N/4 wavefronts
    // of shared memory, N/2 of the tensor core); an SM copies about 40 bytes per cycle from L2; a streamed tile of weights
    // takes 1000 cycles to be handed over and 1 per 15 bytes.
    const double kCopy = 40.0, kStream = 15.0, kTile = 1000.0;
    const int steps = (p.cin + 15)/16;
    auto mma = [](int n) { return std::max(52.0, std::max(44.0 + n/4.0, 10.0 + n/2.0)); };
    double best = 0;
    bool found = false;
    for (int n = std::min(112, p.cout); n >= 16; n -= 16) {
        if (p.cout%n != 0)
            continue;
        for (int zLen = 8; zLen >= 1; zLen /= 2) {
            if (zLen > 1 && (zLen/2 >= p.D || (p.cin == 8 && p.D%zLen != 0)))
                continue;
            SliceParams t = p;
            t.nTile = n;
            t.nBlocks = p.cout/n;
            t.zLen = zLen;
            t.zBlocks = (p.D + zLen - 1)/zLen;
            const long long items = columns*t.zBlocks;
            const double rounds = items*t.nBlocks < 4LL*sms ? (double) ((items*t.nBlocks + sms - 1)/sms)
                                                            : (double) (items*t.nBlocks)/sms;
            const double slices = (zLen + 2)*(double) kSliceVoxels*p.cin*2, weights = (double) kTaps*p.cin*n*2;
            auto consider = [&](int slots, int wSlots, double work, double copies, double before) {
                if (sliceSmemBytes(p.cin, n, slots, wSlots) > kSmemLimit)
                    return false;
                const double cost = rounds*std::max(work, copies/kCopy) + before/kCopy;
                if (!found || cost < best) {
                    best = cost;
                    found = true;
                    t.slots = slots;
                    t.wSlots = wSlots;
                    // Accumulators: three in progress and one being read, more where they cost no CTA its place, so that
                    // their ring seldom wraps around between the planes of a slice.
                    const bool two = sliceSmemBytes(p.cin, n, slots, wSlots) <= kSmemHalf && n <= 64;
                    t.accSlots = p.cin == 8 || wSlots < kTaps ? (n < 32 ? kMaxAcc : 4) : std::min(kMaxAcc, (two ? 256 : 512)/n);
                    t.items = (int) items;
                    p = t;
                }
                return true;
            };
            const double slice = slices/(zLen + 2);
            if (p.cin == 8)
                // The slots of an item are consecutive (a pair of taps spans two slices): two items' worth of them.
                consider(2*(zLen + 2), kTaps, 14.0*zLen*mma(n), slices, weights + 3*slice);
            else {
                const int threes = std::max(0, zLen - 2);
                const double merged = 9.0*steps*(2*mma(n) + (zLen > 1 ? 2*mma(2*n) : mma(n)) + threes*mma(3*n));
                bool resident = false;
                for (int slots = 6; slots >= 3 && n <= 80 && !resident; slots--)
                    if (slots == 3 || sliceSmemBytes(p.cin, n, slots, kTaps) <= kSmemHalf)
                        resident = consider(slots, kTaps, merged, slices, weights + slice);
                const double streamed = zLen*(weights/kStream + kTaps*kTile);
                for (int tiles = 12; tiles >= 2; tiles--)
                    if ((zLen > 1 && consider(3, tiles, 27.0*steps*zLen*mma(n), slices + streamed*kCopy, slice)) ||
                        consider(2, tiles, 27.0*steps*zLen*mma(n), slices + streamed*kCopy, slice))
                        break;
            }
        }
    }
    if (!found)
        return false;
    // More slots where they cost no CTA its place.
    if (p.cin != 8 && p.wSlots == kTaps)
        while (p.slots < 6 && sliceSmemBytes(p.cin, p.nTile, p.slots + 1, kTaps) <= kSmemLimit &&
               (sliceSmemBytes(p.cin, p.nTile, p.slots, kTaps) > kSmemHalf ||
                sliceSmemBytes(p.cin, p.nTile, p.slots + 1, kTaps) <= kSmemHalf))
            p.slots++;
    smem = sliceSmemBytes(p.cin, p.nTile, p.slots, p.wSlots);
    // Several CTAs per SM where shared and tensor memory allow: one thread issues a CTA's MMAs and is slower than the
    // tensor core on narrow layers.
    int perSM = 1;
    while (perSM < 4 && (smem + 1024)*(perSM + 1) <= kSmemLimit + 1024 && tmemColumns(p.accSlots*p.nTile)*(perSM + 1) <= 512)
        perSM++;
    grid = dim3((unsigned) std::max(1, std::min(p.items, perSM*sms/p.nBlocks)), (unsigned) p.nBlocks);
    return true;
}

// The division of a weight gradient; returns the shared memory of a CTA.
size_t planGradient(GradParams& p, int sms, dim3& grid) {
    // At most 15 of an M tile's 16 groups are used (three rows of up to 5 channel groups).
    const int groups = p.cin/8;
    p.chunks = (groups + 4)/5;
    p.groupsX = (groups + p.chunks - 1)/p.chunks;
    p.chunks = (groups + p.groupsX - 1)/p.groupsX;
    // All dz of up to 48 output channels in one CTA (432 columns of tensor memory), else one dz of up to 80 (N <= 240).
    auto divisor = [&](int most) {
        int n = std::min(most, p.cout);
        while (p.cout%n != 0)
            n -= 16;
        return n;
    };
    p.dzCount = p.cout <= 48 ? 3 : 1;
    p.coTile = divisor(p.dzCount == 3 ? 48 : 80);
    p.coBlocks = p.cout/p.coTile;
    // MMAs per sum: an error of about 1e-6 on large volumes; small ones, whose sums are short anyway, keep theirs at 1e-7
    // (that takes items of a plane instead of four there: 16 -> 16 at 35 x 40 x 21 16.6 us with sums of 8, 11.7 with 32; at
    // 16 x 8 x 4 9.3 and 11.4).
    const long long runs = ((long long) p.W*p.H*p.D*p.batch + 15)/16, parts = ((p.cout + 127)/128)*(((long long) 27*p.cin + 255)/256);
    p.chain = (int) std::max(8LL, std::min(p.dzCount == 3 ? 32LL : 48LL, runs/(4*sms/parts + 1)));
    // Planes per item: as many as keep a buffer of dy within 75 KB (a slice of x is read by up to three planes) and an
    // item's MMAs within a sum.
    p.zLen = p.dzCount == 3 ? std::max(1, std::min({4, 76800/gradDyBytes(p.coTile, 1), p.chain/kRowsY})) : 1;
    p.colsX = (p.W + kRunX - 1)/kRunX;
    p.colsY = (p.H + kRowsY - 1)/kRowsY;
    p.zBlocks = (p.D + p.zLen - 1)/p.zLen;
    p.items = (int) ((long long) p.colsX*p.colsY*p.zBlocks*p.batch);
    const size_t smem = gradSmemBytes(p.groupsX, p.coTile, p.zLen);
    const int blocks = p.chunks*p.coBlocks*(p.dzCount == 3 ? 1 : 3);
    grid = dim3((unsigned) std::max(1, std::min(p.items, sms/blocks)), (unsigned) blocks);
    return smem;
}

LbmStatus launchError(cudaError_t e) {
    lbm::setLastError(std::string("conv3d: ") + cudaGetErrorString(e));
    return LBM_ERR_CUDA;
}

LbmStatus invalid(const char* message) {
    lbm::setLastError(message);
    return LBM_ERR_INVALID_ARGUMENT;
}

} // namespace

extern "C" {

LbmStatus lbm_conv3d_forward(const void* x, const void* w, const float* bias, void* y, int batch, int depth, int height,
                             int width, int cin, int cout, int relu, void* stream) {
    if (!x || !w || !y || batch <= 0 || depth <= 0 || height <= 0 || width <= 0)
        return invalid("lbm_conv3d_forward: null pointer or empty volume");
    if (cin <= 0 || cin%8 != 0 || cout < 16 || cout > 256 || cout%16 != 0)
        return invalid("lbm_conv3d_forward: cin must be a multiple of 8 and cout a multiple of 16 up to 256");
    long long voxels = (long long) batch*depth*height*width;
    SliceParams p;
    p.x = (const __nv_bfloat16*) x;
    p.w = (const __nv_bfloat16*) w;
    p.bias = bias;
    p.y = (__nv_bfloat16*) y;
    p.batch = batch; p.D = depth; p.H = height; p.W = width; p.cin = cin; p.cout = cout; p.relu = relu;
    int device = 0, sms = 148;
    dim3 grid;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    size_t smem = 0;
    cudaError_t e;
    if (planSlices(p, sms, smem, grid)) {
        const int mode = cin == 8 ? kSingleGroup : (p.wSlots == kTaps ? kResident : kStreamed);
        auto kernel = mode == kSingleGroup ? convSliceKernel<kSingleGroup>
                    : mode == kResident ? convSliceKernel<kResident> : convSliceKernel<kStreamed>;
        const int threads = mode == kStreamed ? sliceThreads<kStreamed> : sliceThreads<kResident>;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kSmemLimit);
        if (e != cudaSuccess)
            return launchError(e);
        kernel<<<grid, threads, smem, (cudaStream_t) stream>>>(p);
        e = cudaGetLastError();
        return e == cudaSuccess ? LBM_OK : launchError(e);
    }
    smem = stageBytes(cout);
    e = cudaFuncSetAttribute(convForwardKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
    if (e != cudaSuccess)
        return launchError(e);
    convForwardKernel<<<(unsigned) ((voxels + kTileM - 1)/kTileM), kThreads, smem, (cudaStream_t) stream>>>(
        (const __nv_bfloat16*) x, (const __nv_bfloat16*) w, bias, (__nv_bfloat16*) y, batch, depth, height, width, cin,
        cout, relu);
    e = cudaGetLastError();
    return e == cudaSuccess ? LBM_OK : launchError(e);
}

LbmStatus lbm_conv3d_weight_grad(const void* x, const void* dy, float* dw, int batch, int depth, int height, int width,
                                 int cin, int cout, void* stream) {
    if (!x || !dy || !dw || batch <= 0 || depth <= 0 || height <= 0 || width <= 0)
        return invalid("lbm_conv3d_weight_grad: null pointer or empty volume");
    if (cin <= 0 || cin%8 != 0 || cout < 16 || cout > 256 || cout%16 != 0)
        return invalid("lbm_conv3d_weight_grad: cin must be a multiple of 8 and cout a multiple of 16 up to 256");
    GradParams p;
    p.x = (const __nv_bfloat16*) x;
    p.dy = (const __nv_bfloat16*) dy;
    p.dw = dw;
    p.batch = batch; p.D = depth; p.H = height; p.W = width; p.cin = cin; p.cout = cout;
    int device = 0, sms = 148;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    dim3 grid;
    const size_t smem = planGradient(p, sms, grid);
    cudaError_t e = cudaFuncSetAttribute(convSliceGradKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kSmemLimit);
    if (e != cudaSuccess)
        return launchError(e);
    convSliceGradKernel<<<grid, kGradThreads, smem, (cudaStream_t) stream>>>(p);
    e = cudaGetLastError();
    return e == cudaSuccess ? LBM_OK : launchError(e);
}

LbmStatus lbm_conv3d_status(void* stream) {
    cudaError_t e = cudaStreamSynchronize((cudaStream_t) stream);
    if (e != cudaSuccess)
        return launchError(e);
    int status = 0;
    e = cudaMemcpyFromSymbol(&status, convStatus, sizeof(int));
    if (e != cudaSuccess)
        return launchError(e);
    int zero = 0;
    cudaMemcpyToSymbol(convStatus, &zero, sizeof(int));
    if (status != 0) {
        lbm::setLastError("conv3d: a wait for the tensor cores timed out");
        return (LbmStatus) status;
    }
    return LBM_OK;
}

LbmStatus lbm_conv3d_set_wait_limit(long long polls) {
    long long value = polls >= 0 ? polls : kSpinLimit;
    cudaError_t e = cudaMemcpyToSymbol(convWaitPolls, &value, sizeof(long long));
    return e == cudaSuccess ? LBM_OK : launchError(e);
}

} // extern "C"
