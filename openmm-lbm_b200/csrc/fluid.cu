// Fluid kernels of the B200 LBM force kernel (sm_100a).
//
//  streamCollideKernel   the dense, fused step: pull streaming, moments, momentum removal, regularized
//                        collision with Guo forcing (+ particle reaction, + Philox fluctuations), store;
//                        HBM-bound, 2*19 population transfers per fluid node.  Restates, fused, the
//                        reference's computeMoments, removeFluidMomentum and collideAndStream
//                        (platforms/reference/src/ReferenceLBMKernels.cpp:430-501, 1066-1120).
//  bounceBackKernel      halfway bounce-back and wall momentum exchange over the wall links
//                        (ReferenceLBMKernels.cpp:1156-1205), writing into the slots of solid nodes.
//  boundaryKernel        regularized walls and open faces (ReferenceLBMKernels.cpp:1207-1343), writing
//                        into the slots that the boundary node pulls.
//  finishStep, finishKernel   deterministic reduction of the per-block partial sums of a step.
//  momentsKernel         mass, momentum and largest speed of the current state (Mach check, start-up).
//  gather/scatter        conversion between the pull layout and the reference's state layout.
#include "fluid.cuh"
#include "collide.cuh"
#include "collide_pair.cuh"
#include "lbm_device.cuh"
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>
#include <utility>

namespace lbm {

#define CUDA_CHECK(call) do { cudaError_t e_ = (call); if (e_ != cudaSuccess) \
    throw Error(LBM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); } while (0)

namespace {

constexpr int TX = 32, TY = 8, THREADS = TX*TY;
constexpr int NPART = 8;           // doubles per partial record: mass, momentum[3], wall[3], maxSpeed2

// Block reduction of a partial record (sums, and max for the last entry) into partials[slot], deterministic.
__device__ void blockReduceStore(double v[NPART], double* out) {
    __shared__ double red[THREADS/32][NPART];
    int lane = threadIdx.x%32, warp = threadIdx.x/32, warps = blockDim.x/32;
#pragma unroll
    for (int i = 0; i < NPART; i++)
        for (int offset = 16; offset > 0; offset >>= 1) {
            double o = __shfl_down_sync(0xffffffffu, v[i], offset);
            v[i] = (i == NPART-1 ? fmax(v[i], o) : v[i] + o);
        }
    if (lane == 0)
        for (int i = 0; i < NPART; i++)
            red[warp][i] = v[i];
    __syncthreads();
    if (threadIdx.x < NPART) {
        int i = threadIdx.x;
        double s = red[0][i];
        for (int w = 1; w < warps; w++)
            s = (i == NPART-1 ? fmax(s, red[w][i]) : s + red[w][i]);
        out[i] = s;
    }
}

// The sums of `count` partial records in a fixed order, and the statistics from them.  mode 0: the sums of a step (mass,
// momentum, ucm, wall); 1: a moments pass that sets the sums and the largest speed; 2: a moments pass for the largest
// speed only (the sums of the step are kept).  COHERENT: the records were written by other blocks of the launch and are
// read through L2.
template <bool COHERENT>
__device__ __forceinline__ void sumRecords(const double* partials, int count, const FluidView& v, int mode) {
    double acc[NPART] = {0, 0, 0, 0, 0, 0, 0, 0};
    // Several records in flight per thread (the loads do not wait on the sums).
#pragma unroll 4
    for (int i = threadIdx.x; i < count; i += blockDim.x)
#pragma unroll
        for (int k = 0; k < NPART; k++) {
            const double* p = partials + NPART*(long long) i + k;
            const double value = COHERENT ? __ldcg(p) : *p;
            acc[k] = (k == NPART-1 ? fmax(acc[k], value) : acc[k] + value);
        }
    __shared__ double total[NPART];
    blockReduceStore(acc, total);
    __syncthreads();
    if (threadIdx.x == 0) {
        StepStats* s = v.stats;
        if (mode != 2) {
            s->mass = total[0];
            double mass = v.numFluid + total[0];
            for (int a = 0; a < 3; a++) {
                s->momentum[a] = total[1+a];
                s->ucm[a] = total[1+a]/mass;
            }
        }
        if (mode == 0)
            for (int a = 0; a < 3; a++)
                s->wall[a] = total[4+a];
        if (mode != 0)
            s->maxSpeed2 = total[7];
    }
}

// Ends a step whose only pass is the dense kernel: every block has stored its record and takes a ticket; the block with
// the last one adds all records, in the order of the records and not of the blocks' arrival, and resets the ticket.  On
// the device this costs what a launch for the sums costs (a 32^3 step 6.6 us against 3.9 + 2.5), but not the launch: 12.9
// -> 10.6 us per step as the host sees it.  After the sparse passes it would be slower (obstacle channel, 128 x 64 x 64:
// 23 us for one sparse pass and the sums against 18.7 for bounce-back, faces and sums apart; each of their many small
// blocks waits for its stores and its ticket), so there the sums have a launch of their own.
__device__ __forceinline__ void finishStep(const FluidView& v) {
    __shared__ unsigned ticket;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        ticket = atomicAdd(v.ticket, 1u);
    }
    __syncthreads();
    if (ticket != gridDim.x - 1)
        return;
    __threadfence();
    sumRecords<true>(v.partials, (int) gridDim.x, v, 0);
    if (threadIdx.x == 0)
        *v.ticket = 0;
}

// The kernels of a step follow one another as programmatic dependents: a kernel's blocks come onto the SMs while the one
// before it still runs and wait here until that has finished and its stores are visible; then the next kernel may do the
// same.  What a launch costs between two kernels, about 2.5 us, is hidden that way: a 32^3 step 10.0 -> 8.5 us, the
// obstacle channel's four kernels on 128 x 64 x 64 nodes 42 -> 34 us, a ragged 150 x 93 x 67 channel 41 -> 36 us.
// The wait hands `p` on, so that no load through it, read-only ones included, can be moved before the wait.
template <typename P>
__device__ __forceinline__ P* afterPrevious(P* p) {
    asm volatile("griddepcontrol.wait;" : "+l"(p) : : "memory");
    asm volatile("griddepcontrol.launch_dependents;" : : : "memory");
    return p;
}

struct Coords {
    int x, y, z;
};

__device__ __forceinline__ Coords nodeCoords(long long node, int nx, int ny) {
    Coords c;
    c.x = (int) (node%nx);
    long long r = node/nx;
    c.y = (int) (r%ny);
    c.z = (int) (r/ny);
    return c;
}

__device__ __forceinline__ int wrap(int i, int n) {
    return (i < 0 ? i + n : (i >= n ? i - n : i));
}

// Index of node (x + dx, y + dy, z + dz), periodic.
__device__ __forceinline__ long long shifted(const FluidView& v, int x, int y, int z, int dx, int dy, int dz) {
    return wrap(x + dx, v.nx) + (long long) v.nx*(wrap(y + dy, v.ny) + (long long) v.ny*wrap(z + dz, v.nz));
}

__device__ __forceinline__ int cxr(int q) { return cxOf(q); }
__device__ __forceinline__ int cyr(int q) { return cyOf(q); }
__device__ __forceinline__ int czr(int q) { return czOf(q); }

template <typename R>
__device__ __forceinline__ R weightOf(int q) {
    return (q == 0 ? R(1.0/3.0) : (q <= 6 ? R(1.0/18.0) : R(1.0/36.0)));
}

// ---------------------------------------------------------------------------------------------------
// The dense step.
// ---------------------------------------------------------------------------------------------------

// Resident blocks of 256 threads per SM that the register allocation of the dense kernel must allow: 3 for float
// arithmetic (85 registers, 24 warps per SM) and 2 for double.  Measured on B200 at 256^3 (FP32, plain): 0.479 ms
// per launch with 3 blocks, 0.549 ms with 4 (64 registers: the loads of a node are no longer all in flight).
#ifdef LBM_DENSE_MIN_BLOCKS
template <typename R> constexpr int denseMinBlocks() { return LBM_DENSE_MIN_BLOCKS; }
#else
template <typename R> constexpr int denseMinBlocks() { return sizeof(R) == 4 ? 3 : 2; }
#endif

// The dense step over 32 x 8 node tiles (lane = x, warp = y), persistent blocks striding over the tiles.  Node
// indices are 32-bit (the host limits the lattice to 2^32 nodes); the tile coordinates advance by the grid
// stride without divisions.  Solid nodes are skipped by their bit in the solid mask; nodes with a particle
// reaction add it to the body force.
template <typename T, typename R, bool SOLID, bool REACT, bool FLUCT, bool FINISH>
__global__ void __launch_bounds__(THREADS, denseMinBlocks<R>())
streamCollideKernel(const T* __restrict__ input, T* __restrict__ B, FluidView v, int remove, long long step) {
    const T* __restrict__ A = afterPrevious(input);
    if constexpr (REACT)
        asm volatile("" : "+l"(v.reactMask));
    const int lane = threadIdx.x%32, warp = threadIdx.x/32;
    const unsigned N = (unsigned) v.n;
    const int nx = v.nx, ny = v.ny, nz = v.nz;
    const CollideConstants<R> k = collideConstants<R>(v.omega, v.g, v.stats->ucm, remove, v.mu, v.seed);
    R sumMass = 0, sumX = 0, sumY = 0, sumZ = 0;
    const unsigned numTiles = (unsigned) v.numTiles, stride = gridDim.x;
    const int tilesX = v.tilesX, tilesY = v.tilesY;
    int tx = (int) (blockIdx.x%tilesX), ty = (int) ((blockIdx.x/tilesX)%tilesY), tz = (int) (blockIdx.x/tilesX/tilesY);
    const int dtx = (int) (stride%tilesX), dty = (int) ((stride/tilesX)%tilesY), dtz = (int) (stride/tilesX/tilesY);
    for (unsigned t = blockIdx.x; t < numTiles; t += stride) {
        const int x = tx*TX + lane, y = ty*TY + warp, z = tz, tileX = tx;
        tx += dtx;
        int carry = tx >= tilesX;
        tx -= carry ? tilesX : 0;
        ty += dty + carry;
        carry = ty >= tilesY;
        ty -= carry ? tilesY : 0;
        tz += dtz + carry;
        if (x >= nx || y >= ny)
            continue;
        const unsigned row = (unsigned) z*ny + y;
        if (SOLID) {
            uint32_t word = __ldg(&v.solidMask[(size_t) row*v.wordsPerRow + tileX]);
            if ((word >> lane) & 1u)
                continue;
        }
        const unsigned node = row*nx + x;
        R ex = 0, ey = 0, ez = 0;
        if (REACT) {
            uint32_t word = __ldg(&v.reactMask[(size_t) row*v.wordsPerRow + tileX]);
            if ((word >> lane) & 1u) {
                const R* rp = reinterpret_cast<const R*>(v.reaction) + 4*(size_t) node;
                ex = rp[0];
                ey = rp[1];
                ez = rp[2];
            }
        }
        collideNode<T, R, FLUCT>(A, B, N, node, x, y, z, nx, ny, nz, k, ex, ey, ez, step, sumMass, sumX, sumY, sumZ);
    }
    double acc[NPART] = {(double) sumMass, (double) sumX, (double) sumY, (double) sumZ, 0, 0, 0, 0};
    blockReduceStore(acc, v.partials + NPART*(long long) blockIdx.x);
    if (FINISH)
        finishStep(v);
}


// The dense step with two x-adjacent nodes per thread (nx even), the arithmetic of both in packed FP32 pairs; each
// thread loads its pulled words from global memory.  FLAT: the pairs in the order of their nodes; otherwise row tiles of
// PAIR_TX x TY nodes (the launcher says where).
template <typename T, bool SOLID, bool REACT, bool FLUCT, bool FINISH, bool FLAT>
__global__ void __launch_bounds__(THREADS, (sizeof(T) == 2 && !FLUCT) ? LBM_PAIR_MIN_BLOCKS_16BIT : LBM_PAIR_MIN_BLOCKS)
streamCollidePairKernel(const T* __restrict__ input, T* __restrict__ B, FluidView v, int remove, long long step) {
    const T* __restrict__ A = afterPrevious(input);
    if constexpr (REACT)
        asm volatile("" : "+l"(v.reactMask));
    typedef typename PairIO<T>::Word Word;
    const int lane = threadIdx.x%32, warp = threadIdx.x/32;
    const unsigned N = (unsigned) v.n;
    const int nx = v.nx, ny = v.ny, nz = v.nz;
    const Word* __restrict__ aw = reinterpret_cast<const Word*>(A);
    Word* __restrict__ bw = reinterpret_cast<Word*>(B);
    const unsigned halfN = N/2;                       // words per direction plane (N is even)
    const PairConstants c = pairConstants(v, remove, step);
    float sums[4] = {0, 0, 0, 0};
    const int tilesX = (nx + PAIR_TX - 1)/PAIR_TX, tilesY = v.tilesY;
    const unsigned numTiles = FLAT ? (halfN + THREADS - 1)/THREADS : (unsigned) tilesX*tilesY*nz, stride = gridDim.x;
    for (unsigned t = blockIdx.x; t < numTiles; t += stride) {
        int x0, y, z;
        if constexpr (FLAT) {
            // The pairs in the order of their nodes: a warp runs on across the ends of rows.
            const unsigned pair = t*THREADS + threadIdx.x, perRow = (unsigned) nx/2, flatRow = pair/perRow;
            if (pair >= halfN)
                continue;
            x0 = 2*(int) (pair - flatRow*perRow);
            z = (int) (flatRow/(unsigned) ny);
            y = (int) (flatRow - (unsigned) z*ny);
        }
        else {
            const int tx = (int) (t%tilesX);
            const unsigned rr = t/tilesX;
            y = (int) (rr%tilesY)*TY + warp;
            z = (int) (rr/tilesY);
            x0 = tx*PAIR_TX + 2*lane;
            if (x0 >= nx || y >= ny)
                continue;
        }
        const unsigned row = (unsigned) z*ny + y;
        bool solidA = false, solidB = false;
        if (SOLID) {
            uint32_t word = __ldg(&v.solidMask[(size_t) row*v.wordsPerRow + (x0 >> 5)]);
            solidA = (word >> (x0 & 31)) & 1u;
            solidB = (word >> ((x0 + 1) & 31)) & 1u;
            if (solidA && solidB)
                continue;
        }
        const unsigned node = row*nx + x0;
        // Rows of the pull sources: index [1 - cy][1 - cz] (periodic in y and z).
        const int ys[3] = {y == 0 ? ny - 1 : y - 1, y, y == ny - 1 ? 0 : y + 1};
        const int zs[3] = {z == 0 ? nz - 1 : z - 1, z, z == nz - 1 ? 0 : z + 1};
        const int xl = x0 == 0 ? nx - 2 : x0 - 2, xr = x0 + 2 == nx ? 0 : x0 + 2;
        F2 r[19];
        staticFor<19>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            constexpr int cx = cxOf(q), cy = cyOf(q), cz = czOf(q);
            const unsigned base = ((unsigned) zs[1-cz]*ny + ys[1-cy])*nx;
            const Word* plane = aw + (size_t) q*halfN;
            Word w;
            if (cx == 0)
                w = __ldg(plane + (base + x0)/2);
            else if (cx == 1)
                w = PairIO<T>::left(__ldg(plane + (base + xl)/2), __ldg(plane + (base + x0)/2));
            else
                w = PairIO<T>::right(__ldg(plane + (base + x0)/2), __ldg(plane + (base + xr)/2));
            r[q] = PairIO<T>::decode(w);
        });
        bool reactA = false, reactB = false;
        if (REACT) {
            uint32_t word = __ldg(&v.reactMask[(size_t) row*v.wordsPerRow + (x0 >> 5)]);
            reactA = (word >> (x0 & 31)) & 1u;
            reactB = (word >> ((x0 + 1) & 31)) & 1u;
        }
        PairStore<T, SOLID> out{bw + node/2, halfN, solidA, solidB};
        collidePair<T, SOLID, REACT, FLUCT>(r, v, c, remove, step, node, solidA, solidB, reactA, reactB, out, sums);
    }
    double acc[NPART] = {(double) sums[0], (double) sums[1], (double) sums[2], (double) sums[3], 0, 0, 0, 0};
    blockReduceStore(acc, v.partials + NPART*(long long) blockIdx.x);
    if (FINISH)
        finishStep(v);
}

// The dense step for 16-bit storage without fluctuations, four x-adjacent nodes per thread (nx a multiple of 4):
// each direction's four sources are one aligned 64-bit word of the source row, with c_x = +1 the high half of the
// 32-bit word to the left in front of its first three, with c_x = -1 the low half of the word to the right after its
// last three; the four post-collision values of a direction go out as one 64-bit word.  The nodes are collided as two
// pairs (collidePulled, the same arithmetic and dither bits as the paired kernel, so the results are the paired
// kernel's bit for bit); the first pair's packed words wait in registers for the second's.  A warp takes a row tile
// of QUAD_TX nodes.  Against the paired kernel this halves the loads, stores and address arithmetic per node (29 loads
// and 19 stores per 4 nodes) and doubles the bytes in flight per warp: FP16 channel step 0.578 -> 0.511 ms, BF16
// 0.571 -> 0.503 ms.  Measured slower: 4 or 6 blocks per SM (0.527 / 0.548 ms FP16), the first pair's words held in
// shared memory (0.592 ms at 6 blocks), and each pair storing its own 32-bit words (0.599 ms).
constexpr int QUAD_TX = 128;        // nodes per warp row tile: 4 per lane
#ifndef LBM_QUAD_THREADS
#define LBM_QUAD_THREADS 128
#endif
#ifndef LBM_QUAD_MIN_BLOCKS
#define LBM_QUAD_MIN_BLOCKS 5
#endif

// The first pair of a quad: its packed words, held until the second pair's are ready.
template <typename T>
struct QuadHold {
    uint32_t word[19];
    template <int q> __device__ __forceinline__ void put(F2 value, uint32_t dither) {
        word[q] = PairIO<T>::pack(value.v.x, value.v.y, dither);
    }
};

// The second pair: stores both pairs' words of direction q as one 64-bit word (word halves per node when a node of
// the quad is solid).
template <typename T, bool SOLID>
struct QuadStore {
    uint2* out;                   // the quad's word in plane 0
    unsigned quarterN;            // 64-bit words per plane
    const QuadHold<T>& first;
    uint32_t solidBits;           // bit i: node x0 + i is solid
    template <int q> __device__ __forceinline__ void put(F2 value, uint32_t dither) {
        const uint32_t second = PairIO<T>::pack(value.v.x, value.v.y, dither);
        uint2* p = out + (size_t) q*quarterN;
        if (SOLID && solidBits != 0) {
            uint32_t* w = reinterpret_cast<uint32_t*>(p);
            storeWord16<SOLID>(w, first.word[q], solidBits & 1u, solidBits & 2u);
            storeWord16<SOLID>(w + 1, second, solidBits & 4u, solidBits & 8u);
            return;
        }
        *p = make_uint2(first.word[q], second);
    }
};

template <typename T, bool SOLID, bool REACT, bool FINISH, bool FLAT>
__global__ void __launch_bounds__(LBM_QUAD_THREADS, LBM_QUAD_MIN_BLOCKS)
streamCollideQuadKernel(const T* __restrict__ input, T* __restrict__ B, FluidView v, int remove, long long step) {
    const T* __restrict__ A = afterPrevious(input);
    if constexpr (REACT)
        asm volatile("" : "+l"(v.reactMask));
    static_assert(sizeof(T) == 2, "the quad kernel is for 16-bit storage");
    const unsigned N = (unsigned) v.n;
    const int nx = v.nx, ny = v.ny, nz = v.nz;
    const uint32_t* __restrict__ a32 = reinterpret_cast<const uint32_t*>(A);
    const uint2* __restrict__ a64 = reinterpret_cast<const uint2*>(A);
    uint2* __restrict__ b64 = reinterpret_cast<uint2*>(B);
    const unsigned halfN = N/2, quarterN = N/4;     // 32-bit and 64-bit words per direction plane (N % 4 == 0)
    const PairConstants c = pairConstants(v, remove, step);
    float sums[4] = {0, 0, 0, 0};
    const int lane = threadIdx.x%32, tilesX = (nx + QUAD_TX - 1)/QUAD_TX;
    const unsigned numTiles = FLAT ? (quarterN + 31)/32 : (unsigned) tilesX*ny*nz, warps = blockDim.x/32;
    for (unsigned t = blockIdx.x*warps + threadIdx.x/32; t < numTiles; t += gridDim.x*warps) {
        unsigned row;
        int x0;
        if constexpr (FLAT) {
            const unsigned quad = t*32 + lane, perRow = (unsigned) nx/4;
            if (quad >= quarterN)
                continue;
            row = quad/perRow;
            x0 = 4*(int) (quad - row*perRow);
        }
        else {
            row = t/tilesX;
            x0 = (int) (t%tilesX)*QUAD_TX + 4*lane;
            if (x0 >= nx)
                continue;
        }
        const int y = (int) (row%(unsigned) ny), z = (int) (row/(unsigned) ny);
        uint32_t solidBits = 0;
        if (SOLID) {
            // x0 % 4 == 0: the quad's four bits sit in one mask word.
            solidBits = (__ldg(&v.solidMask[(size_t) row*v.wordsPerRow + (x0 >> 5)]) >> (x0 & 31)) & 0xFu;
            if (solidBits == 0xFu)
                continue;
        }
        const unsigned node = row*nx + x0;
        const int ys[3] = {y == 0 ? ny - 1 : y - 1, y, y == ny - 1 ? 0 : y + 1};
        const int zs[3] = {z == 0 ? nz - 1 : z - 1, z, z == nz - 1 ? 0 : z + 1};
        const int xl = x0 == 0 ? nx - 2 : x0 - 2, xr = x0 + 4 == nx ? 0 : x0 + 4;
        uint32_t wa[19], wb[19];
        staticFor<19>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            constexpr int cx = cxOf(q), cy = cyOf(q), cz = czOf(q);
            const unsigned base = ((unsigned) zs[1-cz]*ny + ys[1-cy])*nx;
            const uint2 w = __ldg(a64 + (size_t) q*quarterN + (base + x0)/4);
            if (cx == 0) {
                wa[q] = w.x;
                wb[q] = w.y;
            }
            else if (cx == 1) {
                wa[q] = __byte_perm(__ldg(a32 + (size_t) q*halfN + (base + xl)/2), w.x, 0x5432);
                wb[q] = __byte_perm(w.x, w.y, 0x5432);
            }
            else {
                wa[q] = __byte_perm(w.x, w.y, 0x5432);
                wb[q] = __byte_perm(w.y, __ldg(a32 + (size_t) q*halfN + (base + xr)/2), 0x5432);
            }
        });
        uint32_t reactBits = 0;
        if (REACT)
            reactBits = (__ldg(&v.reactMask[(size_t) row*v.wordsPerRow + (x0 >> 5)]) >> (x0 & 31)) & 0xFu;
        QuadHold<T> first;
        collidePulled<T, SOLID, REACT, false>(PulledWords<T>{wa}, v, c, remove, step, node, solidBits & 1u,
                                              solidBits & 2u, reactBits & 1u, reactBits & 2u, first, sums);
        QuadStore<T, SOLID> out{b64 + node/4, quarterN, first, solidBits};
        collidePulled<T, SOLID, REACT, false>(PulledWords<T>{wb}, v, c, remove, step, node + 2, solidBits & 4u,
                                              solidBits & 8u, reactBits & 4u, reactBits & 8u, out, sums);
    }
    double acc[NPART] = {(double) sums[0], (double) sums[1], (double) sums[2], (double) sums[3], 0, 0, 0, 0};
    blockReduceStore(acc, v.partials + NPART*(long long) blockIdx.x);
    if (FINISH)
        finishStep(v);
}

// ---------------------------------------------------------------------------------------------------
// Bounce-back over the wall links (after the dense step, on the output array).
// ---------------------------------------------------------------------------------------------------

// One wall node per thread (a grid of up to kGridWall blocks covers the channel's wall planes in one pass): the
// node's wall links are known at compile time per direction, so the loads of all its links are issued before any of
// the stores (a store may alias a later load as far as the compiler knows) and do not wait on one another.
template <typename T, typename R>
__global__ void __launch_bounds__(THREADS)
bounceBackKernel(T* __restrict__ output, const int* __restrict__ wall, int numWall, FluidView v, double* partials) {
    T* __restrict__ B = afterPrevious(output);
    double acc[NPART] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int b = blockIdx.x*blockDim.x + threadIdx.x; b < numWall; b += gridDim.x*blockDim.x) {
        const int2 entry = __ldg(reinterpret_cast<const int2*>(wall) + b);
        const long long node = (unsigned) entry.x;
        const int links = entry.y;
        const Coords c = nodeCoords(node, v.nx, v.ny);
        T raw[19];
        staticFor<18>([&](auto qc) {
            constexpr int q = decltype(qc)::value + 1;
            if (links & (1 << q))
                raw[q] = B[(long long) q*v.n + node];
        });
        staticFor<18>([&](auto qc) {
            constexpr int q = decltype(qc)::value + 1;
            if (links & (1 << q)) {
                // The population x built for q streamed into the solid node s = x + c_q; x takes it back along
                // -c_q, so it goes into the slot of s that x pulls for opp(q).  Opposite directions have the same
                // weight, so the stored element is copied as it is.
                const long long s = shifted(v, c.x, c.y, c.z, cxOf(q), cyOf(q), czOf(q));
                B[(long long) oppOf(q)*v.n + s] = raw[q];
                const double value = (double) loadq<T, R>(&raw[q], q);
                const double w = weightOf<double>(q);
                // The fluid momentum of the population is reversed; the wall receives 2 c_q (f + w)
                // (ReferenceLBMKernels.cpp:1176-1205, momentum exchange of Ladd 1994).
                acc[1] -= 2.0*cxOf(q)*value;
                acc[2] -= 2.0*cyOf(q)*value;
                acc[3] -= 2.0*czOf(q)*value;
                acc[4] += 2.0*cxOf(q)*(value + w);
                acc[5] += 2.0*cyOf(q)*(value + w);
                acc[6] += 2.0*czOf(q)*(value + w);
            }
        });
    }
    blockReduceStore(acc, partials + NPART*(long long) blockIdx.x);
}

// ---------------------------------------------------------------------------------------------------
// Regularized walls and open faces (applyBoundaries, ReferenceLBMKernels.cpp:1207-1343), on the boundary
// node list, after the dense step: A is the input of the step (its moments are recomputed from it) and B
// its output.
// ---------------------------------------------------------------------------------------------------

// Equilibrium deviation, Guo term and regularized non-equilibrium part of direction q.
template <typename R, int q>
__device__ __forceinline__ R along(R x, R y, R z) {
    return R(cxOf(q))*x + R(cyOf(q))*y + R(czOf(q))*z;
}

template <typename R, int q>
__device__ __forceinline__ R eqDeviation(R drho, R ux, R uy, R uz) {
    R rho = R(1) + drho;
    R uu = ux*ux + uy*uy + uz*uz;
    R cu = along<R, q>(ux, uy, uz);
    return wOf<R>(q)*(drho + rho*(R(3)*cu + R(4.5)*cu*cu - R(1.5)*uu));
}

template <typename R, int q>
__device__ __forceinline__ R guoAt(R ux, R uy, R uz, R fx, R fy, R fz) {
    R uf = ux*fx + uy*fy + uz*fz;
    R cu = along<R, q>(ux, uy, uz);
    R cf = along<R, q>(fx, fy, fz);
    return wOf<R>(q)*(R(3)*(cf - uf) + R(9)*cu*cf);
}

template <typename R, int q>
__device__ __forceinline__ R fneqAt(const Moments<R>& m) {
    constexpr int cx = cxOf(q), cy = cyOf(q), cz = czOf(q);
    R h0 = R(cx*cx) - R(1.0/3.0), h1 = R(cy*cy) - R(1.0/3.0), h2 = R(cz*cz) - R(1.0/3.0);
    return R(4.5)*wOf<R>(q)*(h0*m.pxx + h1*m.pyy + h2*m.pzz + R(2)*(R(cx*cy)*m.pxy + R(cx*cz)*m.pxz + R(cy*cz)*m.pyz));
}

// A boundary node per thread in blocks of 64: the lists are short (a few thousand nodes per face or wall plane), so the
// time is the latency of one node's work.  Directions are known at compile time (coefficients of 0 and +-1 vanish, the
// moments, modes and neighbours stay in registers), the 19 pulls are issued at once, then everything the node reads
// from the step's output.  Measured: 37.8 -> 9.9 us per step on the inlet and outlet of a 128 x 64 x 64 duct
// (FP32), 210 -> 31 us on the 23,000 nodes of a 95 x 64 x 61 duct of regularized walls with fluctuations
// (FP64), with runtime directions before (arrays in local memory, 15 modes per direction, one load after another).
constexpr int kBoundaryThreads = 64;

template <typename T, typename R, bool FLUCT>
__global__ void __launch_bounds__(kBoundaryThreads)
boundaryKernel(const T* __restrict__ input, T* __restrict__ B, const int* __restrict__ bnd, int numBoundary, FluidView v,
               int remove, long long step, double* partials, const double* faceData) {
    const T* __restrict__ A = afterPrevious(input);
    // faceData: per face (6): velocity[3], density, then boundary stress weight c, and the flags.
    double acc[NPART] = {0, 0, 0, 0, 0, 0, 0, 0};
    const long long N = v.n;
    const int nx = v.nx, ny = v.ny, nz = v.nz;
    const R omega = R(v.omega);
    const R gx = R(v.g[0]), gy = R(v.g[1]), gz = R(v.g[2]);
    for (int b = blockIdx.x*blockDim.x + threadIdx.x; b < numBoundary; b += gridDim.x*blockDim.x) {
        const int4 entry = __ldg(reinterpret_cast<const int4*>(bnd) + b);
        const long long node = (unsigned) entry.x;
        const int unknown = entry.y, solid = entry.z;
        const int kind = entry.w & 255, face = (entry.w >> 8) - 1;
        const Coords c = nodeCoords(node, nx, ny);
        // x - c_q and x + c_q, periodic: index 1 - c along each axis.
        const int xs[3] = {c.x == 0 ? nx - 1 : c.x - 1, c.x, c.x == nx - 1 ? 0 : c.x + 1};
        const int ys[3] = {c.y == 0 ? ny - 1 : c.y - 1, c.y, c.y == ny - 1 ? 0 : c.y + 1};
        const int zs[3] = {c.z == 0 ? nz - 1 : c.z - 1, c.z, c.z == nz - 1 ? 0 : c.z + 1};
        auto source = [&](auto qc) -> long long {
            constexpr int q = decltype(qc)::value;
            return xs[1-cxOf(q)] + (long long) nx*(ys[1-cyOf(q)] + (long long) ny*zs[1-czOf(q)]);
        };
        auto target = [&](auto qc) -> long long {
            constexpr int q = decltype(qc)::value;
            return xs[1+cxOf(q)] + (long long) nx*(ys[1+cyOf(q)] + (long long) ny*zs[1+czOf(q)]);
        };
        // Moments of x at this step, from the input array, as in the dense kernel.
        R f[19];
        staticFor<19>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            f[q] = loadq<T, R>(A + (long long) q*N + source(qc), q);
        });
        // What the node reads of the step's output: for Density faces every arriving population (for an unknown
        // direction the one sent against it), for walls and Velocity faces those of the mass balance, and the values
        // that the rebuilt ones replace (`old`; for a solid source the population that x sent into the wall).
        R in[19], old[19];
        staticFor<18>([&](auto ic) {
            constexpr int q = decltype(ic)::value + 1, p = oppOf(q);
            typedef std::integral_constant<int, q> Q;
            in[q] = old[q] = R(0);
            if (unknown & (1<<q)) {
                const long long src = source(Q());
                if (solid & (1<<q))
                    old[q] = loadq<T, R>(B + (long long) p*N + node, p);
                else {
                    const int x = xs[1-cxOf(q)];
                    const bool solidSource = v.solidMask != nullptr &&
                        ((v.solidMask[(ys[1-cyOf(q)] + (long long) ny*zs[1-czOf(q)])*v.wordsPerRow + x/32] >> (x%32)) & 1u);
                    // Across the face of a solid node the dense step wrote nothing: nothing leaves.
                    if (!solidSource)
                        old[q] = loadq<T, R>(B + (long long) q*N + src, q);
                }
                if (kind == KindDensity || (kind <= KindVelocity && !(solid & (1<<q)) && !(unknown & (1<<p))))
                    in[q] = loadq<T, R>(B + (long long) p*N + target(Q()), p);
            }
            else if (kind == KindDensity)
                in[q] = loadq<T, R>(B + (long long) q*N + source(Q()), q);
        });
        in[0] = kind == KindDensity ? loadq<T, R>(B + node, 0) : R(0);
        Moments<R> m = momentsOf<R>(f);
        R rhoNode = R(1) + m.dr;
        R jx = m.jx, jy = m.jy, jz = m.jz;
        if (remove) {
            jx -= rhoNode*R(v.stats->ucm[0]);
            jy -= rhoNode*R(v.stats->ucm[1]);
            jz -= rhoNode*R(v.stats->ucm[2]);
        }
        R rb = rhoNode, dr = m.dr;
        R ub[3] = {(jx + R(0.5)*(rb*gx))/rb, (jy + R(0.5)*(rb*gy))/rb, (jz + R(0.5)*(rb*gz))/rb};
        if (kind == KindWall || kind == KindDensityAtRest)
            ub[0] = ub[1] = ub[2] = 0;
        if (kind == KindVelocity || kind == KindDensityVelocity)
#pragma unroll
            for (int a = 0; a < 3; a++)
                ub[a] = R(faceData[4*face + a]);
        if (kind == KindDensity || kind == KindDensityAtRest || kind == KindDensityVelocity) {
            dr = R(faceData[4*face + 3]) - R(1);
            rb = R(faceData[4*face + 3]);
        }
        if (kind == KindDensity) {
            const int axis = face/2;
            R inward = (face%2 == 0 ? R(1) : R(-1)), sum = 0;
#pragma unroll
            for (int q = 0; q < 19; q++)
                sum += in[q];
#pragma unroll
            for (int a = 0; a < 3; a++)
                if (a == axis)
                    ub[a] = R(0.5)*(inward*(dr - sum)/rb + ub[a]);
        }
        // The random part of an unknown direction: of a node at equilibrium (D3Q19::equilibriumFluctuation) minus c
        // times the stress part of the random part of the collision of x (ReferenceLBMKernels.cpp:1278-1284), or of
        // a collision at rho_b.  Both are sums over the modes, formed from one set of amplitudes.
        R a[15], r15 = 0, rx = 0, ry = 0, rz = 0;
        if (FLUCT) {
            R mu = R(v.mu);
            if (hasEquilibriumNoise(kind)) {
                const R cw = R(faceData[24]);
                R r[19], rc[15], ac[15];
                philoxNormals<R, 19>(v.seed, PurposeBoundary, node, step, r);
                R oneMinusC = R(1) - cw;
                modeAmplitudes<R>(r, sqrt(mu*rb*(oneMinusC > R(0) ? oneMinusC : R(0))), sqrt(mu*rb), a);
                philoxNormals<R, 15>(v.seed, PurposeFluid, node, step, rc);
                modeAmplitudes<R>(rc, sqrt(mu*rhoNode*omega*(R(2) - omega)), R(0), ac);
                R conserved = sqrt(mu*rb);
#pragma unroll
                for (int k = 0; k < 6; k++)
                    a[k] -= cw*ac[k];
                r15 = conserved*r[15];
                rx = conserved*R(1.7320508075688772)*r[16];
                ry = conserved*R(1.7320508075688772)*r[17];
                rz = conserved*R(1.7320508075688772)*r[18];
            }
            else {
                R r[15];
                philoxNormals<R, 15>(v.seed, PurposeBoundary, node, step, r);
                modeAmplitudes<R>(r, sqrt(mu*rb*omega*(R(2) - omega)), sqrt(mu*rb), a);
            }
        }
        auto noise = [&](auto qc) -> R {
            constexpr int q = decltype(qc)::value;
            return FLUCT ? fluctuationTerm<R, q>(a) + wOf<R>(q)*(r15 + along<R, q>(rx, ry, rz)) : R(0);
        };
        R Fb[3] = {gx*rb, gy*rb, gz*rb};
        if (kind == KindWall || kind == KindVelocity) {
            // Mass balance (ReferenceLBMKernels.cpp:1290-1325), linear in rho_b = 1 + dr.
            R numerator = 0, denominator = 0;
            staticFor<18>([&](auto ic) {
                constexpr int q = decltype(ic)::value + 1, p = oppOf(q);
                typedef std::integral_constant<int, q> Q;
                const bool wall = (solid & (1<<q)) != 0;
                if (!(unknown & (1<<q)) || (!wall && (unknown & (1<<p))))
                    return;
                const R arriving = wall ? old[q] : in[q];
                const R flux = wall ? R(0) : R(6)*wOf<R>(q)*along<R, q>(ub[0], ub[1], ub[2]);
                const R e0 = eqDeviation<R, q>(R(0), ub[0], ub[1], ub[2]);
                const R sg = guoAt<R, q>(ub[0], ub[1], ub[2], gx, gy, gz);
                const R rest = (R(1) - omega)*fneqAt<R, q>(m) + noise(Q());
                numerator += arriving - rest - e0 - R(0.5)*sg + flux;
                denominator += wOf<R>(q) + e0 + R(0.5)*sg - flux;
            });
            if (denominator != R(0)) {
                dr = numerator/denominator;
                rb = R(1) + dr;
                Fb[0] = gx*rb; Fb[1] = gy*rb; Fb[2] = gz*rb;
            }
        }
        staticFor<18>([&](auto ic) {
            constexpr int q = decltype(ic)::value + 1;
            typedef std::integral_constant<int, q> Q;
            if (!(unknown & (1<<q)))
                return;
            const R value = eqDeviation<R, q>(dr, ub[0], ub[1], ub[2]) + (R(1) - omega)*fneqAt<R, q>(m)
                          + R(0.5)*guoAt<R, q>(ub[0], ub[1], ub[2], Fb[0], Fb[1], Fb[2]) + noise(Q());
            T word;
            storeq<T, R>(&word, q, value);
            B[(long long) q*N + source(Q())] = word;
            const double stored = (double) loadq<T, R>(&word, q), leaves = (double) old[q];
            // Mass and momentum bookkeeping of the step sums: the value that would have arrived leaves, the rebuilt
            // one enters.  For a solid source the population that x sent into the wall leaves instead; it moves along
            // -c_q.
            const double momentum = (solid & (1<<q)) ? stored + leaves : stored - leaves;
            acc[0] += stored - leaves;
            acc[1] += momentum*cxOf(q);
            acc[2] += momentum*cyOf(q);
            acc[3] += momentum*czOf(q);
            if (solid & (1<<q)) {
                // The wall receives the momentum of the population sent along -c_q and gives that of the rebuilt
                // one along c_q (full populations, ReferenceLBMKernels.cpp:1332-1338).
                const double given = leaves + (double) value + 2.0*wOf<double>(q);
                acc[4] -= cxOf(q)*given;
                acc[5] -= cyOf(q)*given;
                acc[6] -= czOf(q)*given;
            }
        });
    }
    // Block of 64 threads: pad the reduction to the generic routine.
    blockReduceStore(acc, partials + NPART*(long long) blockIdx.x);
}

// ---------------------------------------------------------------------------------------------------
// The sums of a moments pass, or of a step with sparse passes: one block adds the records in a fixed order.
// ---------------------------------------------------------------------------------------------------

__global__ void __launch_bounds__(THREADS) finishKernel(const double* records, int count, FluidView v, int mode) {
    const double* partials = afterPrevious(records);
    sumRecords<false>(partials, count, v, mode);
}

// ---------------------------------------------------------------------------------------------------
// Moments of the current state (post-stream values pulled from the input array).
// ---------------------------------------------------------------------------------------------------

template <typename T, typename R>
__global__ void __launch_bounds__(THREADS) momentsKernel(const T* __restrict__ A, FluidView v) {
    double acc[NPART] = {0, 0, 0, 0, 0, 0, 0, 0};
    const int lane = threadIdx.x%32, warp = threadIdx.x/32;
    for (long long t = blockIdx.x; t < v.numTiles; t += gridDim.x) {
        int tx = (int) (t%v.tilesX);
        long long rr = t/v.tilesX;
        int ty = (int) (rr%v.tilesY);
        int z = (int) (rr/v.tilesY);
        int x = tx*TX + lane, y = ty*TY + warp;
        if (x >= v.nx || y >= v.ny)
            continue;
        long long row = (long long) z*v.ny + y;
        if (v.solidMask != nullptr && ((__ldg(&v.solidMask[row*v.wordsPerRow + tx]) >> lane) & 1u))
            continue;
        R dr = 0, jx = 0, jy = 0, jz = 0;
        for (int q = 0; q < 19; q++) {
            R fq = loadq<T, R>(A + (long long) q*v.n + shifted(v, x, y, z, -cxr(q), -cyr(q), -czr(q)), q);
            dr += fq;
            jx += cxr(q)*fq;
            jy += cyr(q)*fq;
            jz += czr(q)*fq;
        }
        double r = 1.0 + (double) dr;
        acc[0] += (double) dr;
        acc[1] += (double) jx;
        acc[2] += (double) jy;
        acc[3] += (double) jz;
        double s2 = ((double) jx*jx + (double) jy*jy + (double) jz*jz)/(r*r);
        acc[7] = fmax(acc[7], s2);
    }
    blockReduceStore(acc, v.partials + NPART*(long long) blockIdx.x);
}

// The steady-state residual of the build (the reference defines none): r = max over fluid nodes of |u - u_prev|,
// and max |u|, with u = j/rho of the post-stream state in FP64; u_prev (3N doubles, [a*N + node]) is replaced by u.
// Per block: partials[NPART*b] = max |u - u_prev|^2, partials[NPART*b + 7] = max |u|^2.
template <typename T, typename R>
__global__ void __launch_bounds__(THREADS) residualKernel(const T* __restrict__ A, FluidView v, double* prev, int first) {
    double maxDiff2 = 0, maxU2 = 0;
    const int lane = threadIdx.x%32, warp = threadIdx.x/32;
    for (long long t = blockIdx.x; t < v.numTiles; t += gridDim.x) {
        int tx = (int) (t%v.tilesX);
        long long rr = t/v.tilesX;
        int ty = (int) (rr%v.tilesY);
        int z = (int) (rr/v.tilesY);
        int x = tx*TX + lane, y = ty*TY + warp;
        if (x >= v.nx || y >= v.ny)
            continue;
        long long row = (long long) z*v.ny + y;
        if (v.solidMask != nullptr && ((__ldg(&v.solidMask[row*v.wordsPerRow + tx]) >> lane) & 1u))
            continue;
        double dr = 0, jx = 0, jy = 0, jz = 0;
        for (int q = 0; q < 19; q++) {
            double fq = (double) loadq<T, R>(A + (long long) q*v.n + shifted(v, x, y, z, -cxr(q), -cyr(q), -czr(q)), q);
            dr += fq;
            jx += cxr(q)*fq;
            jy += cyr(q)*fq;
            jz += czr(q)*fq;
        }
        double inv = 1.0/(1.0 + dr);
        double u[3] = {jx*inv, jy*inv, jz*inv};
        long long node = row*v.nx + x;
        double d2 = 0;
        for (int a = 0; a < 3; a++) {
            double* p = prev + a*v.n + node;
            double d = u[a] - *p;
            d2 += d*d;
            *p = u[a];
        }
        if (!first)
            maxDiff2 = fmax(maxDiff2, d2);
        maxU2 = fmax(maxU2, u[0]*u[0] + u[1]*u[1] + u[2]*u[2]);
    }
    for (int o = 16; o > 0; o >>= 1) {
        maxDiff2 = fmax(maxDiff2, __shfl_down_sync(0xffffffffu, maxDiff2, o));
        maxU2 = fmax(maxU2, __shfl_down_sync(0xffffffffu, maxU2, o));
    }
    __shared__ double red[THREADS/32][2];
    if (lane == 0) {
        red[warp][0] = maxDiff2;
        red[warp][1] = maxU2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < THREADS/32; w++) {
            maxDiff2 = fmax(maxDiff2, red[w][0]);
            maxU2 = fmax(maxU2, red[w][1]);
        }
        v.partials[NPART*(long long) blockIdx.x] = maxDiff2;
        v.partials[NPART*(long long) blockIdx.x + 7] = maxU2;
    }
}

// ---------------------------------------------------------------------------------------------------
// Initial state and state transfer.
// ---------------------------------------------------------------------------------------------------

// Equilibrium at the initial velocity on fluid nodes and -w_q on solid nodes, in the pull layout:
// A_q(y) = f_q(y + c_q) (ReferenceLBMKernels.cpp:53-79).
template <typename T, typename R>
__global__ void initKernel(T* A, T* B, FluidView v, const char* fluid, double ux, double uy, double uz) {
    long long total = 19*v.n;
    for (long long i = blockIdx.x*(long long) blockDim.x + threadIdx.x; i < total; i += (long long) gridDim.x*blockDim.x) {
        int q = (int) (i/v.n);
        long long y = i%v.n;
        Coords c = nodeCoords(y, v.nx, v.ny);
        long long target = shifted(v, c.x, c.y, c.z, cxr(q), cyr(q), czr(q));
        double value;
        if (fluid != nullptr && !fluid[target])
            value = -weightOf<double>(q);
        else {
            double uu = ux*ux + uy*uy + uz*uz;
            double cu = cxr(q)*ux + cyr(q)*uy + czr(q)*uz;
            value = weightOf<double>(q)*(0.0 + 1.0*(3.0*cu + 4.5*cu*cu - 1.5*uu));
        }
        storeq<T, R>(A + i, q, (R) value);
        storeq<T, R>(B + i, q, (R) value);
    }
}

// Plane q of the state: out[x] = f_q(x) = A_q(x - c_q).
template <typename T, typename R>
__global__ void gatherKernel(const T* A, int q, FluidView v, double* out) {
    for (long long x = blockIdx.x*(long long) blockDim.x + threadIdx.x; x < v.n; x += (long long) gridDim.x*blockDim.x) {
        Coords c = nodeCoords(x, v.nx, v.ny);
        out[x] = (double) loadq<T, R>(A + (long long) q*v.n + shifted(v, c.x, c.y, c.z, -cxr(q), -cyr(q), -czr(q)), q);
    }
}

template <typename T>
__device__ __forceinline__ bool bitsEqual(const T& a, const T& b) {
    const unsigned char* pa = reinterpret_cast<const unsigned char*>(&a);
    const unsigned char* pb = reinterpret_cast<const unsigned char*>(&b);
    for (int i = 0; i < (int) sizeof(T); i++)
        if (pa[i] != pb[i])
            return false;
    return true;
}

// Plane q of a state into both arrays: A_q(y) = f_q(y + c_q).  *changed is set when a stored element of A
// changes, so that setting the state a kernel already holds keeps the sums of its last step (bitwise restarts).
template <typename T, typename R>
__global__ void scatterKernel(T* A, T* B, int q, FluidView v, const double* in, int* changed) {
    for (long long y = blockIdx.x*(long long) blockDim.x + threadIdx.x; y < v.n; y += (long long) gridDim.x*blockDim.x) {
        Coords c = nodeCoords(y, v.nx, v.ny);
        R value = (R) in[shifted(v, c.x, c.y, c.z, cxr(q), cyr(q), czr(q))];
        T before = A[(long long) q*v.n + y];
        storeq<T, R>(A + (long long) q*v.n + y, q, value);
        T after = A[(long long) q*v.n + y];
        if (!bitsEqual(before, after))
            *changed = 1;
        storeq<T, R>(B + (long long) q*v.n + y, q, value);
    }
}

// Velocity component a of node (x, y, z) in lattice units, 0 at solid nodes; out-of-lattice neighbours (open faces)
// take the value of the node itself.
__device__ __forceinline__ double velocityAt(const FluidView& v, const double* velocity, double scale, int x, int y,
                                            int z, int a, long long self) {
    long long node;
    if (x < 0 || x >= v.nx || y < 0 || y >= v.ny || z < 0 || z >= v.nz) {
        if (v.faceOpen)
            node = self;
        else
            node = wrap(x, v.nx) + (long long) v.nx*(wrap(y, v.ny) + (long long) v.ny*wrap(z, v.nz));
    }
    else
        node = x + (long long) v.nx*(y + (long long) v.ny*z);
    long long row = node/v.nx;
    int xx = (int) (node - row*v.nx);
    if (v.solidMask != nullptr && ((v.solidMask[row*v.wordsPerRow + xx/32] >> (xx%32)) & 1u))
        return 0.0;
    return velocity[3*node + a]/scale;
}

// Populations of given fields (density [N], velocity [N][3] in the units of the fields, divided by the scales into
// lattice units), written in the pull layout of both arrays: slot (q, y) holds the population that node x = y + c_q
// pulls, the equilibrium w_q (rho - 1 + rho (3 c.u + 4.5 (c.u)^2 - 1.5 u^2)) of x plus, with `strain`, the
// Chapman-Enskog non-equilibrium part -3 tau w_q rho (c.S.c - tr S/3) of the strain rate S (central differences of
// the velocity, zero velocity at solid nodes), so that a steady flow starts without the transient of a stress-free
// state; solid nodes hold 0.
template <typename T, typename R>
__global__ void equilibriumKernel(T* A, T* B, FluidView v, const double* density, const double* velocity,
                                  double densityScale, double velocityScale, int strain) {
    for (long long t = blockIdx.x*(long long) blockDim.x + threadIdx.x; t < 19*v.n; t += (long long) gridDim.x*blockDim.x) {
        int q = (int) (t/v.n);
        long long y = t - q*v.n;
        Coords c = nodeCoords(y, v.nx, v.ny);
        long long x = shifted(v, c.x, c.y, c.z, cxr(q), cyr(q), czr(q));
        Coords cx = nodeCoords(x, v.nx, v.ny);
        long long row = (long long) cx.z*v.ny + cx.y;
        double value = 0;
        if (v.solidMask == nullptr || !((v.solidMask[row*v.wordsPerRow + cx.x/32] >> (cx.x%32)) & 1u)) {
            double rho = density[x]/densityScale;
            double u[3] = {velocity[3*x]/velocityScale, velocity[3*x+1]/velocityScale, velocity[3*x+2]/velocityScale};
            double cu = cxr(q)*u[0] + cyr(q)*u[1] + czr(q)*u[2];
            double uu = u[0]*u[0] + u[1]*u[1] + u[2]*u[2];
            value = weightOf<double>(q)*(rho - 1.0 + rho*(3.0*cu + 4.5*cu*cu - 1.5*uu));
            if (strain) {
                // grad[a][b] = d u_b / d x_a
                double grad[3][3];
                int cxyz[3] = {cx.x, cx.y, cx.z};
                for (int a = 0; a < 3; a++) {
                    int p[3] = {cxyz[0], cxyz[1], cxyz[2]}, m[3] = {cxyz[0], cxyz[1], cxyz[2]};
                    p[a]++;
                    m[a]--;
                    for (int b = 0; b < 3; b++)
                        grad[a][b] = 0.5*(velocityAt(v, velocity, velocityScale, p[0], p[1], p[2], b, x)
                                          - velocityAt(v, velocity, velocityScale, m[0], m[1], m[2], b, x));
                }
                double c[3] = {(double) cxr(q), (double) cyr(q), (double) czr(q)};
                double cSc = 0, tr = grad[0][0] + grad[1][1] + grad[2][2];
                for (int a = 0; a < 3; a++)
                    for (int b = 0; b < 3; b++)
                        cSc += c[a]*c[b]*0.5*(grad[a][b] + grad[b][a]);
                value += -3.0*(1.0/v.omega)*weightOf<double>(q)*rho*(cSc - tr/3.0);
            }
        }
        storeq<T, R>(A + t, q, (R) value);
        storeq<T, R>(B + t, q, (R) value);
    }
}

// Density [N] and velocity [N][3], u = j/rho + g/2, of every node, zero at solid nodes (nodeFields,
// ReferenceLBMKernels.cpp:1349-1368), in the layout of the caller's arrays.
template <typename T, typename R>
__global__ void fieldsKernel(const T* A, FluidView v, double* density, double* velocity, double densityScale,
                             double velocityScale) {
    for (long long x = blockIdx.x*(long long) blockDim.x + threadIdx.x; x < v.n; x += (long long) gridDim.x*blockDim.x) {
        const Coords c = nodeCoords(x, v.nx, v.ny);
        const long long row = (long long) c.z*v.ny + c.y;
        if (v.solidMask != nullptr && ((v.solidMask[row*v.wordsPerRow + c.x/32] >> (c.x%32)) & 1u)) {
            density[x] = velocity[3*x] = velocity[3*x+1] = velocity[3*x+2] = 0;
            continue;
        }
        double r = 1.0, jx = 0, jy = 0, jz = 0;
        staticFor<19>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            const double fq = (double) loadq<T, R>(A + (long long) q*v.n + shifted(v, c.x, c.y, c.z, -cxOf(q), -cyOf(q), -czOf(q)), q);
            r += fq;
            jx += cxOf(q)*fq;
            jy += cyOf(q)*fq;
            jz += czOf(q)*fq;
        });
        density[x] = r*densityScale;
        velocity[3*x] = (jx*(1.0/r) + v.g[0]*0.5)*velocityScale;
        velocity[3*x+1] = (jy*(1.0/r) + v.g[1]*0.5)*velocityScale;
        velocity[3*x+2] = (jz*(1.0/r) + v.g[2]*0.5)*velocityScale;
    }
}

// ---------------------------------------------------------------------------------------------------
// Launch tables per storage type.
// ---------------------------------------------------------------------------------------------------

template <typename T> struct ComputeOf { typedef float type; };
template <> struct ComputeOf<double> { typedef double type; };

const long long kFinishInDense = 1LL << 21;   // nodes up to which the dense kernel can add up the step's sums itself

// Launches a kernel of the step, as a programmatic dependent of the one before it on the stream where `follow`
// (FluidEngine::follows).
template <typename... P, typename... Args>
void launch(bool follow, void (*kernel)(P...), int grid, int threads, cudaStream_t stream, Args... args) {
    if (!follow) {
        kernel<<<grid, threads, 0, stream>>>(args...);
        return;
    }
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3((unsigned) grid);
    config.blockDim = dim3((unsigned) threads);
    config.stream = stream;
    config.attrs = &attribute;
    config.numAttrs = 1;
    CUDA_CHECK(cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...));
}

template <typename T>
struct Launcher {
    typedef typename ComputeOf<T>::type R;

    // The paired kernel serves FP32 and 16-bit storage on lattices with an even nx (measured at 256^3, FP32: 0.596
    // against 0.677 ms per launch with fluctuations, 0.464 against 0.482 ms without).  LBM_B200_PAIRED16 = 0 and
    // LBM_B200_PAIRED32 = 0 in the environment select the one-node kernel instead (for comparisons).
    static int pairChoice(const char* name) {
        const char* e = std::getenv(name);
        return e == nullptr ? -1 : (e[0] == '0' ? 0 : 1);
    }
    template <bool FL>
    static bool pairedKernels() {
        static int enabled = -2;
        if (enabled == -2) {
            if (sizeof(T) == 2) {
                int c = pairChoice("LBM_B200_PAIRED16");
                enabled = c == 0 ? 0 : 1;
            }
            else {
                int c = pairChoice("LBM_B200_PAIRED32");
                enabled = c == 0 ? 0 : 1;
            }
        }
        return enabled == 1;
    }

    // The quad kernel for 16-bit storage without fluctuations (nx % 4 == 0); LBM_B200_QUAD16 = 0 in the environment
    // selects the paired kernel instead (for comparisons).
    static bool quadKernels() {
        static int enabled = -2;
        if (enabled == -2)
            enabled = pairChoice("LBM_B200_QUAD16") == 0 ? 0 : 1;
        return enabled == 1;
    }

    // The persistent grid of a kernel variant: one wave of resident blocks (blocks per SM of this variant times
    // the SMs), so that every block processes the same number of tiles in one wave.
    template <bool S, bool RE, bool FL>
    static int residentGrid(const FluidView& v) {
        static int blocks = 0;
        if (blocks == 0) {
            int perSM = 0, device = 0, sms = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, streamCollideKernel<T, R, S, RE, FL, false>, THREADS, 0);
            cudaGetDevice(&device);
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
            blocks = std::max(1, perSM)*std::max(1, sms);
        }
        return (int) std::max(1LL, std::min((long long) blocks, v.numTiles));
    }
    template <bool S, bool RE, bool FL, bool FLAT>
    static int pairGrid(const FluidView& v) {
        static int blocks = 0;
        if (blocks == 0) {
            int perSM = 0, device = 0, sms = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, streamCollidePairKernel<T, S, RE, FL, false, FLAT>, THREADS, 0);
            cudaGetDevice(&device);
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
            blocks = std::max(1, perSM)*std::max(1, sms);
        }
        long long tiles = FLAT ? (v.n/2 + THREADS - 1)/THREADS : (long long) ((v.nx + PAIR_TX - 1)/PAIR_TX)*v.tilesY*v.nz;
        return (int) std::max(1LL, std::min((long long) blocks, tiles));
    }
    template <bool S, bool RE, bool FLAT>
    static int quadGrid(const FluidView& v) {
        static int blocks = 0;
        if (blocks == 0) {
            int perSM = 0, device = 0, sms = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, streamCollideQuadKernel<T, S, RE, false, FLAT>, LBM_QUAD_THREADS, 0);
            cudaGetDevice(&device);
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
            blocks = std::max(1, perSM)*std::max(1, sms);
        }
        const long long warps = LBM_QUAD_THREADS/32;
        long long tiles = FLAT ? (v.n/4 + 31)/32 : (long long) ((v.nx + QUAD_TX - 1)/QUAD_TX)*v.ny*v.nz;
        return (int) std::max(1LL, std::min((long long) blocks, (tiles + warps - 1)/warps));
    }
    // Whether the nodes are taken in their order, which leaves no lane and no row of a tile idle, instead of in row tiles:
    // FP32 44x36x30 8.4 -> 7.1 us, 100x90x80 27.7 -> 22.9, with solid nodes 200x180x170 184 -> 160; 16 bits gain 1.0
    // (128^3) to 1.57 times (136x120x110).  Not where the tiles are the faster ones: FP32 without solid nodes well beyond
    // the L2 cache (160^3 110 us, 118 in the nodes' order; 200x180x170 166 and 174; 192^3 204 and 198) and with particles
    // (128^3 5 us less per step).  And not on a 16-bit lattice with momentum removal: the split sets the order of the sums,
    // whose last bits the removal carries into the rounding of every population.
    template <bool S, bool RE>
    static bool flat(const FluidView& v) {
        if (sizeof(T) == 2)
            return !v.removes;
        return !RE && (S || v.n <= kFinishInDense);
    }
    template <bool S, bool RE, bool FLAT>
    static int quad(const void* A, void* B, const FluidView& v, int remove, long long step, int maxGrid, int finish, bool follow, cudaStream_t s) {
        const int grid = std::min(maxGrid, quadGrid<S, RE, FLAT>(v));
        launch(follow, finish ? streamCollideQuadKernel<T, S, RE, !S, FLAT> : streamCollideQuadKernel<T, S, RE, false, FLAT>,
               grid, LBM_QUAD_THREADS, s, (const T*) A, (T*) B, v, remove, step);
        return grid;
    }
    template <bool S, bool RE, bool FL, bool FLAT>
    static int pair(const void* A, void* B, const FluidView& v, int remove, long long step, int maxGrid, int finish, bool follow, cudaStream_t s) {
        const int grid = std::min(maxGrid, pairGrid<S, RE, FL, FLAT>(v));
        launch(follow, finish ? streamCollidePairKernel<T, S, RE, FL, !S, FLAT> : streamCollidePairKernel<T, S, RE, FL, false, FLAT>,
               grid, THREADS, s, (const T*) A, (T*) B, v, remove, step);
        return grid;
    }
    template <bool S, bool RE, bool FL>
    static int dense(const void* A, void* B, const FluidView& v, int remove, long long step, int maxGrid, int finish, bool follow, cudaStream_t s) {
        if constexpr (sizeof(T) == 2 && !FL) {
            if (v.nx%4 == 0 && pairedKernels<FL>() && quadKernels()) {
                return flat<S, RE>(v) ? quad<S, RE, true>(A, B, v, remove, step, maxGrid, finish, follow, s)
                                              : quad<S, RE, false>(A, B, v, remove, step, maxGrid, finish, follow, s);
            }
        }
        if constexpr (sizeof(T) <= 4) {
            if (v.nx%2 == 0 && pairedKernels<FL>()) {
                return flat<S, RE>(v) ? pair<S, RE, FL, true>(A, B, v, remove, step, maxGrid, finish, follow, s)
                                              : pair<S, RE, FL, false>(A, B, v, remove, step, maxGrid, finish, follow, s);
            }
        }
        int grid = std::min(maxGrid, residentGrid<S, RE, FL>(v));
        auto kernel = finish ? streamCollideKernel<T, R, S, RE, FL, !S> : streamCollideKernel<T, R, S, RE, FL, false>;
        launch(follow, kernel, grid, THREADS, s, (const T*) A, (T*) B, v, remove, step);
        return grid;
    }
    template <bool S, bool RE>
    static int denseF(bool fl, const void* A, void* B, const FluidView& v, int remove, long long step, int grid, int finish, bool follow, cudaStream_t s) {
        return fl ? dense<S, RE, true>(A, B, v, remove, step, grid, finish, follow, s) : dense<S, RE, false>(A, B, v, remove, step, grid, finish, follow, s);
    }
    template <bool S>
    static int denseR(bool re, bool fl, const void* A, void* B, const FluidView& v, int remove, long long step, int grid, int finish, bool follow, cudaStream_t s) {
        return re ? denseF<S, true>(fl, A, B, v, remove, step, grid, finish, follow, s) : denseF<S, false>(fl, A, B, v, remove, step, grid, finish, follow, s);
    }
    // Launch the dense step; returns the grid it used (one partial record per block).
    static int denseAny(bool so, bool re, bool fl, const void* A, void* B, const FluidView& v, int remove, long long step,
                        int grid, int finish, bool follow, cudaStream_t s) {
        return so ? denseR<true>(re, fl, A, B, v, remove, step, grid, finish, follow, s) : denseR<false>(re, fl, A, B, v, remove, step, grid, finish, follow, s);
    }
    static int occupancy() {
        // The largest grid any variant uses (the partial sums are sized for it).
        int best = 1;
        auto probe = [&](auto kernel) {
            int blocks = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, THREADS, 0);
            best = std::max(best, blocks);
        };
        probe(streamCollideKernel<T, R, false, false, false, false>);
        probe(streamCollideKernel<T, R, false, false, true, false>);
        probe(streamCollideKernel<T, R, true, true, true, false>);
        probe(streamCollideKernel<T, R, true, false, false, false>);
        if constexpr (sizeof(T) <= 4) {
            probe(streamCollidePairKernel<T, false, false, false, false, false>);
            probe(streamCollidePairKernel<T, false, true, true, false, false>);
            probe(streamCollidePairKernel<T, true, true, true, false, false>);
        }
        if constexpr (sizeof(T) == 2) {
            auto probeQuad = [&](auto kernel) {
                int blocks = 0;
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, LBM_QUAD_THREADS, 0);
                best = std::max(best, blocks);
            };
            probeQuad(streamCollideQuadKernel<T, false, false, false, false>);
            probeQuad(streamCollideQuadKernel<T, true, true, false, false>);
        }
        return best;
    }
    static void bounceBack(void* B, const int* wall, int numWall, const FluidView& v, double* partials, int grid, bool follow, cudaStream_t s) {
        launch(follow, bounceBackKernel<T, R>, grid, THREADS, s, (T*) B, wall, numWall, v, partials);
    }
    static void boundary(bool fl, const void* A, void* B, const int* bnd, int count, const FluidView& v, int remove, long long step,
                         double* partials, const double* faceData, int grid, bool follow, cudaStream_t s) {
        launch(follow, fl ? boundaryKernel<T, R, true> : boundaryKernel<T, R, false>, grid, kBoundaryThreads, s, (const T*) A, (T*) B,
                    bnd, count, v, remove, step, partials, faceData);
    }
    static void moments(const void* A, const FluidView& v, int grid, cudaStream_t s) {
        momentsKernel<T, R><<<grid, THREADS, 0, s>>>((const T*) A, v);
    }
    static void equilibrium(void* A, void* B, const FluidView& v, const double* rho, const double* u, double ds,
                            double vs, int strain, cudaStream_t s) {
        equilibriumKernel<T, R><<<1184, 256, 0, s>>>((T*) A, (T*) B, v, rho, u, ds, vs, strain);
    }
    static void residual(const void* A, const FluidView& v, double* prev, int first, int grid, cudaStream_t s) {
        residualKernel<T, R><<<grid, THREADS, 0, s>>>((const T*) A, v, prev, first);
    }
    static void init(void* A, void* B, const FluidView& v, const char* fluid, const double* u, cudaStream_t s) {
        initKernel<T, R><<<1184, 256, 0, s>>>((T*) A, (T*) B, v, fluid, u[0], u[1], u[2]);
    }
    static void gather(const void* A, int q, const FluidView& v, double* out, cudaStream_t s) {
        gatherKernel<T, R><<<1184, 256, 0, s>>>((const T*) A, q, v, out);
    }
    static void scatter(void* A, void* B, int q, const FluidView& v, const double* in, int* changed, cudaStream_t s) {
        scatterKernel<T, R><<<1184, 256, 0, s>>>((T*) A, (T*) B, q, v, in, changed);
    }
    static void fields(const void* A, const FluidView& v, double* rho, double* u, double ds, double vs, cudaStream_t s) {
        fieldsKernel<T, R><<<1184, 256, 0, s>>>((const T*) A, v, rho, u, ds, vs);
    }
};

template <typename F>
void dispatchStorage(int storage, F&& f) {
    switch (storage) {
    case LBM_STORAGE_F64: f(Launcher<double>()); break;
    case LBM_STORAGE_F32: f(Launcher<float>()); break;
    case LBM_STORAGE_F16: f(Launcher<__half>()); break;
    case LBM_STORAGE_BF16: f(Launcher<__nv_bfloat16>()); break;
    default: throw Error(LBM_ERR_NOT_SUPPORTED, "unknown storage type");
    }
}

size_t elementSizeOf(int storage) {
    switch (storage) {
    case LBM_STORAGE_F64: return 8;
    case LBM_STORAGE_F32: return 4;
    case LBM_STORAGE_F16: return 2;
    case LBM_STORAGE_BF16: return 2;
    default: throw Error(LBM_ERR_NOT_SUPPORTED, "unknown storage type");
    }
}

const int kGridSparse = 4*148;    // blocks of the boundary pass (a boundary node per thread up to 38,000 nodes)
const int kGridWall = 4*148;      // blocks of the bounce-back pass (a wall node per thread on the largest lattices)

} // namespace

FluidEngine::FluidEngine(const LbmLatticeParameters& l, int storage, const Geometry& g, cudaStream_t s)
        : lattice(l), storageType(storage), elementSize(elementSizeOf(storage)), stream(s), cur(0), gridBlocks(0),
          solidMaskDev(nullptr), reactMaskDev(nullptr), reactionDev(nullptr), partialsDev(nullptr), statsDev(nullptr),
          numWall(0), numBoundary(0), wallDev(nullptr), boundaryDev(nullptr), equilibriumNoise(false),
          stagingDev(nullptr), extraBlocks(0), faceDev(nullptr), profiling(false), profileUsed(0) {
    launches = 0;
    pop[0] = pop[1] = nullptr;
    std::memset(&view, 0, sizeof(view));
    view.nx = l.nx;
    view.ny = l.ny;
    view.nz = l.nz;
    view.n = (long long) l.nx*l.ny*l.nz;
    // The dense kernel indexes nodes with 32-bit unsigned integers (4.29e9 nodes: 163 GB of FP16 populations).
    if (view.n >= (1LL << 32) || (long long) l.nx*l.ny >= (1LL << 31))
        throw Error(LBM_ERR_INVALID_ARGUMENT, "The lattice has too many nodes for one device (at most 2^32 nodes, "
                    "and nx*ny below 2^31)");
    view.wordsPerRow = (l.nx + 31)/32;
    view.tilesX = (l.nx + TX - 1)/TX;
    view.tilesY = (l.ny + TY - 1)/TY;
    view.numTiles = (long long) view.tilesX*view.tilesY*l.nz;
    view.numFluid = (double) (view.n - (long long) g.solidNodes.size());
    solidNodes = g.solidNodes;
    try {
        CUDA_CHECK(cudaMalloc(&faceDev, sizeof(double)*32));
        setParameters(l);
        size_t bytes = (size_t) 19*view.n*elementSize;
        CUDA_CHECK(cudaMalloc(&pop[0], bytes));
        CUDA_CHECK(cudaMalloc(&pop[1], bytes));
        int device = 0, sms = 0;
        CUDA_CHECK(cudaGetDevice(&device));
        hostCopy = HostCopy::forDevice(device);
        CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
        int occupancy = 1;
        dispatchStorage(storage, [&](auto L) { occupancy = decltype(L)::occupancy(); });
        long long wanted = (long long) sms*occupancy;
        gridBlocks = (int) std::max(1LL, std::min(wanted, view.numTiles));
        extraBlocks = kGridWall + kGridSparse;
        CUDA_CHECK(cudaMalloc(&partialsDev, sizeof(double)*NPART*(size_t) (gridBlocks + extraBlocks + 1)));
        CUDA_CHECK(cudaMalloc(&statsDev, sizeof(StepStats) + sizeof(unsigned)));
        CUDA_CHECK(cudaMemsetAsync(statsDev, 0, sizeof(StepStats) + sizeof(unsigned), stream));
        view.partials = partialsDev;
        view.stats = statsDev;
        view.ticket = reinterpret_cast<unsigned*>(statsDev + 1);

        // Solid mask, rows padded to 32-bit words.
        char* fluidDev = nullptr;
        if (!g.solidNodes.empty()) {
            size_t words = (size_t) view.wordsPerRow*l.ny*l.nz;
            std::vector<uint32_t> mask(words, 0u);
            for (int sn : g.solidNodes) {
                long long row = sn/l.nx;
                int x = (int) (sn%l.nx);
                mask[row*view.wordsPerRow + x/32] |= 1u << (x%32);
            }
            CUDA_CHECK(cudaMalloc(&solidMaskDev, sizeof(uint32_t)*words));
            CUDA_CHECK(cudaMemcpyAsync(solidMaskDev, mask.data(), sizeof(uint32_t)*words, cudaMemcpyHostToDevice, stream));
            CUDA_CHECK(cudaMalloc(&fluidDev, view.n));
            CUDA_CHECK(cudaMemcpyAsync(fluidDev, g.fluid.data(), view.n, cudaMemcpyHostToDevice, stream));
        }
        view.solidMask = solidMaskDev;
        numWall = (int) g.wallNodes.size();
        if (numWall > 0) {
            std::vector<int> w(2*numWall);
            for (int i = 0; i < numWall; i++) {
                w[2*i] = g.wallNodes[i];
                w[2*i+1] = g.wallLinks[i];
            }
            CUDA_CHECK(cudaMalloc(&wallDev, sizeof(int)*w.size()));
            CUDA_CHECK(cudaMemcpyAsync(wallDev, w.data(), sizeof(int)*w.size(), cudaMemcpyHostToDevice, stream));
        }
        numBoundary = (int) g.boundaryNodes.size();
        if (numBoundary > 0) {
            std::vector<int> b(4*numBoundary);
            for (int i = 0; i < numBoundary; i++) {
                b[4*i] = g.boundaryNodes[i];
                b[4*i+1] = g.unknown[i];
                b[4*i+2] = g.solidBits[i];
                b[4*i+3] = g.kind[i] | ((g.face[i] + 1) << 8);
                equilibriumNoise = equilibriumNoise || hasEquilibriumNoise(g.kind[i]);
            }
            CUDA_CHECK(cudaMalloc(&boundaryDev, sizeof(int)*b.size()));
            CUDA_CHECK(cudaMemcpyAsync(boundaryDev, b.data(), sizeof(int)*b.size(), cudaMemcpyHostToDevice, stream));
        }
        double u[3] = {l.initial_velocity[0], l.initial_velocity[1], l.initial_velocity[2]};
        dispatchStorage(storage, [&](auto L) { decltype(L)::init(pop[0], pop[1], view, fluidDev, u, stream); });
        CUDA_CHECK(cudaGetLastError());
        if (fluidDev) {
            CUDA_CHECK(cudaStreamSynchronize(stream));
            cudaFree(fluidDev);
        }
        momentsPass(true);
        CUDA_CHECK(cudaStreamSynchronize(stream));
    }
    catch (...) {
        release();
        throw;
    }
}

FluidEngine::~FluidEngine() {
    release();
}

void FluidEngine::release() {
    cudaFree(pop[0]);
    cudaFree(pop[1]);
    cudaFree(solidMaskDev);
    cudaFree(reactMaskDev);
    cudaFree(reactionDev);
    cudaFree(partialsDev);
    cudaFree(statsDev);
    cudaFree(wallDev);
    cudaFree(boundaryDev);
    cudaFree(stagingDev);
    cudaFree(faceDev);
    cudaFree(residualPrevDev);
    residualPrevDev = nullptr;
    faceDev = nullptr;
    for (cudaEvent_t e : profileEvents)
        cudaEventDestroy(e);
    profileEvents.clear();
    pop[0] = pop[1] = nullptr;
    solidMaskDev = reactMaskDev = nullptr;
    reactionDev = stagingDev = nullptr;
    partialsDev = nullptr;
    statsDev = nullptr;
    wallDev = boundaryDev = nullptr;
}

void FluidEngine::setParameters(const LbmLatticeParameters& l) {
    lattice = l;
    view.omega = l.omega;
    for (int a = 0; a < 3; a++)
        view.g[a] = l.body_acceleration[a];
    uint32_t seed = (uint32_t) l.random_number_seed;
    view.seed = seed;
    view.removes = l.momentum_removal_frequency > 0;
    view.faceOpen = 0;
    for (int f = 0; f < 6; f++)
        if (l.face_boundary[f] != LBM_BOUNDARY_PERIODIC)
            view.faceOpen = 1;
    double cellMass = l.density*l.dx*l.dx*l.dx;
    bool fluctuate = l.fluid_fluctuations && l.fluid_kT > 0;
    view.mu = fluctuate ? 3.0*l.fluid_kT*l.dt*l.dt/(cellMass*l.dx*l.dx) : 0.0;
    // Face velocities and densities, and the boundary stress weight c = (1 - omega)^2/(omega (2 - omega))
    // (D3Q19.h:206-208), for the boundary kernel.
    for (int f = 0; f < 6; f++) {
        for (int a = 0; a < 3; a++)
            faceHost[4*f + a] = l.face_velocity[f][a];
        faceHost[4*f + 3] = l.face_density[f];
    }
    faceHost[24] = (1.0-l.omega)*(1.0-l.omega)/(l.omega*(2.0-l.omega));
    CUDA_CHECK(cudaMemcpyAsync(faceDev, faceHost, sizeof(double)*25, cudaMemcpyHostToDevice, stream));
    CUDA_CHECK(cudaStreamSynchronize(stream));
}

void FluidEngine::enableReaction() {
    if (reactionDev != nullptr)
        return;
    size_t words = (size_t) view.wordsPerRow*lattice.ny*lattice.nz;
    size_t r = (storageType == LBM_STORAGE_F64 ? 8 : 4);
    CUDA_CHECK(cudaMalloc(&reactMaskDev, sizeof(uint32_t)*words));
    CUDA_CHECK(cudaMemsetAsync(reactMaskDev, 0, sizeof(uint32_t)*words, stream));
    CUDA_CHECK(cudaMalloc(&reactionDev, 4*r*(size_t) view.n));
    CUDA_CHECK(cudaMemsetAsync(reactionDev, 0, 4*r*(size_t) view.n, stream));
    view.reactMask = reactMaskDev;
    view.reaction = reactionDev;
}

void FluidEngine::clearReactMask(cudaStream_t s) {
    if (reactMaskDev != nullptr)
        CUDA_CHECK(cudaMemsetAsync(reactMaskDev, 0, sizeof(uint32_t)*(size_t) view.wordsPerRow*lattice.ny*lattice.nz, s));
}

// Whether the kernels of a step follow one another as programmatic dependents.  Not in a step with particles, whose
// kernels follow those of the coupling and whose arrays the host waits for: such a launch costs the host more
// (32^3 with 64 particles and host arrays: 50 steps 5.0 ms, 4.9 in the plain order).  On the legacy default stream and
// under capture the plain order is kept.
bool FluidEngine::follows(bool react) const {
    if ((react && reactionDev != nullptr) || stream == nullptr || stream == cudaStreamLegacy)
        return false;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    CUDA_CHECK(cudaStreamIsCapturing(stream, &capture));
    return capture == cudaStreamCaptureStatusNone;
}

void FluidEngine::step(long long stepIndex, bool remove, bool react) {
    const void* A = pop[cur];
    void* B = pop[1-cur];
    bool fluct = view.mu > 0;
    bool solids = solidMaskDev != nullptr;
    if (profiling) {
        if (profileUsed + 2 > profileEvents.size())
            for (int i = 0; i < 2; i++) {
                cudaEvent_t e;
                CUDA_CHECK(cudaEventCreate(&e));
                profileEvents.push_back(e);
            }
        CUDA_CHECK(cudaEventRecord(profileEvents[profileUsed], stream));
    }
    // Small lattices without solid nodes and open faces add up the step's sums in the dense kernel
    // (finishStep), where the launch that this saves shows; at 192^3 nothing is gained, and the coupled step at 256^3 was
    // 1% slower with it.
    const bool separate = solids || numBoundary > 0 || view.n > kFinishInDense;
    const bool follow = follows(react);
    int denseGrid = gridBlocks;
    dispatchStorage(storageType, [&](auto L) {
        denseGrid = decltype(L)::denseAny(solids, react && reactionDev != nullptr, fluct, A, B, view, remove ? 1 : 0,
                                          stepIndex, gridBlocks, separate ? 0 : 1, follow, stream);
    });
    CUDA_CHECK(cudaGetLastError());
    launches++;
    if (profiling) {
        CUDA_CHECK(cudaEventRecord(profileEvents[profileUsed + 1], stream));
        profileUsed += 2;
    }
    int count = denseGrid;
    if (numWall > 0) {
        int grid = std::min(kGridWall, (numWall + THREADS - 1)/THREADS);
        double* part = partialsDev + NPART*(size_t) count;
        dispatchStorage(storageType, [&](auto L) { decltype(L)::bounceBack(B, wallDev, numWall, view, part, grid, follow, stream); });
        CUDA_CHECK(cudaGetLastError());
        launches++;
        count += grid;
    }
    if (numBoundary > 0) {
        int grid = std::min(kGridSparse, (numBoundary + kBoundaryThreads - 1)/kBoundaryThreads);
        double* part = partialsDev + NPART*(size_t) count;
        // Face velocities and densities, and the boundary stress weight c (D3Q19.h:206-208), in a small table
        // that lives in the partials buffer tail (read-only for the kernel).
        dispatchStorage(storageType, [&](auto L) {
            decltype(L)::boundary(fluct, A, B, boundaryDev, numBoundary, view, remove ? 1 : 0, stepIndex, part,
                                  faceDev, grid, follow, stream);
        });
        CUDA_CHECK(cudaGetLastError());
        launches++;
        count += grid;
    }
    if (separate) {
        launch(follow, finishKernel, 1, THREADS, stream, partialsDev, count, view, 0);
        CUDA_CHECK(cudaGetLastError());
        launches++;
    }
    cur = 1-cur;
}

void FluidEngine::profileDense(bool enable) {
    profiling = enable;
    if (enable)
        profileUsed = 0;
}

void FluidEngine::denseTime(long long* launches, double* totalMs) {
    CUDA_CHECK(cudaStreamSynchronize(stream));
    double total = 0;
    for (size_t i = 0; i + 1 < profileUsed; i += 2) {
        float ms = 0;
        CUDA_CHECK(cudaEventElapsedTime(&ms, profileEvents[i], profileEvents[i+1]));
        total += ms;
    }
    *launches = (long long) (profileUsed/2);
    *totalMs = total;
}

void FluidEngine::momentsPass(bool setSums) {
    dispatchStorage(storageType, [&](auto L) { decltype(L)::moments(pop[cur], view, gridBlocks, stream); });
    CUDA_CHECK(cudaGetLastError());
    finishKernel<<<1, THREADS, 0, stream>>>(partialsDev, gridBlocks, view, setSums ? 1 : 2);
    CUDA_CHECK(cudaGetLastError());
    launches += 2;
}

double FluidEngine::steadyResidual(int interval) {
    bool first = residualPrevDev == nullptr;
    if (first)
        CUDA_CHECK(cudaMalloc(&residualPrevDev, sizeof(double)*3*(size_t) view.n));
    dispatchStorage(storageType, [&](auto L) {
        decltype(L)::residual(pop[cur], view, residualPrevDev, first ? 1 : 0, gridBlocks, stream);
    });
    CUDA_CHECK(cudaGetLastError());
    launches++;
    std::vector<double> partials((size_t) NPART*gridBlocks);
    CUDA_CHECK(cudaMemcpyAsync(partials.data(), partialsDev, sizeof(double)*partials.size(), cudaMemcpyDeviceToHost, stream));
    CUDA_CHECK(cudaStreamSynchronize(stream));
    double maxDiff2 = 0, maxU2 = 0;
    for (int b = 0; b < gridBlocks; b++) {
        maxDiff2 = std::max(maxDiff2, partials[(size_t) NPART*b]);
        maxU2 = std::max(maxU2, partials[(size_t) NPART*b + 7]);
    }
    if (first || maxU2 == 0)
        return HUGE_VAL;
    return std::sqrt(maxDiff2)/(interval*std::sqrt(maxU2));
}

void FluidEngine::restoreStats(const StepStats& stats) {
    statsHost = stats;
    CUDA_CHECK(cudaMemcpyAsync(statsDev, &statsHost, sizeof(StepStats), cudaMemcpyHostToDevice, stream));
    CUDA_CHECK(cudaStreamSynchronize(stream));
}

StepStats FluidEngine::readStats() {
    StepStats s;
    CUDA_CHECK(cudaMemcpyAsync(&s, statsDev, sizeof(StepStats), cudaMemcpyDeviceToHost, stream));
    CUDA_CHECK(cudaStreamSynchronize(stream));
    return s;
}

void FluidEngine::getState(double* host) {
    if (stagingDev == nullptr)
        CUDA_CHECK(cudaMalloc(&stagingDev, sizeof(double)*4*(size_t) view.n));
    // Four planes at a time, straight into the caller's array.
    for (int q0 = 0; q0 < 19; q0 += 4) {
        const int count = std::min(4, 19 - q0);
        for (int k = 0; k < count; k++)
            dispatchStorage(storageType, [&](auto L) {
                decltype(L)::gather(pop[cur], q0 + k, view, (double*) stagingDev + (size_t) k*view.n, stream);
            });
        CUDA_CHECK(cudaGetLastError());
        hostCopy->download({{host + (size_t) q0*view.n, stagingDev, sizeof(double)*(size_t) count*view.n}}, stream);
    }
}

void FluidEngine::getStateByDirection(const std::function<void(int, const double*)>& sink) {
    if (stagingDev == nullptr)
        CUDA_CHECK(cudaMalloc(&stagingDev, sizeof(double)*4*(size_t) view.n));
    std::vector<double> plane((size_t) view.n);
    for (int q = 0; q < 19; q++) {
        dispatchStorage(storageType, [&](auto L) { decltype(L)::gather(pop[cur], q, view, (double*) stagingDev, stream); });
        CUDA_CHECK(cudaGetLastError());
        CUDA_CHECK(cudaMemcpyAsync(plane.data(), stagingDev, sizeof(double)*view.n, cudaMemcpyDeviceToHost, stream));
        CUDA_CHECK(cudaStreamSynchronize(stream));
        sink(q, plane.data());
    }
}

void FluidEngine::setState(const double* host) {
    setStateByDirection([&](int q, double* values) {
        std::memcpy(values, host + (size_t) q*view.n, sizeof(double)*view.n);
    });
}

void FluidEngine::setStateByDirection(const std::function<void(int, double*)>& source) {
    if (stagingDev == nullptr)
        CUDA_CHECK(cudaMalloc(&stagingDev, sizeof(double)*4*(size_t) view.n));
    int* changedDev = reinterpret_cast<int*>(partialsDev);
    CUDA_CHECK(cudaMemsetAsync(changedDev, 0, sizeof(int), stream));
    std::vector<double> plane((size_t) view.n);
    for (int q = 0; q < 19; q++) {
        source(q, plane.data());
        CUDA_CHECK(cudaMemcpyAsync(stagingDev, plane.data(), sizeof(double)*view.n, cudaMemcpyHostToDevice, stream));
        dispatchStorage(storageType, [&](auto L) {
            decltype(L)::scatter(pop[cur], pop[1-cur], q, view, (const double*) stagingDev, changedDev, stream);
        });
        CUDA_CHECK(cudaGetLastError());
        CUDA_CHECK(cudaStreamSynchronize(stream));
    }
    int changed = 0;
    CUDA_CHECK(cudaMemcpy(&changed, changedDev, sizeof(int), cudaMemcpyDeviceToHost));
    if (changed)
        momentsPass(true);
    CUDA_CHECK(cudaStreamSynchronize(stream));
}

void FluidEngine::setEquilibrium(const double* density, const double* velocity, bool onDevice, double densityScale,
                                 double velocityScale, bool strain) {
    const double* rho = density;
    const double* u = velocity;
    if (!onDevice) {
        if (stagingDev == nullptr)
            CUDA_CHECK(cudaMalloc(&stagingDev, sizeof(double)*4*(size_t) view.n));
        double* staging = (double*) stagingDev;
        CUDA_CHECK(cudaMemcpyAsync(staging, density, sizeof(double)*view.n, cudaMemcpyHostToDevice, stream));
        CUDA_CHECK(cudaMemcpyAsync(staging + view.n, velocity, sizeof(double)*3*view.n, cudaMemcpyHostToDevice, stream));
        rho = staging;
        u = staging + view.n;
    }
    dispatchStorage(storageType, [&](auto L) {
        decltype(L)::equilibrium(pop[cur], pop[1-cur], view, rho, u, densityScale, velocityScale, strain ? 1 : 0, stream);
    });
    CUDA_CHECK(cudaGetLastError());
    launches++;
    momentsPass(true);
    CUDA_CHECK(cudaStreamSynchronize(stream));
}

void FluidEngine::fields(double* density, double* velocity, double densityScale, double velocityScale) {
    if (stagingDev == nullptr)
        CUDA_CHECK(cudaMalloc(&stagingDev, sizeof(double)*4*(size_t) view.n));
    double* rho = (double*) stagingDev;
    double* u = rho + view.n;
    dispatchStorage(storageType, [&](auto L) {
        decltype(L)::fields(pop[cur], view, rho, u, densityScale, velocityScale, stream);
    });
    CUDA_CHECK(cudaGetLastError());
    hostCopy->download({{density, rho, sizeof(double)*(size_t) view.n}, {velocity, u, 3*sizeof(double)*(size_t) view.n}},
                       stream);
}

void FluidEngine::copyStateOut(void* host) {
    CUDA_CHECK(cudaMemcpyAsync(host, pop[cur], stateBytes(), cudaMemcpyDeviceToHost, stream));
    CUDA_CHECK(cudaStreamSynchronize(stream));
}

void FluidEngine::copyStateIn(const void* host) {
    CUDA_CHECK(cudaMemcpyAsync(pop[cur], host, stateBytes(), cudaMemcpyHostToDevice, stream));
    CUDA_CHECK(cudaMemcpyAsync(pop[1-cur], pop[cur], stateBytes(), cudaMemcpyDeviceToDevice, stream));
    momentsPass(true);
    CUDA_CHECK(cudaStreamSynchronize(stream));
}

} // namespace lbm
