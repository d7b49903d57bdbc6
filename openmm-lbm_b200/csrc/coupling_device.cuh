// Device functions of the particle coupling, shared by the kernels of one lattice (coupling.cu) and of the replica
// batch (batch.cu): stencil weights and slots, the pulled moments of a node, the explicit drag of a particle and the
// reaction on the fluid, after the reference (platforms/reference/src/ReferenceLBMKernels.cpp:503-1018,
// openmmapi/include/internal/LBMStencils.h).
#pragma once

#include "fluid.cuh"
#include "lbm_device.cuh"
#include <cstring>
#include <type_traits>

namespace lbm {

// The coupling parameters in lattice units, by value to the kernels.
struct CouplingView {
    int np, width, slots, stencil;
    int nx, ny, nz;
    int open[3];
    long long n;
    int wordsPerRow;
    double dx, velocityScale, forceScale;
    double gamma, kT, h, a;
    double g[3];
    uint32_t seed;
    int randomForce;
    const uint32_t* solidMask;
    const double* mass;          // m/m_c per particle
};

// The coupling parameters in lattice units (ReferenceLBMKernels.cpp:520-525).
inline CouplingView makeCouplingView(const LbmLatticeParameters& l, const FluidView& f, int np, int width, const double* mass) {
    CouplingView c;
    std::memset(&c, 0, sizeof(c));
    c.np = np;
    c.width = width;
    c.slots = width*width*width;
    c.stencil = l.interpolation_stencil;
    c.nx = l.nx; c.ny = l.ny; c.nz = l.nz;
    for (int a = 0; a < 3; a++)
        c.open[a] = l.face_boundary[2*a] != LBM_BOUNDARY_PERIODIC;
    c.n = f.n;
    c.wordsPerRow = f.wordsPerRow;
    double cellMass = l.density*l.dx*l.dx*l.dx;
    c.dx = l.dx;
    c.velocityScale = l.dx/l.dt;
    c.forceScale = cellMass*l.dx/(l.dt*l.dt);
    c.gamma = l.friction*l.dt;
    c.kT = l.kT*l.dt*l.dt/(cellMass*l.dx*l.dx);
    c.h = 0.5;
    c.a = c.gamma*c.h;
    for (int a = 0; a < 3; a++)
        c.g[a] = l.body_acceleration[a];
    c.seed = (uint32_t) l.random_number_seed;
    c.randomForce = (c.kT > 0 && c.gamma > 0) ? 1 : 0;
    c.solidMask = f.solidMask;
    c.mass = mass;
    return c;
}

namespace {

template <typename R> struct Vec4;
template <> struct Vec4<float> {
    typedef float4 type;
    static __device__ __forceinline__ float4 make(float a, float b, float c, float d) { return make_float4(a, b, c, d); }
};
template <> struct Vec4<double> {
    typedef double4 type;
    static __device__ __forceinline__ double4 make(double a, double b, double c, double d) { return make_double4(a, b, c, d); }
};

// Loads of a slot's 4-vector through the read-only path (data of an earlier launch) or through L2 (data written by the
// same launch); double4 as two double2.
__device__ __forceinline__ float4 loadReadOnly(const float4* p) { return __ldg(p); }
__device__ __forceinline__ double4 loadReadOnly(const double4* p) {
    const double2 a = __ldg(reinterpret_cast<const double2*>(p)), b = __ldg(reinterpret_cast<const double2*>(p) + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float4 loadCoherent(const float4* p) { return __ldcg(p); }
__device__ __forceinline__ double4 loadCoherent(const double4* p) {
    const double2 a = __ldcg(reinterpret_cast<const double2*>(p)), b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}

// r[0..2] += (x, y, z): one vector atomic for float (sm_90 and later), three for double.
__device__ __forceinline__ void atomicAdd3(float* r, double x, double y, double z) {
    atomicAdd(reinterpret_cast<float4*>(r), make_float4((float) x, (float) y, (float) z, 0.0f));
}
__device__ __forceinline__ void atomicAdd3(double* r, double x, double y, double z) {
    atomicAdd(&r[0], x);
    atomicAdd(&r[1], y);
    atomicAdd(&r[2], z);
}

// Node indices are below 2^32 (the fluid checks it), so 32-bit division finds their rows.
__device__ __forceinline__ bool isSolid(const uint32_t* mask, int wordsPerRow, int nx, long long node) {
    if (mask == nullptr)
        return false;
    const unsigned row = (unsigned) node/(unsigned) nx;
    const int x = (int) ((unsigned) node - row*(unsigned) nx);
    return (__ldg(&mask[(size_t) row*wordsPerRow + x/32]) >> (x%32)) & 1u;
}

// Lattice coordinate of a position along an axis, wrapped into [0, n) (ReferenceLBMKernels.cpp:978-979).
__device__ __forceinline__ double latticeCoordinate(double x, double dx, int n) {
    double s = x/dx;
    s -= floor(s/n)*n;
    return s;
}

// LBMStencils::kernel (LBMStencils.h:42-62).
__device__ double stencilKernel1(int stencil, double r) {
    double s = fabs(r);
    switch (stencil) {
    case LBM_STENCIL_TRILINEAR:
        return (s < 1.0 ? 1.0-s : 0.0);
    case LBM_STENCIL_THREEPOINT:
        if (s <= 0.5)
            return (1.0 + sqrt(1.0-3.0*s*s))/3.0;
        if (s < 1.5)
            return (5.0 - 3.0*s - sqrt(fmax(0.0, 1.0-3.0*(1.0-s)*(1.0-s))))/6.0;
        return 0.0;
    case LBM_STENCIL_KEYS:
        if (s <= 1.0)
            return 1.0 - 2.5*s*s + 1.5*s*s*s;
        if (s < 2.0)
            return 2.0 - 4.0*s + 2.5*s*s - 0.5*s*s*s;
        return 0.0;
    default:
        return (r >= -0.5 && r < 0.5 ? 1.0 : 0.0);
    }
}

// Density deviation and momentum of the post-stream populations of a node (pulled from the input array).
template <typename T>
__device__ void pullMomentsAt(const T* A, const FluidView& f, int x, int y, int z, double& dr, double& jx, double& jy,
                              double& jz) {
    typedef typename std::conditional<std::is_same<T, double>::value, double, float>::type R;
    int xs[3] = {x == 0 ? f.nx-1 : x-1, x, x == f.nx-1 ? 0 : x+1};
    int ys[3] = {y == 0 ? f.ny-1 : y-1, y, y == f.ny-1 ? 0 : y+1};
    int zs[3] = {z == 0 ? f.nz-1 : z-1, z, z == f.nz-1 ? 0 : z+1};
    R d = 0, a = 0, b = 0, c = 0;
#pragma unroll
    for (int q = 0; q < 19; q++) {
        const int cx = cxOf(q), cy = cyOf(q), cz = czOf(q);
        long long src = xs[1-cx] + (long long) f.nx*(ys[1-cy] + (long long) f.ny*zs[1-cz]);
        R v = loadq<T, R>(A + (long long) q*f.n + src, q);
        d += v;
        a += cx*v;
        b += cy*v;
        c += cz*v;
    }
    dr = d; jx = a; jy = b; jz = c;
}

// Entry k = lane % 4 of axis lane/4 % 4 (the last group repeats axis 2) of particle i's stencil (LBMStencils::axisWeights,
// LBMStencils.h:73-95: clamped at open faces, repeated nodes merged into their first entry); lanes 12 and on of a group of
// 16 hold nothing of use.  Entries past the width: a negative index, weight 0.  Called by a whole warp.  COHERENT: the
// positions were written by the same launch.
template <bool COHERENT>
__device__ __forceinline__ void stencilEntry(const CouplingView& c, const double* __restrict__ pos, int i, int lane, int& index,
                                             double& weight) {
    const int axis = min((lane >> 2) & 3, 2), k = lane & 3;
    const int size = axis == 0 ? c.nx : (axis == 1 ? c.ny : c.nz);
    const double x = COHERENT ? __ldcg(&pos[3*i+axis]) : pos[3*i+axis];
    const double s = latticeCoordinate(x, c.dx, size);
    index = -1 - k;
    weight = 0.0;
    if (c.stencil == LBM_STENCIL_NEAREST) {
        if (k == 0) {
            index = ((int) floor(s + 0.5))%size;
            weight = 1.0;
        }
    }
    else if (k < c.width) {
        const int first = c.stencil == LBM_STENCIL_THREEPOINT ? (int) floor(s + 0.5) - 1
                        : (int) floor(s) - (c.stencil == LBM_STENCIL_KEYS ? 1 : 0);
        weight = stencilKernel1(c.stencil, s - (first + k));
        const int idx = first + k;
        const bool open = axis == 0 ? c.open[0] : (axis == 1 ? c.open[1] : c.open[2]);
        index = open ? min(max(idx, 0), size - 1) : ((idx%size) + size)%size;
    }
    // A node that the axis meets more than once keeps the sum of its weights in its first entry.
    double merged = weight;
    bool repeated = false;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const int other = __shfl_sync(0xffffffffu, index, (lane & ~3) + j);
        const double w = __shfl_sync(0xffffffffu, weight, (lane & ~3) + j);
        if (other == index && j < k)
            repeated = true;
        if (other == index && j > k)
            merged += w;
    }
    weight = repeated ? 0.0 : merged;
}

// The stencil slots t = i*slots + s of particle i by one warp: the node and weight of each slot (LBMStencils::axisWeights,
// LBMStencils.h:73-95) and u = j/rho of the node pulled from the populations (after the momentum removal, :539, :672; a
// solid node has rho = 0).  Lane 4 a + k < 12 forms entry k of axis a (stencilEntry), and each slot's lane takes its three
// entries by shuffles: a thread per slot formed all its particle's entries again, nine to twelve kernel values in double
// with their roots, for the three that it uses (47 us per step of 10,530 beads with the three-point stencil).  COHERENT:
// the positions were written by the same launch (a persistent kernel): they are read through L2.
template <typename T, typename R, bool COHERENT = false>
__device__ __forceinline__ void stencilParticle(const T* __restrict__ A, const FluidView& f, const CouplingView& c,
                                                const double* __restrict__ pos, int i, int lane, int remove,
                                                int* slotNode, R* slotWeight, typename Vec4<R>::type* slotU) {
    int index;
    double weight;
    stencilEntry<COHERENT>(c, pos, i, lane, index, weight);
    const long long t0 = (long long) i*c.slots;
    for (int s0 = 0; s0 < c.slots; s0 += 32) {
        const int slot = s0 + lane, at = min(slot, c.slots - 1);
        const int sub[3] = {at%c.width, (at/c.width)%c.width, at/(c.width*c.width)};
        int idx[3];
        double w = 1.0;
        for (int a = 0; a < 3; a++) {
            idx[a] = __shfl_sync(0xffffffffu, index, 4*a + sub[a]);
            w *= __shfl_sync(0xffffffffu, weight, 4*a + sub[a]);
        }
        if (slot >= c.slots)
            continue;
        const long long node = idx[0] + (long long) c.nx*(idx[1] + (long long) c.ny*idx[2]);
        double ux = 0, uy = 0, uz = 0, rho = 0;
        if (w != 0.0 && !isSolid(c.solidMask, c.wordsPerRow, c.nx, node)) {
            double dr, jx, jy, jz;
            pullMomentsAt<T>(A, f, idx[0], idx[1], idx[2], dr, jx, jy, jz);
            rho = 1.0 + dr;
            if (remove) {
                jx -= rho*f.stats->ucm[0];
                jy -= rho*f.stats->ucm[1];
                jz -= rho*f.stats->ucm[2];
            }
            ux = jx*(1.0/rho);
            uy = jy*(1.0/rho);
            uz = jz*(1.0/rho);
        }
        slotNode[t0 + slot] = (int) node;
        slotWeight[t0 + slot] = (R) w;
        slotU[t0 + slot] = Vec4<R>::make((R) ux, (R) uy, (R) uz, (R) rho);
    }
}

// The node and weight of stencil slot t, as stencilParticle (from the particle's axis indices and weights, computed once
// per particle by stencilAxesKernel), with the moments computed once per node: the first slot of a fluid node to claim it in
// this pass (nodeStamp[node] set to `stamp`) pulls the node's moments into nodeU[node]; stencilGatherSlot then copies
// them to every slot of the node.  The moments of a node are the same for all its slots, and overlapping stencils
// share most of their nodes.  With `mark` (the fluid's reaction mask, for the pass of a step) the claiming slot also
// flags the node and zeroes its reaction, once per node: every fluid node of a slot with a nonzero weight receives a
// reaction in this step, so the reactions are then added without touching the mask, and the end of a step clears the
// mask alone.
// W: the stencil width when it is known at compile time (the slot's particle and axis entries then come from
// divisions by constants), 0 for c.width.  The slots of all particles are fewer than 2^31.
template <typename T, typename R, int W = 0>
__device__ __forceinline__ void stencilClaimSlot(const T* __restrict__ A, const FluidView& f, const CouplingView& c,
                                                 const int4* __restrict__ axisIndex,
                                                 const double2* __restrict__ axisWeight, long long t, int remove,
                                                 int centred, int* slotNode, R* slotWeight, unsigned* nodeStamp,
                                                 unsigned stamp, typename Vec4<R>::type* nodeU, uint32_t* mark,
                                                 R* reaction) {
    const int width = W > 0 ? W : c.width, slots = W > 0 ? W*W*W : c.slots;
    const int i = (int) t/slots, s = (int) t - i*slots;
    const int sub[3] = {s%width, (s/width)%width, s/(width*width)};
    int idx[3];
    double w = 1.0;
    for (int a = 0; a < 3; a++) {
        const int4 ia = axisIndex[3*i + a];
        const double2 wa = axisWeight[6*i + 2*a + sub[a]/2];
        idx[a] = sub[a] == 0 ? ia.x : sub[a] == 1 ? ia.y : sub[a] == 2 ? ia.z : ia.w;
        w *= (sub[a] & 1) ? wa.y : wa.x;
    }
    long long node = idx[0] + (long long) c.nx*(idx[1] + (long long) c.ny*idx[2]);
    slotNode[t] = (int) node;
    slotWeight[t] = (R) w;
    if (w == 0.0)
        return;
    if (c.solidMask != nullptr) {
        const long long row = idx[1] + (long long) c.ny*idx[2];
        if ((__ldg(&c.solidMask[row*c.wordsPerRow + idx[0]/32]) >> (idx[0]%32)) & 1u)
            return;
    }
    if (atomicExch(&nodeStamp[node], stamp) != stamp) {
        double dr, jx, jy, jz;
        pullMomentsAt<T>(A, f, idx[0], idx[1], idx[2], dr, jx, jy, jz);
        double rho = 1.0 + dr;
        if (remove) {
            jx -= rho*f.stats->ucm[0];
            jy -= rho*f.stats->ucm[1];
            jz -= rho*f.stats->ucm[2];
        }
        if (centred) {
            jx += c.h*rho*c.g[0];
            jy += c.h*rho*c.g[1];
            jz += c.h*rho*c.g[2];
        }
        nodeU[node] = Vec4<R>::make((R) (jx*(1.0/rho)), (R) (jy*(1.0/rho)), (R) (jz*(1.0/rho)), (R) rho);
        if (mark != nullptr) {
            const size_t row = (size_t) idx[1] + (size_t) c.ny*idx[2];
            atomicOr(&mark[row*f.wordsPerRow + idx[0]/32], 1u << (idx[0]%32));
            // The node's reaction starts from zero (the last step's were left in place; only their flags were cleared).
            *reinterpret_cast<typename Vec4<R>::type*>(reaction + 4*node) = Vec4<R>::make(0, 0, 0, 0);
        }
    }
}

template <typename R>
// With `coef` (the coupling matrix's solve) it also stores w/rho of the slot (0 where rho is 0).
__device__ __forceinline__ void stencilGatherSlot(long long t, const int* __restrict__ slotNode,
                                                  const R* __restrict__ slotWeight, const unsigned* __restrict__ nodeStamp,
                                                  unsigned stamp, const typename Vec4<R>::type* __restrict__ nodeU,
                                                  typename Vec4<R>::type* slotU, R* coef) {
    const long long node = slotNode[t];
    const R weight = slotWeight[t];
    typename Vec4<R>::type u = Vec4<R>::make(0, 0, 0, 0);
    if (weight != (R) 0 && nodeStamp[node] == stamp)
        u = nodeU[node];
    slotU[t] = u;
    if (coef != nullptr) {
        const double w = (double) weight, rho = (double) u.w;
        coef[t] = (R) (rho > 0 ? w/rho : 0.0);
    }
}

// Reaction (fx, fy, fz) on a node: added into the fluid's reaction buffer and the node flagged in `mask` (nullptr: the
// stencil pass flagged it), or for a solid node counted as momentum given to the wall (applyReaction,
// ReferenceLBMKernels.cpp:959-971).
template <typename R>
__device__ void addReaction(const FluidView& f, const CouplingView& c, R* reaction, uint32_t* mask, double* wall,
                            long long node, double fx, double fy, double fz) {
    if (isSolid(c.solidMask, c.wordsPerRow, c.nx, node)) {
        atomicAdd(&wall[0], fx);
        atomicAdd(&wall[1], fy);
        atomicAdd(&wall[2], fz);
        return;
    }
    atomicAdd3(reaction + 4*node, fx, fy, fz);
    if (mask == nullptr)
        return;
    const unsigned row = (unsigned) node/(unsigned) f.nx;
    const int x = (int) ((unsigned) node - row*(unsigned) f.nx);
    uint32_t bit = 1u << (x%32);
    uint32_t* word = &mask[(size_t) row*f.wordsPerRow + x/32];
    if (!(*((volatile uint32_t*) word) & bit))
        atomicOr(word, bit);
}

// Three normals of particle i for step `step` (Philox, purpose 2), in double.
__device__ __forceinline__ void particleNoise(uint32_t seed, int i, long long step, double xi[3]) {
    philoxNormals<double, 3>(seed, PurposeParticle, i, step, xi);
}

__device__ __forceinline__ double warpSum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Explicit drag of particle i, nearest node or stencil (ReferenceLBMKernels.cpp:503-553, 643-697), by one warp (the
// lanes over the stencil slots): F = -gamma m (v - u) + sqrt(2 gamma m kT) xi with u interpolated over the stencil,
// written to fout; on a lattice step the reaction -w F goes to the stencil nodes.
template <typename R, bool COHERENT = false>
__device__ __forceinline__ void explicitParticle(const FluidView& f, const CouplingView& c, const double* vel,
                                                 const int* slotNode, const R* slotWeight,
                                                 const typename Vec4<R>::type* slotU, int i, int lane,
                                                 long long step, int isStep, double* fout, R* reaction, uint32_t* mask,
                                                 double* wall, const double* removal = nullptr) {
    // COHERENT: the slots and velocities were written by the same launch (a persistent kernel): loads through L2.
    // removal: the velocity that this step's momentum removal subtracts from every node, where the slots hold the
    // nodes' j/rho before the removal (the persistent batch step); (j - rho ucm)/rho = j/rho - ucm, so the fluid
    // velocity at the particle is sum w j/rho - ucm sum w over the fluid slots.
    typedef typename Vec4<R>::type V;
    auto slotU_ = [&](long long t) { if constexpr (COHERENT) return loadCoherent(slotU + t); else return loadReadOnly(slotU + t); };
    auto weight_ = [&](long long t) { if constexpr (COHERENT) return __ldcg(slotWeight + t); else return __ldg(slotWeight + t); };
    auto node_ = [&](long long t) { if constexpr (COHERENT) return __ldcg(slotNode + t); else return __ldg(slotNode + t); };
    auto vel_ = [&](int k) { if constexpr (COHERENT) return __ldcg(vel + k); else return __ldg(vel + k); };
    double u[3] = {0, 0, 0}, wsum = 0;
    for (int s = lane; s < c.slots; s += 32) {
        long long t = (long long) i*c.slots + s;
        V su = slotU_(t);
        if (su.w > 0) {
            double w = (double) weight_(t);
            u[0] += (double) su.x*w;
            u[1] += (double) su.y*w;
            u[2] += (double) su.z*w;
            wsum += w;
        }
    }
    for (int a = 0; a < 3; a++)
        u[a] = warpSum(u[a]);
    if (removal != nullptr) {
        wsum = warpSum(wsum);
        for (int a = 0; a < 3; a++)
            u[a] -= __ldcg(&removal[a])*wsum;
    }
    double m = c.mass[i];
    double xi[3] = {0, 0, 0};
    if (c.randomForce)
        particleNoise(c.seed, i, step, xi);
    double F[3];
    for (int a = 0; a < 3; a++) {
        double v = vel_(3*i+a)*(1.0/c.velocityScale);
        F[a] = (v - u[a])*(-c.gamma*m);
        if (c.randomForce)
            F[a] += xi[a]*sqrt(2.0*c.gamma*m*c.kT);
    }
    if (lane == 0)
        for (int a = 0; a < 3; a++)
            fout[3*i+a] = F[a]*c.forceScale;
    if (isStep)
        for (int s = lane; s < c.slots; s += 32) {
            long long t = (long long) i*c.slots + s;
            double w = (double) weight_(t);
            if (w != 0.0)
                addReaction<R>(f, c, reaction, mask, wall, node_(t), -w*F[0], -w*F[1], -w*F[2]);
        }
}

} // namespace
} // namespace lbm
