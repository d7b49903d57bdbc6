// The learned warm start's passes between the convolutions (include/lbm_b200_warmstart.h), on channels-last BF16 volumes
// [n][d][h][w][c] with 8 channels (16 bytes) per thread: pooling, upsampling into the concatenation with the skip, their
// gradients, the gradient through a layer's ReLU with its bias's, and the network's input.  They are bound by memory;
// each reads and writes every volume once, in the layout the convolutions use.  The library passes that they stand in for
// worked in planar order between layout copies.  Per training step on two 64 x 64 x 128 volumes: upsampling with the
// concatenation 43 us (262, and the copies around it), its gradients 37 us (140 and copies), the ReLU's and biases'
// gradients of 15 layers 132 us (980 in five passes), pooling 9 us (56), the input 5 us per mask (twelve launches).
#include "lbm_b200_warmstart.h"
#include "lbm_internal.h"
#include <cuda_bf16.h>
#include <algorithm>
#include <string>

namespace {

constexpr int kThreads = 256;

struct Row {
    int n, z, y;
};
__device__ __forceinline__ Row rowOf(unsigned row, int depth, int height) {
    Row r;
    r.y = (int) (row%(unsigned) height);
    row /= (unsigned) height;
    r.z = (int) (row%(unsigned) depth);
    r.n = (int) (row/(unsigned) depth);
    return r;
}

// The 16-byte word of channel group g of voxel (z, y, x).
__device__ __forceinline__ size_t wordAt(int n, int z, int y, int x, int D, int H, int W, int groups, int g) {
    return ((((size_t) n*D + z)*H + y)*W + x)*groups + g;
}

__device__ __forceinline__ void unpack(uint4 v, float (&f)[8]) {
    const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        f[2*i] = __uint_as_float(w[i] << 16);
        f[2*i+1] = __uint_as_float(w[i] & 0xFFFF0000u);
    }
}
__device__ __forceinline__ uint4 pack(const float (&f)[8]) {
    unsigned w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(f[2*i], f[2*i+1]);
        w[i] = *reinterpret_cast<const unsigned*>(&h);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Sums of 8 children in the order of the window (z, y, x), in float, rounded once.
__device__ __forceinline__ uint4 sumChildren(const uint4* __restrict__ v, int n, int z, int y, int x, int D, int H, int W,
                                             int groups, int g, float scale) {
    uint4 word[8];
#pragma unroll
    for (int i = 0; i < 8; i++)
        word[i] = __ldg(v + wordAt(n, 2*z + i/4, 2*y + i/2%2, 2*x + i%2, D, H, W, groups, g));
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 8; i++) {
        float f[8];
        unpack(word[i], f);
#pragma unroll
        for (int k = 0; k < 8; k++)
            s[k] += f[k];
    }
#pragma unroll
    for (int k = 0; k < 8; k++)
        s[k] *= scale;
    return pack(s);
}

// y [n][d][h][w] = mean of x's 2 x 2 x 2 windows; a block per row of y.
__global__ void __launch_bounds__(kThreads)
poolKernel(const uint4* __restrict__ x, uint4* __restrict__ y, int D, int H, int W, int groups) {
    const int d = D/2, h = H/2, w = W/2;
    const Row r = rowOf(blockIdx.x, d, h);
    for (int i = threadIdx.x; i < w*groups; i += blockDim.x) {
        const int xx = i/groups, g = i - xx*groups;
        y[(size_t) blockIdx.x*w*groups + i] = sumChildren(x, r.n, r.z, r.y, xx, D, H, W, groups, g, 0.125f);
    }
}

// The gradient of the pooling: dx = dy/8 in every window's voxels (D, H, W of dx, even or with an untouched last plane).
__global__ void __launch_bounds__(kThreads)
poolGradKernel(const uint4* __restrict__ dy, uint4* __restrict__ dx, int D, int H, int W, int groups) {
    const int d = D/2, h = H/2, w = W/2;
    const Row r = rowOf(blockIdx.x, d, h);
    for (int i = threadIdx.x; i < w*groups; i += blockDim.x) {
        const int xx = i/groups, g = i - xx*groups;
        float f[8];
        unpack(__ldg(dy + (size_t) blockIdx.x*w*groups + i), f);
#pragma unroll
        for (int k = 0; k < 8; k++)
            f[k] *= 0.125f;
        const uint4 v = pack(f);
#pragma unroll
        for (int c = 0; c < 8; c++)
            dx[wordAt(r.n, 2*r.z + c/4, 2*r.y + c/2%2, 2*xx + c%2, D, H, W, groups, g)] = v;
    }
}

// y = [nearest 2x upsampling of x, skip] along the channels; a block per row of y (D, H, W).
__global__ void __launch_bounds__(kThreads)
upsampleConcatKernel(const uint4* __restrict__ x, const uint4* __restrict__ skip, uint4* __restrict__ y, int D, int H, int W,
                     int groupsX, int groupsSkip) {
    const int groups = groupsX + groupsSkip;
    const Row r = rowOf(blockIdx.x, D, H);
    for (int i = threadIdx.x; i < W*groups; i += blockDim.x) {
        const int xx = i/groups, g = i - xx*groups;
        y[(size_t) blockIdx.x*W*groups + i] = g < groupsX
            ? __ldg(x + wordAt(r.n, r.z/2, r.y/2, xx/2, D/2, H/2, W/2, groupsX, g))
            : __ldg(skip + ((size_t) blockIdx.x*W + xx)*groupsSkip + (g - groupsX));
    }
}

// Its gradients: dx the sums of dy over the upsampled voxels, dskip the other channels; a block per row of dx.
__global__ void __launch_bounds__(kThreads)
upsampleConcatGradKernel(const uint4* __restrict__ dy, uint4* __restrict__ dx, uint4* __restrict__ dskip, int D, int H, int W,
                         int groupsX, int groupsSkip) {
    const int groups = groupsX + groupsSkip, d = D/2, h = H/2, w = W/2;
    const Row r = rowOf(blockIdx.x, d, h);
    for (int i = threadIdx.x; i < w*groupsX; i += blockDim.x) {
        const int xx = i/groupsX, g = i - xx*groupsX;
        dx[(size_t) blockIdx.x*w*groupsX + i] = sumChildren(dy, r.n, r.z, r.y, xx, D, H, W, groups, g, 1.0f);
    }
    for (int i = threadIdx.x; i < 4*W*groupsSkip; i += blockDim.x) {
        const int line = i/(W*groupsSkip), j = i - line*W*groupsSkip, xx = j/groupsSkip, g = j - xx*groupsSkip;
        const int z = 2*r.z + line/2, y = 2*r.y + line%2;
        dskip[wordAt(r.n, z, y, xx, D, H, W, groupsSkip, g)] = __ldg(dy + wordAt(r.n, z, y, xx, D, H, W, groups, groupsX + g));
    }
}

// The gradient of a layer's output before its ReLU, dy (y > 0) (y == nullptr: no ReLU, and out is not written), and its
// sums over the voxels: a thread keeps one channel group and adds up its voxels, a block its threads as a tree, and
// biasSumKernel the blocks, in their order, so that the sums are the same bits every time.  Bound by the volumes' bytes, read
// and written once.  592 blocks, two voxels of a thread in flight: 16 channels on two 64 x 64 x 128 volumes 15.0 us (18.6 with
// one voxel and FP32 atomics into zeroed sums; four in flight 5 us more than two, 1184 blocks 5 us more than 592), 160
// channels at 8 x 8 x 16 4.9 us (3.7).  A ticket, by which the last block adds the blocks' sums, costs more than the second
// launch does: 24.6 and 12.5 us.
constexpr int kBiasBlocks = 592, kBiasAhead = 2;

// Leaves in the rows of part 0 the sums of `parts` rows of `stride` elements, added as a tree (thread part*stride + i holds
// element i of a row, kThreads apart for each of the N sums).
template <int N>
__device__ __forceinline__ void treeSum(float* sums, int part, int parts, int stride) {
    for (int h = parts > 1 ? 1 << (31 - __clz(parts - 1)) : 0; h > 0; h /= 2) {
        __syncthreads();
        if (part < h && part + h < parts)
#pragma unroll
            for (int k = 0; k < N; k++)
                sums[k*kThreads + threadIdx.x] += sums[k*kThreads + threadIdx.x + h*stride];
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kThreads)
reluBiasGradKernel(const uint4* __restrict__ dy, const uint4* __restrict__ y, uint4* __restrict__ out,
                   float* __restrict__ partials, size_t voxels, int groups) {
    __shared__ float sums[8*kThreads];
    const int lanes = kThreads/groups;                    // voxels a block takes at a time
    const int g = threadIdx.x%groups, lane = threadIdx.x/groups, channels = 8*groups;
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const size_t step = (size_t) gridDim.x*lanes;
    if (lane < lanes)
        for (size_t v = (size_t) blockIdx.x*lanes + lane; v < voxels; v += kBiasAhead*step) {
            // The loads of several voxels in flight, then their sums in the voxels' order.
            uint4 word[kBiasAhead], act[kBiasAhead];
#pragma unroll
            for (int a = 0; a < kBiasAhead; a++)
                if (v + a*step < voxels) {
                    word[a] = __ldg(dy + (v + a*step)*groups + g);
                    if (y != nullptr)
                        act[a] = __ldg(y + (v + a*step)*groups + g);
                }
#pragma unroll
            for (int a = 0; a < kBiasAhead; a++)
                if (v + a*step < voxels) {
                    float f[8];
                    unpack(word[a], f);
                    if (y != nullptr) {
                        float on[8];
                        unpack(act[a], on);
#pragma unroll
                        for (int k = 0; k < 8; k++)
                            f[k] = on[k] > 0.0f ? f[k] : 0.0f*f[k];
                        out[(v + a*step)*groups + g] = pack(f);
                    }
#pragma unroll
                    for (int k = 0; k < 8; k++)
                        s[k] += f[k];
                }
        }
#pragma unroll
    for (int k = 0; k < 8; k++)
        sums[k*kThreads + threadIdx.x] = s[k];
    treeSum<8>(sums, lane, lanes, groups);
    for (int c = threadIdx.x; c < channels; c += kThreads)
        partials[(size_t) blockIdx.x*channels + c] = sums[(c%8)*kThreads + c/8];
}

// db = (or with `add` +=) the blocks' sums, of 8 channels per block, in their order.
__global__ void __launch_bounds__(kThreads)
biasSumKernel(const float* __restrict__ partials, int blocks, int channels, float* __restrict__ db, bool add) {
    __shared__ float sums[kThreads];
    const int c = blockIdx.x*8 + threadIdx.x%8, part = threadIdx.x/8;
    constexpr int parts = kThreads/8;
    float t[4] = {0, 0, 0, 0};
#pragma unroll 5
    for (int b = part; b < blocks; b += 4*parts)
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (b + j*parts < blocks)
                t[j] += __ldg(partials + (size_t) (b + j*parts)*channels + c);
    sums[threadIdx.x] = (t[0] + t[1]) + (t[2] + t[3]);
    treeSum<1>(sums, part, parts, 8);
    if (part == 0)
        db[c] = add ? db[c] + sums[threadIdx.x] : sums[threadIdx.x];
}

// The network's input for one mask: solid, scaled inlet and the coordinates along x, y, z, then zeros; 8 channels a voxel.
__global__ void __launch_bounds__(kThreads)
inputKernel(const unsigned char* __restrict__ mask, float inlet, const float* __restrict__ xs, const float* __restrict__ ys,
            const float* __restrict__ zs, uint4* __restrict__ out, int H, int W) {
    const float y = ys[blockIdx.x%(unsigned) H], z = zs[blockIdx.x/(unsigned) H];
    for (int x = threadIdx.x; x < W; x += blockDim.x) {
        const size_t v = (size_t) blockIdx.x*W + x;
        const float f[8] = {mask[v] ? 1.0f : 0.0f, inlet, xs[x], y, z, 0.0f, 0.0f, 0.0f};
        out[v] = pack(f);
    }
}

// The convolutions' weights as they read them: w16 the FP32 weights [cout][27][cin] in BF16, wt (where asked for) the
// flipped, transposed ones [cin][26 - tap][cout] of the input gradient.  A block takes 32 x 32 weights of a tap; the
// layers of a launch come in a table in its parameters.  Bound by launches, not by its bytes: the 15 layers of the network
// are one launch of 6 us, 9 us with the transposed ones (a cast per layer, and for the gradient a flip and a copy, were
// 43 launches and 180 us of the device, and 6 us each of the host).
constexpr int kLayers = 32, kTile = 32;
struct WeightTable {
    const float* w[kLayers];
    __nv_bfloat16* w16[kLayers];
    __nv_bfloat16* wt[kLayers];
    int cout[kLayers], cin[kLayers];
    unsigned first[kLayers + 1];       // blocks of the layers before
};

__global__ void __launch_bounds__(kThreads) weightsKernel(const __grid_constant__ WeightTable t) {
    __shared__ __nv_bfloat16 tile[kTile][kTile + 2];
    int layer = 0;
    while (blockIdx.x >= t.first[layer + 1])
        layer++;
    const int cout = t.cout[layer], cin = t.cin[layer], tilesI = (cin + kTile - 1)/kTile;
    unsigned r = blockIdx.x - t.first[layer];
    const int tap = (int) (r%27u);
    r /= 27u;
    const int i0 = (int) (r%(unsigned) tilesI)*kTile, o0 = (int) (r/(unsigned) tilesI)*kTile;
    const int lane = threadIdx.x%kTile, row = threadIdx.x/kTile;
    const float* w = t.w[layer];
    __nv_bfloat16 *w16 = t.w16[layer], *wt = t.wt[layer];
    constexpr int kRows = kThreads/kTile, kEach = kTile/kRows;
    const size_t at = ((size_t) (o0 + row)*27 + tap)*cin + i0 + lane, step = (size_t) kRows*27*cin;
    float v[kEach];
#pragma unroll
    for (int k = 0; k < kEach; k++)
        v[k] = o0 + row + k*kRows < cout && i0 + lane < cin ? __ldg(w + at + k*step) : 0.0f;
#pragma unroll
    for (int k = 0; k < kEach; k++)
        if (o0 + row + k*kRows < cout && i0 + lane < cin) {
            tile[row + k*kRows][lane] = __float2bfloat16_rn(v[k]);
            w16[at + k*step] = tile[row + k*kRows][lane];
        }
    if (wt == nullptr)
        return;
    __syncthreads();
    for (int i = row; i < kTile; i += kRows)
        if (i0 + i < cin && o0 + lane < cout)
            wt[((size_t) (i0 + i)*27 + 26 - tap)*cout + o0 + lane] = tile[lane][i];
}

LbmStatus invalid(const char* message) {
    lbm::setLastError(message);
    return LBM_ERR_INVALID_ARGUMENT;
}

LbmStatus launched(const char* name) {
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        return LBM_OK;
    lbm::setLastError(std::string(name) + ": " + cudaGetErrorString(e));
    return LBM_ERR_CUDA;
}

// A block per row: their number must fit a grid.
bool rowsFit(int batch, int depth, int height) {
    return batch > 0 && depth > 0 && height > 0 && (long long) batch*depth*height < (1LL << 31);
}

// Blocks of the bias gradient: two voxels per thread at least.
int biasBlocks(long long voxels, int channels) {
    const long long lanes = 2*(kThreads/(channels/8));
    return (int) std::min<long long>(kBiasBlocks, (voxels + lanes - 1)/lanes);
}

LbmStatus reluBiasGrad(const void* dy, const void* y, void* out, float* db, bool add, float* scratch, long long voxels,
                       int channels, cudaStream_t stream) {
    const int blocks = biasBlocks(voxels, channels);
    reluBiasGradKernel<<<(unsigned) blocks, kThreads, 0, stream>>>((const uint4*) dy, (const uint4*) y, (uint4*) out, scratch,
                                                                   (size_t) voxels, channels/8);
    biasSumKernel<<<(unsigned) (channels/8), kThreads, 0, stream>>>(scratch, blocks, channels, db, add);
    return launched("lbm_net_relu_bias_grad");
}

} // namespace

extern "C" {

LbmStatus lbm_net_pool(const void* x, void* y, int batch, int depth, int height, int width, int channels, void* stream) {
    if (!x || !y || channels <= 0 || channels%8 != 0 || !rowsFit(batch, depth/2, height/2) || width < 2)
        return invalid("lbm_net_pool: null pointer, empty volume or channels not a multiple of 8");
    poolKernel<<<(unsigned) (batch*(depth/2)*(height/2)), kThreads, 0, (cudaStream_t) stream>>>(
        (const uint4*) x, (uint4*) y, depth, height, width, channels/8);
    return launched("lbm_net_pool");
}

LbmStatus lbm_net_pool_grad(const void* dy, void* dx, int batch, int depth, int height, int width, int channels, void* stream) {
    if (!dy || !dx || channels <= 0 || channels%8 != 0 || !rowsFit(batch, depth/2, height/2) || width < 2)
        return invalid("lbm_net_pool_grad: null pointer, empty volume or channels not a multiple of 8");
    poolGradKernel<<<(unsigned) (batch*(depth/2)*(height/2)), kThreads, 0, (cudaStream_t) stream>>>(
        (const uint4*) dy, (uint4*) dx, depth, height, width, channels/8);
    return launched("lbm_net_pool_grad");
}

LbmStatus lbm_net_upsample_concat(const void* x, const void* skip, void* y, int batch, int depth, int height, int width,
                                  int channels, int skip_channels, void* stream) {
    if (!x || !skip || !y || channels <= 0 || channels%8 != 0 || skip_channels <= 0 || skip_channels%8 != 0 ||
        !rowsFit(batch, depth, height) || width <= 0 || depth%2 != 0 || height%2 != 0 || width%2 != 0)
        return invalid("lbm_net_upsample_concat: null pointer, odd or empty volume or channels not a multiple of 8");
    upsampleConcatKernel<<<(unsigned) (batch*depth*height), kThreads, 0, (cudaStream_t) stream>>>(
        (const uint4*) x, (const uint4*) skip, (uint4*) y, depth, height, width, channels/8, skip_channels/8);
    return launched("lbm_net_upsample_concat");
}

LbmStatus lbm_net_upsample_concat_grad(const void* dy, void* dx, void* dskip, int batch, int depth, int height, int width,
                                       int channels, int skip_channels, void* stream) {
    if (!dy || !dx || !dskip || channels <= 0 || channels%8 != 0 || skip_channels <= 0 || skip_channels%8 != 0 ||
        !rowsFit(batch, depth, height) || width <= 0 || depth%2 != 0 || height%2 != 0 || width%2 != 0)
        return invalid("lbm_net_upsample_concat_grad: null pointer, odd or empty volume or channels not a multiple of 8");
    upsampleConcatGradKernel<<<(unsigned) (batch*(depth/2)*(height/2)), kThreads, 0, (cudaStream_t) stream>>>(
        (const uint4*) dy, (uint4*) dx, (uint4*) dskip, depth, height, width, channels/8, skip_channels/8);
    return launched("lbm_net_upsample_concat_grad");
}

size_t lbm_net_relu_bias_scratch(long long voxels, int channels) {
    if (voxels <= 0 || channels <= 0 || channels%8 != 0 || channels > 8*kThreads)
        return 0;
    return sizeof(float)*(size_t) biasBlocks(voxels, channels)*channels;
}

LbmStatus lbm_net_relu_bias_grad_with(const void* dy, const void* y, void* out, float* db, float* scratch, long long voxels,
                                      int channels, void* stream) {
    if (!dy || !db || !scratch || (y && !out) || lbm_net_relu_bias_scratch(voxels, channels) == 0)
        return invalid("lbm_net_relu_bias_grad_with: null pointer, empty volume or channels not a multiple of 8");
    return reluBiasGrad(dy, y, out, db, false, scratch, voxels, channels, (cudaStream_t) stream);
}

LbmStatus lbm_net_relu_bias_grad(const void* dy, const void* y, void* out, float* db, long long voxels, int channels,
                                 void* stream) {
    const size_t bytes = lbm_net_relu_bias_scratch(voxels, channels);
    if (!dy || !db || (y && !out) || bytes == 0)
        return invalid("lbm_net_relu_bias_grad: null pointer, empty volume or channels not a multiple of 8");
    float* scratch = nullptr;
    const cudaError_t e = cudaMallocAsync((void**) &scratch, bytes, (cudaStream_t) stream);
    if (e != cudaSuccess) {
        lbm::setLastError(std::string("lbm_net_relu_bias_grad: ") + cudaGetErrorString(e));
        return LBM_ERR_CUDA;
    }
    const LbmStatus status = reluBiasGrad(dy, y, out, db, true, scratch, voxels, channels, (cudaStream_t) stream);
    cudaFreeAsync(scratch, (cudaStream_t) stream);
    return status;
}

LbmStatus lbm_net_input(const void* mask, float inlet, const float* xs, const float* ys, const float* zs, void* out,
                        int depth, int height, int width, void* stream) {
    if (!mask || !xs || !ys || !zs || !out || !rowsFit(1, depth, height) || width <= 0)
        return invalid("lbm_net_input: null pointer or empty volume");
    inputKernel<<<(unsigned) (depth*height), kThreads, 0, (cudaStream_t) stream>>>((const unsigned char*) mask, inlet, xs, ys,
                                                                                  zs, (uint4*) out, height, width);
    return launched("lbm_net_input");
}

LbmStatus lbm_net_weights(int layers, const float* const* w, void* const* w16, void* const* wt, const int* cout,
                          const int* cin, void* stream) {
    if (layers <= 0 || !w || !w16 || !wt || !cout || !cin)
        return invalid("lbm_net_weights: null pointer or no layers");
    for (int i = 0; i < layers; i++)
        if (!w[i] || !w16[i] || cout[i] <= 0 || cin[i] <= 0)
            return invalid("lbm_net_weights: null pointer or empty layer");
    for (int done = 0; done < layers; done += kLayers) {
        WeightTable t{};
        const int count = std::min(kLayers, layers - done);
        long long blocks = 0;
        for (int i = 0; i < count; i++) {
            t.w[i] = w[done + i];
            t.w16[i] = (__nv_bfloat16*) w16[done + i];
            t.wt[i] = (__nv_bfloat16*) wt[done + i];
            t.cout[i] = cout[done + i];
            t.cin[i] = cin[done + i];
            t.first[i] = (unsigned) blocks;
            blocks += 27LL*((t.cout[i] + kTile - 1LL)/kTile)*((t.cin[i] + kTile - 1LL)/kTile);
            if (blocks > 0x7FFFFFFFLL)
                return invalid("lbm_net_weights: too many weights");
        }
        t.first[count] = (unsigned) blocks;
        weightsKernel<<<(unsigned) blocks, kThreads, 0, (cudaStream_t) stream>>>(t);
        const LbmStatus status = launched("lbm_net_weights");
        if (status != LBM_OK)
            return status;
    }
    return LBM_OK;
}

} // extern "C"
