// pct_unet.cu -- learned DROP initializer: a 3-D convolutional encoder-decoder in bf16 on the
// tensor cores (tcgen05, fp32 accumulation in TMEM), with its own training kernels.
//
// The reference has no learned component; this is the engine's option to replace the FBP start
// x_0 = FBP_median x hull (define_initial_iterate, B.cu:8582-8646) by a network's estimate of the
// converged DROP image.  The FBP start stays the fallback.
//
// Network (4 levels, 16 -> 128 channels, 3x3x3 kernels, padding 1, ReLU):
//   encoder  L0: 16 -> 16 -> 16   avg-pool 2  L1: 16 -> 32 -> 32   pool  L2: 32 -> 64 -> 64
//            pool  L3: 64 -> 128 -> 128
//   decoder  nearest x2 up, conv to the level's width, + the encoder output of that level, ReLU,
//            conv, ReLU: L2 128 -> 64 -> 64, L1 64 -> 32 -> 32, L0 32 -> 16 -> 16
//   output   conv 16 -> 1 (channel 0 of a 16-wide conv whose other weights stay zero);
//            image = x_0 + (hull ? output : 0), so an untrained (zero) output layer gives back x_0.
//   input    channels-last bf16, channel 0 = x_0, channel 1 = hull, channels 2..15 = 0.
// Activations are channels-last bf16 [slice][row][column][channel] in the reference voxel order.
// Grids must have COLUMNS, ROWS and SLICES divisible by 8.
//
// Kernels:
//  * conv3_slab_kernel: implicit GEMM over patches of 128 positions, all 27 taps read from one copy of
//    the input slices in shared memory, accumulators of consecutive output slices side by side in TMEM.
//    The same kernel computes the data gradient with the flipped, transposed weights
//    W'[ci][26-t][co] = W[co][t][ci].  Epilogue: bias, residual, ReLU, ReLU-mask (for gradients), bf16
//    store; or the image output.
//  * conv3_wgrad_slab_kernel: dW[co][t][ci] = sum_v dZ[v][co] X[v + t][ci]: M = taps in y and input
//    channels, N = taps in z and output channels, K = voxels; partial sums are added with atomics.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "pct_api.h"
#include "pct_context.h"
#include "pct_tc.cuh"

namespace pct {
namespace unet {

using bf16 = __nv_bfloat16;
constexpr int kSmemPerSm = 233472;  // shared memory per SM on sm_100
constexpr int kTmemColumns = 512;   // TMEM columns per SM

__device__ __forceinline__ uint32_t pack_bf16(float a, float b)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ void unpack8(const uint4& u, float* f)
{
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 t = __bfloat1622float2(h[i]);
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
    }
}

// ----------------------------------------------------------------------------- convolutions --

struct ConvFwdArgs {
    const bf16* in;      // [nz>>up][ny>>up][nx>>up][cin]
    int cin, up;
    const bf16* weight;  // [cout][27][cin]
    int cout;
    int nx, ny, nz;      // output grid (= the input grid after the optional x2 upsampling)
    const float* bias;   // [cout] or null
    const bf16* residual;  // [V][cout] or null: added before the ReLU
    const bf16* mask;      // [V][cout] or null: output zeroed where mask <= 0
    int relu;
    bf16* out;             // [V][cout]
    const float* base;     // image mode: image[v] = base[v] + (hull[v] ? acc0 + bias0 : 0)
    const uint8_t* hull;
    float* image;
    int* status;           // set to 1 when a bounded wait expired
    int overlap;           // launched as a programmatic dependent of the kernel before it in the stream
};

// Epilogue of a forward / data-gradient convolution for 16 channels from c0 on: this thread's TMEM lane
// (row) holds voxel v's accumulators; whole warps call it (tcgen05.ld is warp-collective).  What it
// adds and masks with is requested before the wait for the accumulators.
struct EpilogueInputs {
    uint4 r[2], m[2];
};
__device__ __forceinline__ EpilogueInputs epilogue_request(const ConvFwdArgs& p, long long v, int c0, bool row_ok)
{
    EpilogueInputs e{};
    const size_t o = static_cast<size_t>(v) * p.cout + c0;
    if (p.residual && row_ok) {
        e.r[0] = reinterpret_cast<const uint4*>(p.residual + o)[0];
        e.r[1] = reinterpret_cast<const uint4*>(p.residual + o)[1];
    }
    if (p.mask && row_ok) {
        e.m[0] = reinterpret_cast<const uint4*>(p.mask + o)[0];
        e.m[1] = reinterpret_cast<const uint4*>(p.mask + o)[1];
    }
    return e;
}
__device__ __forceinline__ void conv_epilogue(const ConvFwdArgs& p, uint32_t trow, long long v, int c0, bool row_ok,
                                              const EpilogueInputs& e, const float* bias)
{
    float acc[16];
    tc::tmem_load16(trow, acc);
    if (!row_ok) return;
    if (p.image) {
        const float o = acc[0] + (p.bias ? bias[0] : 0.f);
        p.image[v] = p.base[v] + (p.hull[v] ? o : 0.f);
        return;
    }
    if (p.bias) {
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] += bias[i];
    }
    if (p.residual) {
        float r[16];
        unpack8(e.r[0], r);
        unpack8(e.r[1], r + 8);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] += r[i];
    }
    if (p.relu) {
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = fmaxf(acc[i], 0.f);
    }
    if (p.mask) {
        float m[16];
        unpack8(e.m[0], m);
        unpack8(e.m[1], m + 8);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = m[i] > 0.f ? acc[i] : 0.f;
    }
    uint4 w0, w1;
    w0.x = pack_bf16(acc[0], acc[1]);
    w0.y = pack_bf16(acc[2], acc[3]);
    w0.z = pack_bf16(acc[4], acc[5]);
    w0.w = pack_bf16(acc[6], acc[7]);
    w1.x = pack_bf16(acc[8], acc[9]);
    w1.y = pack_bf16(acc[10], acc[11]);
    w1.z = pack_bf16(acc[12], acc[13]);
    w1.w = pack_bf16(acc[14], acc[15]);
    uint4* out = reinterpret_cast<uint4*>(p.out + static_cast<size_t>(v) * p.cout + c0);
    out[0] = w0;
    out[1] = w1;
}

// ---- slab convolution -------------------------------------------------------------------------
// One CTA computes nc output channels of a patch of W x H voxels over a run of zt slices.  It keeps the
// 27 taps' weights for its channels in shared memory and streams the run's input slices, each with its
// one-voxel halo, through a ring; every slice is brought from L2 once per CTA instead of once per tap.
//
// In shared memory a slice is [channels / 8][position][8 channels], positions being the patch with its
// halo in rows of W + 2.  In the no-swizzle K-major layout eight consecutive rows of 16 bytes are a
// core matrix, and here every position is a row, so a tap (dy, dx) is the same matrix from a start
// address (dy (W + 2) + dx) 16 bytes further: all nine taps of a slice read one copy.  The M = 128 rows
// of an MMA are 128 consecutive positions from there; the rows of the halo columns come out unused.
//
// The three taps in z are the N side: the weights of dz = +1, 0, -1 lie one below the other, and the
// accumulators of consecutive output slices in consecutive TMEM columns, so one MMA of N = 3 nc adds
// an input slice to the three output slices that it reaches.  For every output the products are added
// in the order of the taps 0 to 26 and channels ascending.
//
// What bounds it is shared memory: an MMA of N = 48 reads 5.5 KB for 128 x 48 x 16 products, 44 of its
// 54 cycles.  One pass over 200x200x32 takes, in us (the kernels that brought every tap's inputs
// apart, by TMA or by threads for an upsampled input, in brackets): 16 to 16 channels 50 (263), 32 to 16
// upsampled with a skip 98 (466); 100x100x16, 32 to 32 27, 64 to 32 upsampled 39; 50x50x8, 64 to 64 20;
// 25x25x4, 128 to 128 20.  The network's forward pass 0.55 ms (2.04).
//
// Four warps bring the slices (cp.async, zero fill outside the grid, indices halved for an upsampled
// input), `ahead` of them in flight; one thread of the fifth issues the MMAs; four more write each
// output slice as soon as its last input slice is done.  A CTA keeps its weights and goes on with every
// gridDim.x-th tile (patch and run); with two accumulator stages the MMAs of a tile run while the
// previous tile is written.
constexpr int kSlabProducers = 128;
constexpr int kSlabThreads = kSlabProducers + 32 + 128;  // 416 with a second group of writers: one CTA per SM fewer
constexpr int kSlabMaxRing = 6;
constexpr int kSlabMaxSlices = 32;
constexpr int kSlabMaxPositions = 512;
constexpr int kSlabSmemLimit = 224 * 1024;  // dynamic; the per-block maximum (227 KB) also holds the static part
constexpr int kSlabSlack = 4096 + 128;       // what unused rows read past the last plane, and the alignment

struct SlabShape {
    int W, H, tiles_x, tiles_y;  // patch and patches
    int tiles, ctas;             // patches x runs; CTAs that share them
    int nc, nc_log2, zt;         // channels and slices of a tile
    int stages;                  // accumulator stages, 1 or 2
    int ring, ahead;             // input slices in shared memory, requested before the first is awaited
    int positions;               // (W + 2) (H + 2)
    int chunk_bytes;             // one 8-channel plane of a slice
    int slice_bytes, weight_bytes, smem;
    unsigned columns;            // TMEM
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool fill)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(fill ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A tile: its patch corner, output slices [z0, z1) and input slices [zi0, zi1).
struct SlabTile {
    int x0, y0, z0, z1, zi0, zi1;
};
__device__ __forceinline__ SlabTile slab_tile(const SlabShape& sh, int tile, int nz)
{
    const int patches = sh.tiles_x * sh.tiles_y;
    const int run = tile / patches, patch = tile - run * patches;
    const int py = patch / sh.tiles_x;
    SlabTile t;
    t.x0 = (patch - py * sh.tiles_x) * sh.W;
    t.y0 = py * sh.H;
    t.z0 = run * sh.zt;
    t.z1 = t.z0 + sh.zt < nz ? t.z0 + sh.zt : nz;
    t.zi0 = t.z0 > 0 ? t.z0 - 1 : 0;
    t.zi1 = t.z1 < nz ? t.z1 + 1 : nz;
    return t;
}

template <int kCin>
__global__ void __launch_bounds__(kSlabThreads) conv3_slab_kernel(const __grid_constant__ ConvFwdArgs p,
                                                                  const __grid_constant__ SlabShape sh)
{
    constexpr int kc = kCin / 8, kcl = kc == 2 ? 1 : kc == 4 ? 2 : kc == 8 ? 3 : 4;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[kSlabMaxRing];
    __shared__ __align__(8) uint64_t empty[kSlabMaxRing];
    __shared__ __align__(8) uint64_t ready[2 * kSlabMaxSlices];  // output slices of a stage
    __shared__ __align__(8) uint64_t drained[2];                 // stages written out
    __shared__ __align__(8) uint64_t weighed;                    // weights in place
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    __shared__ float bias[64];
    __shared__ uint32_t corner[kSlabMaxPositions];  // y << 16 | x of a position within the patch and its halo
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t base = (tc::smem_addr(smem_raw) + 127u) & ~127u;
    const uint32_t weights = base + sh.ring * sh.slice_bytes;
    const int pitch = sh.W + 2;
    const int c_first = blockIdx.y * sh.nc;

    if (warp == 4) tc::tmem_alloc(tc::smem_addr(&tmem_slot), sh.columns);
    if (tid < kSlabMaxRing) {
        tc::mbar_init(tc::smem_addr(&full[tid]), 4);
        tc::mbar_init(tc::smem_addr(&empty[tid]), 1);
    }
    if (tid < 2 * kSlabMaxSlices) tc::mbar_init(tc::smem_addr(&ready[tid]), 1);
    if (tid < 2) tc::mbar_init(tc::smem_addr(&drained[tid]), 4);
    if (tid == 2) tc::mbar_init(tc::smem_addr(&weighed), (kSlabThreads - kSlabProducers) / 32);
    if (tid < 2 * kSlabMaxSlices) tc::mbar_init_fence();
    if (tid == 0) failed = 0;
    if (p.bias && tid < sh.nc) bias[tid] = p.bias[c_first + tid];
    for (int q = tid; q < sh.positions; q += kSlabThreads) {
        const int yy = q / pitch;
        corner[q] = static_cast<uint32_t>(yy) << 16 | static_cast<uint32_t>(q - yy * pitch);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;
    if (tid >= kSlabProducers) {
        // weights [cout][27][cin] -> [tap of the slice][channels / 8][dz = 2, 1, 0][nc][8 channels]
        for (int u = tid - kSlabProducers; u < 27 * sh.nc << kcl; u += kSlabThreads - kSlabProducers) {
            const int c = u & (kc - 1), w = u >> kcl;
            const int co = w & (sh.nc - 1), tap = w >> sh.nc_log2;  // tap: 3 (tap of the slice) + (2 - dz)
            const int t = tap / 3, r = tap - 3 * t;
            cp_async16(weights + ((((t << kcl) + c) * 3 + r) * sh.nc + co) * 16,
                       p.weight + (static_cast<size_t>(c_first + co) * 27 + (2 - r) * 9 + t) * kCin + c * 8, true);
        }
        cp_async_commit();
    }
    // What follows reads what the kernels before wrote; the weights are written by no kernel of a pass.
    // The next kernel may start once every CTA is here: by then all earlier ones have ended.
    grid_dependency_wait();
    allow_dependent_launch();
    auto weights_here = [&]() {
        cp_async_wait<0>();
        tc::fence_proxy_async();
        __syncwarp();
        if ((tid & 31) == 0) tc::mbar_arrive(tc::smem_addr(&weighed));
    };

    if (warp < 4) {
        // One commit group per slice.  A slice is announced when `ahead` more have been requested, or at
        // once when there is no free slot to request into: the slot may become free only by the MMAs of
        // what is to be announced.
        const int sx = p.nx >> p.up, sy = p.ny >> p.up;
        const int units = sh.positions << kcl;
        bool ok = true;
        int slot = 0, round = 0, told = 0, pending = 0;
        auto announce = [&](int keep) {
            if (keep == 0) cp_async_wait<0>();
            else if (keep == 1) cp_async_wait<1>();
            else cp_async_wait<2>();
            tc::fence_proxy_async();
            __syncwarp();
            for (; pending > keep; --pending) {
                if ((tid & 31) == 0) tc::mbar_arrive(tc::smem_addr(&full[told]));
                if (++told == sh.ring) told = 0;
            }
        };
        for (int tile = blockIdx.x; tile < sh.tiles && ok; tile += sh.ctas) {
            const SlabTile t = slab_tile(sh, tile, p.nz);
            for (int zi = t.zi0; zi < t.zi1 && ok; ++zi) {
                if (round > 0 && !__all_sync(0xffffffffu, tc::mbar_test(tc::smem_addr(&empty[slot]), (round - 1) & 1))) {
                    if (pending > 0) announce(0);
                    ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&empty[slot]), (round - 1) & 1));
                    if (!ok) break;
                }
                const bf16* plane = p.in + static_cast<size_t>(zi >> p.up) * sy * sx * kCin;
                const uint32_t dst = base + slot * sh.slice_bytes;
                for (int u = tid; u < units; u += kSlabProducers) {
                    const int q = u >> kcl, c = u & (kc - 1);
                    const uint32_t at = corner[q];
                    const int y = t.y0 + static_cast<int>(at >> 16) - 1, x = t.x0 + static_cast<int>(at & 0xffffu) - 1;
                    const bool inside = static_cast<unsigned>(x) < static_cast<unsigned>(p.nx) &&
                                        static_cast<unsigned>(y) < static_cast<unsigned>(p.ny);
                    const int from = inside ? (y >> p.up) * sx + (x >> p.up) : 0;
                    cp_async16(dst + c * sh.chunk_bytes + q * 16, plane + static_cast<size_t>(from) * kCin + c * 8, inside);
                }
                if (++slot == sh.ring) {
                    slot = 0;
                    ++round;
                }
                cp_async_commit();
                if (++pending > sh.ahead) announce(sh.ahead);
            }
        }
        announce(0);
        if (!ok) failed = 1;
    } else if (warp == 4) {
        constexpr int ksteps = kCin / 16;
        const uint32_t leader = tc::elect_one();
        const uint32_t rows = 3u * sh.nc;
        const uint32_t a_step = 2 * (sh.chunk_bytes >> 4), b_step = 2 * rows;
        const uint64_t a_base = tc::smem_desc(base, sh.chunk_bytes, 128), b_base = tc::smem_desc(weights, rows * 16, 128);
        const uint32_t a_hi = static_cast<uint32_t>(a_base >> 32), b_hi = static_cast<uint32_t>(b_base >> 32);
        weights_here();
        bool ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&weighed), 0));
        int slot = 0, phase = 0, k = 0;
        for (int tile = blockIdx.x; tile < sh.tiles && ok; tile += sh.ctas, ++k) {
            const SlabTile t = slab_tile(sh, tile, p.nz);
            const int stage = sh.stages == 2 ? k & 1 : 0, use = sh.stages == 2 ? k >> 1 : k;
            if (use > 0) {
                ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&drained[stage]), (use - 1) & 1));
                tc::fence_after_sync();
            }
            const uint32_t acc = tmem + stage * sh.zt * sh.nc;
            const uint32_t done = tc::smem_addr(ready + stage * kSlabMaxSlices);
            int reached = t.z0 - 1;  // last output slice that has a product
            for (int zi = t.zi0; zi < t.zi1 && ok; ++zi) {
                ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&full[slot]), phase));
                if (!ok) break;
                tc::fence_after_sync();
                const int lo = zi - 1 > t.z0 ? zi - 1 : t.z0, hi = zi + 1 < t.z1 ? zi + 1 : t.z1 - 1;  // reached by it
                const uint32_t a0 = static_cast<uint32_t>(a_base) + slot * (sh.slice_bytes >> 4);
                const uint32_t b0 = static_cast<uint32_t>(b_base) + (lo - (zi - 1)) * sh.nc;
                const uint32_t d = acc + (lo - t.z0) * sh.nc;
                const uint32_t idesc = tc::idesc_bf16_f32((hi - lo + 1) * sh.nc, false);
                if (hi > reached) {
                    // output slices without a product yet start here: the first MMA in two parts
                    if (reached >= lo)
                        tc::mma_bf16_warp(d, a0, a_hi, b0, b_hi, tc::idesc_bf16_f32((reached - lo + 1) * sh.nc, false), 1, leader);
                    const int fresh = reached >= lo ? reached + 1 - lo : 0;
                    tc::mma_bf16_warp(d + fresh * sh.nc, a0, a_hi, b0 + fresh * sh.nc, b_hi,
                                      tc::idesc_bf16_f32((hi - lo + 1 - fresh) * sh.nc, false), 0, leader);
                } else {
                    tc::mma_bf16_warp(d, a0, a_hi, b0, b_hi, idesc, 1, leader);
                }
#pragma unroll
                for (int i = 1; i < 9 * ksteps; ++i) {  // tap i / ksteps, channels 16 (i % ksteps) and on
                    const int tap = i / ksteps;
                    tc::mma_bf16_warp(d, a0 + (tap / 3 * pitch + tap % 3) + (i % ksteps) * a_step, a_hi, b0 + i * b_step, b_hi,
                                      idesc, 1, leader);
                }
                reached = hi;
                // an output slice is complete after the input slice above it, or the grid's last
                tc::mma_commit_warp(tc::smem_addr(&empty[slot]), leader);
                if (zi > t.z0) tc::mma_commit_warp(done + 8 * (zi - 1 - t.z0), leader);
                if (zi + 1 == p.nz) tc::mma_commit_warp(done + 8 * (zi - t.z0), leader);
                if (++slot == sh.ring) {
                    slot = 0;
                    phase ^= 1;
                }
            }
        }
        if (!ok) failed = 1;
    } else {
        // row m of the MMAs is TMEM lane m; a warp reads the lanes 32 (warp % 4) and on
        const int m = (warp & 3) * 32 + (tid & 31);
        const int yy = m / pitch, xx = m - yy * pitch;
        const uint32_t lane = tmem + (static_cast<uint32_t>(warp & 3) * 32u << 16);
        const long long plane = static_cast<long long>(p.nx) * p.ny;
        weights_here();
        bool ok = true;
        int k = 0;
        for (int tile = blockIdx.x; tile < sh.tiles && ok; tile += sh.ctas, ++k) {
            const SlabTile t = slab_tile(sh, tile, p.nz);
            const int stage = sh.stages == 2 ? k & 1 : 0, use = sh.stages == 2 ? k >> 1 : k;
            const uint32_t acc = lane + stage * sh.zt * sh.nc;
            const int x = t.x0 + xx, y = t.y0 + yy;
            const bool row_ok = xx < sh.W && yy < sh.H && x < p.nx && y < p.ny;
            // a piece is 16 channels of a slice; the next piece's inputs are requested before this one is written
            int z = t.z0, c = 0;
            long long v = (static_cast<long long>(z) * p.ny + y) * p.nx + x;
            EpilogueInputs e = epilogue_request(p, v, c_first, row_ok && z < t.z1);
            while (z < t.z1) {
                if (c == 0) {
                    ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&ready[stage * kSlabMaxSlices + z - t.z0]), use & 1));
                    if (!ok) break;
                    tc::fence_after_sync();
                }
                int zn = z, cn = c + 16;
                long long vn = v;
                if (cn == sh.nc) {
                    cn = 0;
                    zn += 1;
                    vn += plane;
                }
                const EpilogueInputs next = epilogue_request(p, vn, c_first + cn, row_ok && zn < t.z1);
                conv_epilogue(p, acc + (z - t.z0) * sh.nc + c, v, c_first + c, row_ok, e, bias + c);
                e = next;
                z = zn;
                c = cn;
                v = vn;
            }
            tc::fence_before_sync();
            __syncwarp();
            if ((tid & 31) == 0) tc::mbar_arrive(tc::smem_addr(&drained[stage]));
        }
        if (!ok) failed = 1;
    }
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0 && failed) atomicExch(p.status, 1);
    if (warp == 4) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, sh.columns);
    }
}

// ---- slab weight gradient ---------------------------------------------------------------------
// dW[co][t][ci] = sum_v dZ[v][co] X[v + t][ci], and db[co] = sum_v dZ[v][co].
//
// A GEMM whose K side is the voxels.  Both operands are kept as the convolution keeps its input, [channels
// / 8][position][8 channels], which is the MN-major no-swizzle layout: eight positions are a core matrix,
// so a tap's shift is again a start address.  A tile is a patch of W x 2 voxels over a run of slices; X
// has four rows of pitch W + 2 per slice and 8-channel plane, dZ two rows with zeros in the two columns
// between them, so that K is one run of 2 W + 2 positions (W = 7 mod 8: whole steps of 16).
//
// M = 128 rows are 16 groups of 8 channels, one pitch apart: group 4 c + dy is plane c read dy rows
// further, so one MMA covers the three taps in y of 32 channels (dy = 3 is not used); with 16 input
// channels the upper eight groups are the next slice.  N is dZ of the slices that an input slice meets
// through the three taps in z (four for a pair of slices), times the output channels.  The taps in x are
// three MMAs with accumulators of their own.  So every voxel of X and dZ is brought once per CTA, and 27
// taps cost three MMAs per 16 positions.
//
// Eight warps bring the tiles (two stages), sum dZ for the bias, take each tile's accumulators into registers
// and add the sums to dw with atomics; the ninth issues the MMAs.  The tensor core's accumulation truncates,
// and its error grows by about 1e-8 of the result per K step: with accumulators of at least 96 steps the
// error was up to 1.7 times that of shorter ones on small grids and deep layers.  A tile takes at most a few
// tens, and reading it costs nothing, since the next tile arrives meanwhile.  A CTA computes 32 (or 16) x 32
// (or 16) channels of dW for its share of the tiles.
//
// One pass, in us (in brackets with accumulators of 96 steps or more, then the kernel that gathered each
// tap's rows by threads, 128 rows of dW a CTA): 200x200x32, 16 to 16 channels 52 (70, 394), 32 to 16 82
// (120); 100x100x16, 32 to 32 24 (37, 160 with its bias sums), 64 to 32 35 (48); 50x50x8, 64 to 64 18 (18, 56),
// 128 to 64 22 (28); 25x25x4, 128 to 128 15 (15, 18); 32 to 128 at 50x50x8 21 (18).  All layers of the
// 200x200x32 network 0.68 ms (0.77; 3.23, and 0.22 for the bias sums).  The bytes brought bound it: halos
// double X, and dZ is read with two more slices per run.
struct ConvWgradArgs {
    const bf16* in;  // forward input, [nz>>up][ny>>up][nx>>up][cin]
    int cin, up;
    const bf16* dz;  // gradient at the conv output (before bias/ReLU), [V][cout]
    int cout;
    int nx, ny, nz;
    float* dw;       // [cout][27][cin], accumulated
    float* db;       // [cout], accumulated, or null
    int* status;
};

struct WgradShape {
    int W, positions, steps;  // patch width, positions of an X plane (4 pitch), K steps of 16
    int tiles_x, tiles_y, zt; // patches, slices of a run
    int tiles, ctas;          // patches x runs, CTAs per channel tile
    int ci_tiles, co_tiles, co;  // channel tiles, output channels of a tile
    int x_plane, x_slice, z_plane, z_slice, stage, smem;  // bytes
    unsigned columns;
};

constexpr int kWgradLoaders = 256;
constexpr int kWgradThreads = kWgradLoaders + 32;

// The elements `which` (bits: output channels from co on) of a CTA's tiles, summed from memory and
// added to dw: those whose accumulator is not finite.  The zeros of dZ between a patch's rows meet
// values of X there, and an infinity or a NaN among these would reach taps that never see it.  The
// check for it costs 1 us of 70 a call at 100x100x16, 32 to 32 channels, and none at 200x200x32.
template <bool kPair>
__device__ __forceinline__ void wgrad_direct(const ConvWgradArgs& p, const WgradShape& sh, int tiles, unsigned which,
                                          int half, int dz, int dy, int dx, int ci, int co)
{
    const int patches = sh.tiles_x * sh.tiles_y, sx = p.nx >> p.up, sy = p.ny >> p.up;
    for (; which; which &= which - 1) {
        const int c = co + __ffs(which) - 1;
        float sum = 0.f;
        for (int k = 0; k < tiles && !isnan(sum); ++k) {
            const int tile = blockIdx.x + k * sh.ctas, run = tile / patches, patch = tile - run * patches;
            const int py = patch / sh.tiles_x, x0 = (patch - py * sh.tiles_x) * sh.W, y0 = py * 2, z0 = run * sh.zt;
            for (int zi = z0 + half; zi < min(z0 + sh.zt, p.nz); zi += kPair ? 2 : 1) {
                const int z = zi + 1 - dz;
                if (z < 0 || z >= p.nz) continue;
                for (int y = y0; y < min(y0 + 2, p.ny); ++y)
#pragma unroll 4
                    for (int x = x0; x < min(x0 + sh.W, p.nx); ++x) {
                        const int yi = y + dy - 1, xi = x + dx - 1;
                        float in = 0.f;
                        if (yi >= 0 && yi < p.ny && xi >= 0 && xi < p.nx)
                            in = __bfloat162float(p.in[((static_cast<size_t>(zi >> p.up) * sy + (yi >> p.up)) * sx + (xi >> p.up)) * p.cin + ci]);
                        sum += in * __bfloat162float(p.dz[((static_cast<size_t>(z) * p.ny + y) * p.nx + x) * p.cout + c]);
                    }
            }
        }
        atomicAdd(p.dw + (static_cast<size_t>(c) * 27 + dz * 9 + dy * 3 + dx) * p.cin + ci, sum);
    }
}

template <bool kPair, int kCo>
__global__ void __launch_bounds__(kWgradThreads, 1) conv3_wgrad_slab_kernel(const __grid_constant__ ConvWgradArgs p,
                                                                         const __grid_constant__ WgradShape sh)
{
    constexpr int kXPlanes = kPair ? 2 : 4, kXLog = kPair ? 1 : 2;  // 8-channel planes of an input tile
    constexpr int kWindow = kPair ? 4 : 3;                         // dZ slices that an MMA covers
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[2];
    __shared__ __align__(8) uint64_t empty[2];
    __shared__ __align__(8) uint64_t taken;  // a tile's accumulators read
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    __shared__ uint32_t corner[272];  // row << 16 | column of a position
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t base = (tc::smem_addr(smem_raw) + 127u) & ~127u;
    const int pitch = sh.W + 2;
    const int ci0 = blockIdx.y % sh.ci_tiles * 32, co0 = blockIdx.y / sh.ci_tiles * kCo;
    constexpr int zc = kCo >> 3, zcl = zc == 2 ? 1 : 2;  // 8-channel planes of dZ
    const int patches = sh.tiles_x * sh.tiles_y;

    if (warp == 8) tc::tmem_alloc(tc::smem_addr(&tmem_slot), sh.columns);
    if (tid < 2) {
        tc::mbar_init(tc::smem_addr(&full[tid]), kWgradLoaders / 32);
        tc::mbar_init(tc::smem_addr(&empty[tid]), 1);
    }
    if (tid == 2) tc::mbar_init(tc::smem_addr(&taken), kWgradLoaders / 32);
    if (tid < 3) tc::mbar_init_fence();
    if (tid == 0) failed = 0;
    for (int q = tid; q < sh.positions; q += kWgradThreads) {
        const int row = q / pitch;
        corner[q] = static_cast<uint32_t>(row) << 16 | static_cast<uint32_t>(q - row * pitch);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tmem_slot;

    if (warp < 8) {
        const int sx = p.nx >> p.up, sy = p.ny >> p.up;
        const int x_units = sh.positions << kXLog, z_units = (sh.steps * 16) << zcl;
        const bool sums = p.db != nullptr && ci0 == 0;
        float bias[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // of dZ plane tid % zc
        // TMEM lane (row) m of the M side: plane, row shift and channel; upper half: the next slice
        const int m = (warp & 3) * 32 + (tid & 31);
        const int half = kPair ? m >> 6 : 0, dy = (m >> 3) & 3;
        const int ci = ci0 + (kPair ? (m & 63) >> 5 : m >> 5) * 8 + (m & 7);
        const uint32_t lane = tmem + (static_cast<uint32_t>(warp & 3) * 32u << 16);
        // The tiles' sums wait in registers, and go back to TMEM before they are added to dw, so that the code
        // for that is there once (unrolled it cost 3 us of instruction fetches).
        constexpr int n = kWindow * kCo, kBlocks = 3 * n / 16, kHeld = (kBlocks + 1) / 2;  // 16 columns each; of this warp
        const int first = warp >> 2;
        float sum[kHeld][16];
#pragma unroll
        for (int h = 0; h < kHeld; ++h)
#pragma unroll
            for (int i = 0; i < 16; ++i) sum[h][i] = 0.f;
        bool ok = true;
        int tiles = 0;  // requested so far
        auto multiplied = [&](int k) {  // waits for the MMAs of tile k
            const bool in_time = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&empty[k & 1]), (k >> 1) & 1));
            tc::fence_after_sync();
            return in_time;
        };
        for (int tile = blockIdx.x; tile < sh.tiles && ok; tile += sh.ctas, ++tiles) {
            const int run = tile / patches, patch = tile - run * patches, py = patch / sh.tiles_x;
            const int x0 = (patch - py * sh.tiles_x) * sh.W, y0 = py * 2, z0 = run * sh.zt;
            const int stage = tiles & 1;  // free: the MMAs of tile tiles - 2 have been waited for
            const uint32_t dst = base + stage * sh.stage, dst_z = dst + sh.zt * sh.x_slice;
            for (int u = tid; u < x_units; u += kWgradLoaders) {
                const int q = u >> kXLog, c = u & (kXPlanes - 1);
                const uint32_t at = corner[q];
                const int y = y0 + static_cast<int>(at >> 16) - 1, x = x0 + static_cast<int>(at & 0xffffu) - 1;
                const bool inside = static_cast<unsigned>(x) < static_cast<unsigned>(p.nx) &&
                                    static_cast<unsigned>(y) < static_cast<unsigned>(p.ny);
                const bf16* from = p.in + static_cast<size_t>(inside ? (y >> p.up) * sx + (x >> p.up) : 0) * p.cin + ci0 + c * 8;
                const uint32_t to = dst + c * sh.x_plane + q * 16;
                for (int s = 0; s < sh.zt; ++s) {
                    const bool there = inside && z0 + s < p.nz;
                    cp_async16(to + s * sh.x_slice,
                               from + (there ? static_cast<size_t>((z0 + s) >> p.up) * sy * sx * p.cin : 0), there);
                }
            }
            for (int u = tid; u < z_units; u += kWgradLoaders) {
                const int q = u >> zcl, c = u & (zc - 1);
                const uint32_t at = corner[q];
                const int row = static_cast<int>(at >> 16), column = static_cast<int>(at & 0xffffu);
                const int y = y0 + row, x = x0 + column;
                const bool inside = row < 2 && column < sh.W && x < p.nx && y < p.ny;
                const bf16* from = p.dz + (inside ? static_cast<size_t>(y) * p.nx + x : 0) * p.cout + co0 + c * 8;
                const uint32_t to = dst_z + c * sh.z_plane + q * 16;
                for (int s = 0; s < sh.zt + 2; ++s) {
                    const int z = z0 - 1 + s;
                    const bool there = inside && z >= 0 && z < p.nz;
                    cp_async16(to + s * sh.z_slice, from + (there ? static_cast<size_t>(z) * p.ny * p.nx * p.cout : 0), there);
                }
            }
            cp_async_commit();
            cp_async_wait<0>();
            tc::fence_proxy_async();
            __syncwarp();
            if ((tid & 31) == 0) tc::mbar_arrive(tc::smem_addr(&full[stage]));
            if (sums) {  // this thread adds up the dZ units it brought
                const uint32_t from = dst_z + (tid & (zc - 1)) * sh.z_plane;
                for (int s = 1; s <= sh.zt; ++s)  // the run's own slices
                    for (int u = tid; u < z_units; u += kWgradLoaders) {
                        uint4 raw;
                        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                     : "=r"(raw.x), "=r"(raw.y), "=r"(raw.z), "=r"(raw.w)
                                     : "r"(from + s * sh.z_slice + (u >> zcl) * 16) : "memory");
                        float f[8];
                        unpack8(raw, f);
#pragma unroll
                        for (int i = 0; i < 8; ++i) bias[i] += f[i];
                    }
            }
            if (tiles == 0) continue;
            ok = multiplied(tiles - 1);
            if (!ok) break;
#pragma unroll
            for (int h = 0; h < kHeld; ++h)
                if (2 * h + first < kBlocks) {
                    float acc[16];
                    tc::tmem_load16(lane + (2 * h + first) * 16, acc);
#pragma unroll
                    for (int i = 0; i < 16; ++i) sum[h][i] += acc[i];
                }
            tc::fence_before_sync();
            __syncwarp();
            if ((tid & 31) == 0) tc::mbar_arrive(tc::smem_addr(&taken));
        }
        ok = ok && tiles > 0 && multiplied(tiles - 1);
        if (ok) {
            if (tiles > 1) {
#pragma unroll
                for (int h = 0; h < kHeld; ++h)
                    if (2 * h + first < kBlocks) {
                        float acc[16];
                        tc::tmem_load16(lane + (2 * h + first) * 16, acc);
#pragma unroll
                        for (int i = 0; i < 16; ++i) acc[i] += sum[h][i];
                        tc::tmem_store16(lane + (2 * h + first) * 16, acc);
                    }
                tc::tmem_store_wait();
            }
            for (int b = first; b < kBlocks; b += 2) {  // one tap in x, dZ slice, output channels
                float acc[16];
                tc::tmem_load16(lane + b * 16, acc);
                const int dx = b * 16 / n, column = b * 16 - dx * n;
                const int w = column / kCo, co = co0 + column - w * kCo;
                const int dz = half + 2 - w;
                if (dy < 3 && dz >= 0 && dz < 3) {
                    float finite = 0.f;
#pragma unroll
                    for (int i = 0; i < 16; ++i) finite = fmaf(acc[i], 0.f, finite);
                    float* dw = p.dw + (static_cast<size_t>(co) * 27 + dz * 9 + dy * 3 + dx) * p.cin + ci;
                    if (finite == 0.f) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) atomicAdd(dw + static_cast<size_t>(i) * 27 * p.cin, acc[i]);
                    } else {
                        unsigned direct = 0;
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            if (isfinite(acc[i])) atomicAdd(dw + static_cast<size_t>(i) * 27 * p.cin, acc[i]);
                            else direct |= 1u << i;
                        wgrad_direct<kPair>(p, sh, tiles, direct, half, dz, dy, dx, ci, co);
                    }
                }
                __syncwarp();
            }
        }
        if (sums && ok) {
            // lanes of the same plane
#pragma unroll
            for (int o = 16; o >= 2; o >>= 1)
                if (o >= zc)
#pragma unroll
                    for (int i = 0; i < 8; ++i) bias[i] += __shfl_xor_sync(0xffffffffu, bias[i], o);
            if ((tid & 31) < zc)
#pragma unroll
                for (int i = 0; i < 8; ++i) atomicAdd(p.db + co0 + (tid & 31) * 8 + i, bias[i]);
        }
        if (!ok) failed = 1;
    } else {
        const uint32_t leader = tc::elect_one();
        constexpr uint32_t n = kWindow * kCo;
        const uint32_t idesc = tc::idesc_bf16_f32(static_cast<int>(n), true);
        const uint64_t a_base = tc::smem_desc(base, 128, pitch * 16), b_base = tc::smem_desc(base + sh.zt * sh.x_slice, 128, sh.z_plane);
        const uint32_t a_hi = static_cast<uint32_t>(a_base >> 32), b_hi = static_cast<uint32_t>(b_base >> 32);
        bool ok = true;
        int k = 0;
        for (int tile = blockIdx.x; tile < sh.tiles && ok; tile += sh.ctas, ++k) {
            const int z0 = tile / patches * sh.zt, stage = k & 1;
            ok = __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&full[stage]), (k >> 1) & 1)) &&
                 (k == 0 || __all_sync(0xffffffffu, tc::mbar_wait(tc::smem_addr(&taken), (k - 1) & 1)));
            if (!ok) break;
            tc::fence_after_sync();
            const int slices = z0 + sh.zt < p.nz ? sh.zt : p.nz - z0;
            uint32_t started = 0;
            for (int s = 0; s < slices; s += kPair ? 2 : 1) {
                // the descriptors' address fields count 16 bytes: one position
                uint32_t a = static_cast<uint32_t>(a_base) + ((stage * sh.stage + s * sh.x_slice) >> 4);
                uint32_t b = static_cast<uint32_t>(b_base) + ((stage * sh.stage + s * sh.z_slice) >> 4);
                for (int j = 0; j < sh.steps; ++j, a += 16, b += 16) {
                    tc::mma_bf16_warp(tmem, a, a_hi, b, b_hi, idesc, started, leader);
                    tc::mma_bf16_warp(tmem + n, a + 1, a_hi, b, b_hi, idesc, started, leader);
                    tc::mma_bf16_warp(tmem + 2 * n, a + 2, a_hi, b, b_hi, idesc, started, leader);
                    started = 1;
                }
            }
            tc::mma_commit_warp(tc::smem_addr(&empty[stage]), leader);
        }
        if (!ok) failed = 1;
    }
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0 && failed) atomicExch(p.status, 1);
    if (warp == 8) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem, sh.columns);
    }
}

// --------------------------------------------------------------------- elementwise kernels --

__global__ void pack_input_kernel(const float* __restrict__ x0, const uint8_t* __restrict__ hull, long long V,
                                  bf16* __restrict__ out)
{
    for (long long v = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; v < V;
         v += static_cast<long long>(gridDim.x) * blockDim.x) {
        uint4 a = make_uint4(pack_bf16(x0[v], hull[v] ? 1.f : 0.f), 0, 0, 0);
        reinterpret_cast<uint4*>(out + v * 16)[0] = a;
        reinterpret_cast<uint4*>(out + v * 16)[1] = make_uint4(0, 0, 0, 0);
    }
}

// 2x2x2 average; one thread per (coarse voxel, 8 channels).
__global__ void avgpool_kernel(const bf16* in, int nx, int ny, int nz, int c, bf16* __restrict__ out)
{
    grid_dependency_wait();  // `in` is not read through the read-only path: its writer may have just ended
    allow_dependent_launch();
    const int cx = nx / 2, cy = ny / 2, cz = nz / 2, g = c / 8;
    const long long n = static_cast<long long>(cx) * cy * cz * g;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int cg = static_cast<int>(i % g);
        const long long cv = i / g;
        const int x = static_cast<int>(cv % cx), y = static_cast<int>((cv / cx) % cy), z = static_cast<int>(cv / (static_cast<long long>(cx) * cy));
        float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int d = 0; d < 8; ++d) {
            const long long fv = (static_cast<long long>(2 * z + (d >> 2)) * ny + 2 * y + ((d >> 1) & 1)) * nx + 2 * x + (d & 1);
            float f[8];
            unpack8(*(reinterpret_cast<const uint4*>(in + fv * c) + cg), f);
#pragma unroll
            for (int k = 0; k < 8; ++k) s[k] += f[k];
        }
        uint4 o;
        o.x = pack_bf16(s[0] * 0.125f, s[1] * 0.125f);
        o.y = pack_bf16(s[2] * 0.125f, s[3] * 0.125f);
        o.z = pack_bf16(s[4] * 0.125f, s[5] * 0.125f);
        o.w = pack_bf16(s[6] * 0.125f, s[7] * 0.125f);
        reinterpret_cast<uint4*>(out + cv * c)[cg] = o;
    }
}

// Gradient through avg-pool and a skip: out = (dp[parent] / 8 + dskip) * (act > 0), fine grid.
__global__ void unpool_add_mask_kernel(const bf16* __restrict__ dp, const bf16* __restrict__ dskip,
                                       const bf16* __restrict__ act, int nx, int ny, int nz, int c,
                                       bf16* __restrict__ out)
{
    const int g = c / 8;
    const long long n = static_cast<long long>(nx) * ny * nz * g;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int cg = static_cast<int>(i % g);
        const long long v = i / g;
        const int x = static_cast<int>(v % nx), y = static_cast<int>((v / nx) % ny), z = static_cast<int>(v / (static_cast<long long>(nx) * ny));
        const long long pv = (static_cast<long long>(z / 2) * (ny / 2) + y / 2) * (nx / 2) + x / 2;
        float a[8], s[8], m[8];
        unpack8(__ldg(reinterpret_cast<const uint4*>(dp + pv * c) + cg), a);
        unpack8(__ldg(reinterpret_cast<const uint4*>(dskip + v * c) + cg), s);
        unpack8(__ldg(reinterpret_cast<const uint4*>(act + v * c) + cg), m);
        float r[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) r[k] = m[k] > 0.f ? a[k] * 0.125f + s[k] : 0.f;
        uint4 o;
        o.x = pack_bf16(r[0], r[1]);
        o.y = pack_bf16(r[2], r[3]);
        o.z = pack_bf16(r[4], r[5]);
        o.w = pack_bf16(r[6], r[7]);
        reinterpret_cast<uint4*>(out + v * c)[cg] = o;
    }
}

// Gradient through nearest x2 upsampling: out[coarse] = sum of the 8 fine children, * (act > 0).
__global__ void upsum_mask_kernel(const bf16* __restrict__ du, const bf16* __restrict__ act, int cx, int cy, int cz,
                                  int c, bf16* __restrict__ out)
{
    const int g = c / 8, nx = 2 * cx, ny = 2 * cy;
    const long long n = static_cast<long long>(cx) * cy * cz * g;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const int cg = static_cast<int>(i % g);
        const long long cv = i / g;
        const int x = static_cast<int>(cv % cx), y = static_cast<int>((cv / cx) % cy), z = static_cast<int>(cv / (static_cast<long long>(cx) * cy));
        float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int d = 0; d < 8; ++d) {
            const long long fv = (static_cast<long long>(2 * z + (d >> 2)) * ny + 2 * y + ((d >> 1) & 1)) * nx + 2 * x + (d & 1);
            float f[8];
            unpack8(__ldg(reinterpret_cast<const uint4*>(du + fv * c) + cg), f);
#pragma unroll
            for (int k = 0; k < 8; ++k) s[k] += f[k];
        }
        float m[8];
        unpack8(__ldg(reinterpret_cast<const uint4*>(act + cv * c) + cg), m);
        uint4 o;
        o.x = pack_bf16(m[0] > 0.f ? s[0] : 0.f, m[1] > 0.f ? s[1] : 0.f);
        o.y = pack_bf16(m[2] > 0.f ? s[2] : 0.f, m[3] > 0.f ? s[3] : 0.f);
        o.z = pack_bf16(m[4] > 0.f ? s[4] : 0.f, m[5] > 0.f ? s[5] : 0.f);
        o.w = pack_bf16(m[6] > 0.f ? s[6] : 0.f, m[7] > 0.f ? s[7] : 0.f);
        reinterpret_cast<uint4*>(out + cv * c)[cg] = o;
    }
}

// The sum over a CTA of 256 threads, in its first thread: one atomic per CTA on the address that all
// share.  With one per warp, 19,000 of them, the loss took 34 us on 200x200x32 voxels.
template <class T>
__device__ __forceinline__ T cta_sum(T v)
{
    __shared__ T part[8];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < 8; ++w) v += part[w];
    return v;
}

__global__ void count_kernel(const uint8_t* __restrict__ hull, long long V, unsigned long long* __restrict__ count)
{
    unsigned long long n = 0;
    for (long long v = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; v < V;
         v += static_cast<long long>(gridDim.x) * blockDim.x)
        n += hull[v] ? 1 : 0;
    n = cta_sum(n);
    if (threadIdx.x == 0 && n) atomicAdd(count, n);
}

// Masked mean-squared error over the hull voxels: loss += (y - t)^2 / count, and the gradient
// dL/dy = 2 (y - t) / count as channel 0 of a 16-channel bf16 tensor (other channels 0).
__global__ void loss_kernel(const float* __restrict__ y, const float* __restrict__ target, const uint8_t* __restrict__ hull,
                            long long V, const unsigned long long* __restrict__ count, bf16* __restrict__ dy,
                            double* __restrict__ loss)
{
    const double inv = *count ? 1.0 / static_cast<double>(*count) : 0.0;
    double acc = 0.0;
    for (long long v = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; v < V;
         v += static_cast<long long>(gridDim.x) * blockDim.x) {
        const float d = hull[v] ? y[v] - target[v] : 0.f;
        acc += static_cast<double>(d) * d;
        const float g = static_cast<float>(2.0 * d * inv);
        reinterpret_cast<uint4*>(dy + v * 16)[0] = make_uint4(pack_bf16(g, 0.f), 0, 0, 0);
        reinterpret_cast<uint4*>(dy + v * 16)[1] = make_uint4(0, 0, 0, 0);
    }
    const double sum = cta_sum(acc);
    if (threadIdx.x == 0) atomicAdd(loss, sum * inv);
}

__global__ void nonfinite_kernel(const float* __restrict__ y, long long V, unsigned long long* __restrict__ count)
{
    unsigned long long n = 0;
    for (long long v = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; v < V;
         v += static_cast<long long>(gridDim.x) * blockDim.x)
        n += isfinite(y[v]) ? 0 : 1;
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(count, n);
}

__global__ void adam_kernel(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ s, long long n, float lr, float b1, float b2, float eps, float bc1,
                            float bc2)
{
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.f - b1) * gi;
        const float si = b2 * s[i] + (1.f - b2) * gi * gi;
        m[i] = mi;
        s[i] = si;
        w[i] -= lr * (mi / bc1) / (sqrtf(si / bc2) + eps);
    }
}

// bf16 copies of one layer's weights: W[co][t][ci] and the data-gradient form W'[ci][26-t][co].
__global__ void emit_weights_kernel(const float* __restrict__ w, int cin, int cout, bf16* __restrict__ wb,
                                    bf16* __restrict__ wt)
{
    const int n = cout * 27 * cin;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int ci = i % cin, t = (i / cin) % 27, co = i / (27 * cin);
        const bf16 h = __float2bfloat16_rn(w[i]);
        wb[i] = h;
        wt[(static_cast<size_t>(ci) * 27 + (26 - t)) * cout + co] = h;
    }
}

// ------------------------------------------------------------------------ launch helpers --

int grid_for(long long n, int threads)
{
    long long b = (n + threads - 1) / threads;
    if (b > 148LL * 16) b = 148LL * 16;
    return static_cast<int>(b < 1 ? 1 : b);
}

cudaError_t set_smem_limits()
{
    static bool done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
    for (auto kernel : {conv3_slab_kernel<16>, conv3_slab_kernel<32>, conv3_slab_kernel<64>, conv3_slab_kernel<128>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSlabSmemLimit);
    for (auto kernel : {conv3_wgrad_slab_kernel<false, 16>, conv3_wgrad_slab_kernel<false, 32>, conv3_wgrad_slab_kernel<true, 16>, conv3_wgrad_slab_kernel<true, 32>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSlabSmemLimit);
    if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = true;
    return e;
}

bool valid_channels(int c) { return c == 16 || c == 32 || c == 64 || c == 128; }

// The slab kernel's shape for a convolution: the patch that covers the grid with the fewest patches
// (rows of W + 2 positions, 128 positions in all) among those of which two slices fit beside the weights
// of 16 channels (with 128 input channels a patch one row high may hold 223 positions, not 384), and the channels, slices and ring of a CTA with the
// least estimated time.  The estimate takes per input slice the larger of its MMAs (32 + N/4 cycles each:
// both operands are read from shared memory at 128 bytes a cycle) and its bytes at 48 a cycle, for each
// of the CTAs that share an SM, or the latency of one request over the requests in flight; and once per
// CTA its weights, start and end.
SlabShape slab_shape(int cin, int cout, int nx, int ny, int nz)
{
    SlabShape best{};
    long long fewest = 0;
    for (int W = 1; W <= 126 && W <= nx; ++W) {
        int H = (128 - W) / (W + 2) + 1;
        if (H > ny) H = ny;
        const int positions = (W + 2) * (H + 2);
        if (positions > kSlabMaxPositions || 2 * positions * 16 * (cin / 8) + 27 * cin * 16 * 2 + kSlabSlack > kSlabSmemLimit) continue;
        const int tx = (nx + W - 1) / W, ty = (ny + H - 1) / H;
        const long long cost = static_cast<long long>(tx) * ty * (256 + positions);
        if (fewest == 0 || cost < fewest) {
            fewest = cost;
            best.W = W;
            best.H = H;
            best.tiles_x = tx;
            best.tiles_y = ty;
            best.positions = positions;
        }
    }
    // rows of an MMA reach 2 (W + 2) + 2 + 127 positions into a plane; the last plane's excess falls in
    // the weights or the slack behind them
    best.chunk_bytes = best.positions * 16;
    best.slice_bytes = best.chunk_bytes * (cin / 8);
    double least = 0.0;
    SlabShape chosen = best;
    for (int nc = cout < 64 ? cout : 64; nc >= 16; nc /= 2)
        for (int zt = 1; zt <= nz && zt <= kSlabMaxSlices && zt * nc <= kTmemColumns; zt = zt < nz && 2 * zt > nz ? nz : 2 * zt)
            for (int ring = 2; ring <= kSlabMaxRing; ++ring) {
                SlabShape t = best;
                t.nc = nc;
                t.nc_log2 = nc == 64 ? 6 : nc == 32 ? 5 : 4;
                t.zt = zt;
                t.ring = ring;
                t.ahead = ring - 1 < 2 ? ring - 1 : 2;
                t.weight_bytes = 27 * cin * nc * 2;
                t.tiles = t.tiles_x * t.tiles_y * ((nz + zt - 1) / zt);
                t.smem = ring * t.slice_bytes + t.weight_bytes + kSlabSlack;
                if (t.smem > kSlabSmemLimit) continue;
                const int groups = cout / nc;
                for (t.stages = 1; t.stages <= 2 && t.stages * zt * nc <= kTmemColumns; ++t.stages) {
                    SlabShape u = t;
                    u.columns = 32;
                    while (u.columns < static_cast<unsigned>(u.stages * zt * nc)) u.columns *= 2;
                    int per_sm = kTmemColumns / static_cast<int>(u.columns);
                    if (per_sm > 4) per_sm = 4;
                    const int floor_bytes = kSmemPerSm / (per_sm + 1) + 1;  // no more CTAs than TMEM holds
                    if (u.smem < floor_bytes) u.smem = floor_bytes;
                    const int fit = kSmemPerSm / (u.smem + 4096);
                    if (per_sm > fit) per_sm = fit;
                    if (per_sm < 1) per_sm = 1;
                    long long ctas = 148LL * per_sm / groups;
                    if (ctas < 1) ctas = 1;
                    u.ctas = static_cast<int>(ctas < u.tiles ? ctas : u.tiles);
                    const double laps = ceil(static_cast<double>(u.tiles) / u.ctas);
                    const double share = ceil(static_cast<double>(u.ctas) * groups / 148.0);
                    const int slices = zt + 2 < nz ? zt + 2 : nz;
                    const double mma = 9.0 * (cin / 16) * (32 + 0.75 * nc) * share, load = u.slice_bytes / 48.0 * share;
                    const double wait = 1500.0 / u.ahead;
                    double slice = mma > load ? mma : load;
                    if (wait > slice) slice = wait;
                    // the MMAs need a slice or two in hand while others are on their way
                    slice *= ring >= 5 ? 1.0 : ring == 4 ? 1.1 : ring == 3 ? 1.25 : 1.5;
                    // with one stage a tile's MMAs wait until the last one is written
                    const double tile = slices * slice + (u.stages == 1 ? 1500.0 : 0.0);
                    const double time = 6000.0 + u.weight_bytes * share / 32.0 + laps * tile;
                    if (least == 0.0 || time < least) {
                        least = time;
                        chosen = u;
                    }
                }
            }
    return chosen;
}

cudaError_t launch_conv_fwd(const ConvFwdArgs& a, cudaStream_t s)
{
    cudaError_t e = set_smem_limits();
    if (e != cudaSuccess) return e;
    const SlabShape sh = slab_shape(a.cin, a.cout, a.nx, a.ny, a.nz);
    if (sh.smem == 0) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sh.ctas, a.cout / sh.nc);
    cfg.blockDim = dim3(kSlabThreads);
    cfg.dynamicSmemBytes = sh.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.overlap ? 1 : 0;
    switch (a.cin) {
        case 16: return cudaLaunchKernelEx(&cfg, conv3_slab_kernel<16>, a, sh);
        case 32: return cudaLaunchKernelEx(&cfg, conv3_slab_kernel<32>, a, sh);
        case 64: return cudaLaunchKernelEx(&cfg, conv3_slab_kernel<64>, a, sh);
        default: return cudaLaunchKernelEx(&cfg, conv3_slab_kernel<128>, a, sh);
    }
}

// The weight gradient's shape: patch width, run length and CTAs with the least estimated time among those whose
// estimated error is at most that of a split of the voxels in chunks of 64 over 888 CTAs of 128 rows of
// dW.  That was a kernel of one accumulation per CTA, whose errors are the bar.
//  * Error, relative, fitted to those of both from 24x24x4 to 200x200x32 (within 10%): 1e-8 for each K step of
//    an accumulator, its truncation, and 1.8e-8 times the root of the additions to an element of dw.
//  * Time, cycles, fitted to 250 shapes of 18 layers (12% rms; the shape it picks is the fastest of those
//    tried or within 10% of it): per tile its MMAs at 1.27 (32 + N/4) or its bytes at 16.4 a cycle,
//    whichever is more, and 2600 for the rest; and the first tile's bytes, which nothing overlaps.
WgradShape wgrad_shape(int cin, int cout, int nx, int ny, int nz)
{
    const bool pair = cin == 16;
    const int planes = pair ? 2 : 4;
    WgradShape best{};
    best.ci_tiles = pair ? 1 : cin / 32;
    best.co = cout == 16 ? 16 : 32;
    best.co_tiles = cout / best.co;
    best.tiles_y = (ny + 1) / 2;
    const int n = (pair ? 4 : 3) * best.co;
    best.columns = 3 * n <= 256 ? 256 : 512;
    const int groups = best.ci_tiles * best.co_tiles;
    auto error = [](double steps, double additions) { return 1e-16 * steps * steps + 3.24e-16 * additions; };  // squared
    const long long chunks = (static_cast<long long>(nx) * ny * nz + 63) / 64, rows = (27 * cin + 127) / 128;
    const long long splits = (888 + rows - 1) / rows < chunks ? (888 + rows - 1) / rows : chunks;
    const long long share = (chunks + splits - 1) / splits;
    const long long parts = (chunks + share - 1) / share, halves = pair ? 2 : 1;  // halves: additions of a CTA to an element
    const double allowed = error(4.0 * share, static_cast<double>(parts));
    auto patch_cost = [&](int W) { return (nx + W - 1) / W * (2 * W + 2 + 16); };
    int fewest = patch_cost(7);
    for (int W = 15; W <= 63; W += 8)
        if (patch_cost(W) < fewest) fewest = patch_cost(W);
    WgradShape chosen = best;
    double least = 0.0, nearest = 0.0;  // the nearest error, until one is allowed
    for (int W = 7; W <= 63; W += 8) {
        if (patch_cost(W) > fewest * 5 / 4) continue;
        best.W = W;
        best.positions = 4 * (W + 2);
        best.steps = (2 * W + 2) / 16;
        best.tiles_x = (nx + W - 1) / W;
        best.x_plane = best.positions * 16;
        best.x_slice = best.x_plane * planes;
        best.z_plane = best.steps * 256;
        best.z_slice = best.z_plane * (best.co / 8);
        for (int zt = pair ? 2 : 1; zt <= (pair ? nz + 1 : nz) && zt <= 32; zt += pair ? 2 : 1) {
            WgradShape t = best;
            t.zt = zt;
            t.stage = (zt * t.x_slice + (zt + 2) * t.z_slice + 127) & ~127;
            // rows that are not used read up to a pitch and a step past the last plane
            t.smem = 2 * t.stage + (t.W + 24) * 16 + 128;
            const int per_tile = (pair ? zt / 2 : zt) * t.steps;
            if (t.smem > kSlabSmemLimit || (per_tile > 4 * share && nearest != 0.0)) break;
            t.tiles = t.tiles_x * t.tiles_y * ((nz + zt - 1) / zt);
            const double mma = per_tile * 3.8 * (32 + n / 4.0), load = (zt * t.x_slice + (zt + 2.0) * t.z_slice) / 16.4;
            for (const long long most : {148LL, groups * (parts / halves)}) {  // CTAs: all, or for as many additions
                const long long ctas = (most < 148 ? most : 148) / groups;
                t.ctas = static_cast<int>(ctas < 1 ? 1 : ctas < t.tiles ? ctas : t.tiles);
                const int laps = (t.tiles + t.ctas - 1) / t.ctas;
                const double time = laps * ((mma > load ? mma : load) + 2600.0) + load;
                const double e = error(per_tile, static_cast<double>(t.ctas) * halves);
                if (e <= allowed ? least == 0.0 || time < least : least == 0.0 && (nearest == 0.0 || e < nearest)) {
                    if (e <= allowed) least = time;
                    nearest = e;
                    chosen = t;
                }
            }
        }
    }
    return chosen;
}

cudaError_t launch_conv_wgrad(const ConvWgradArgs& a, cudaStream_t s)
{
    cudaError_t e = set_smem_limits();
    if (e != cudaSuccess) return e;
    const WgradShape sh = wgrad_shape(a.cin, a.cout, a.nx, a.ny, a.nz);
    if (sh.smem == 0) return cudaErrorInvalidConfiguration;
    const dim3 grid(sh.ctas, sh.ci_tiles * sh.co_tiles);
    const auto kernel = a.cin == 16 ? (a.cout == 16 ? conv3_wgrad_slab_kernel<true, 16> : conv3_wgrad_slab_kernel<true, 32>)
                                    : (a.cout == 16 ? conv3_wgrad_slab_kernel<false, 16> : conv3_wgrad_slab_kernel<false, 32>);
    kernel<<<grid, kWgradThreads, sh.smem, s>>>(a, sh);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------ the network --

struct LayerSpec {
    int cin, cout, level, input, up, residual;  // input/residual: activation index (-1 = network input / none)
};

// Activation k is the output of layer k; pooled tensors are separate buffers (pool[level]).
constexpr int kLayers = 15;
constexpr int kPoolInput = 100;  // input code: pool[level] of the layer's level
const LayerSpec kSpec[kLayers] = {
    {16, 16, 0, -1, 0, -1},          {16, 16, 0, 0, 0, -1},            // e1a, e1
    {16, 32, 1, kPoolInput, 0, -1},  {32, 32, 1, 2, 0, -1},            // e2a, e2
    {32, 64, 2, kPoolInput, 0, -1},  {64, 64, 2, 4, 0, -1},            // e3a, e3
    {64, 128, 3, kPoolInput, 0, -1}, {128, 128, 3, 6, 0, -1},          // e4a, e4
    {128, 64, 2, 7, 1, 5},           {64, 64, 2, 8, 0, -1},            // d3a (+e3), d3
    {64, 32, 1, 9, 1, 3},            {32, 32, 1, 10, 0, -1},           // d2a (+e2), d2
    {32, 16, 0, 11, 1, 1},           {16, 16, 0, 12, 0, -1},           // d1a (+e1), d1
    {16, 16, 0, 13, 0, -1},                                            // output (channel 0)
};

}  // namespace unet
}  // namespace pct

using namespace pct::unet;

struct pct_unet {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int nx[4], ny[4], nz[4];
    long long nv[4];
    size_t w_off[kLayers], b_off[kLayers];
    size_t n_params = 0;
    float *params = nullptr, *grads = nullptr, *adam_m = nullptr, *adam_v = nullptr;
    bf16 *wb = nullptr, *wt = nullptr;  // bf16 weights, forward and data-gradient forms
    size_t wb_off[kLayers];
    bf16* input = nullptr;
    bf16* act[kLayers] = {};
    bf16* pool[4] = {};
    bf16* dz[kLayers] = {};
    bf16* tmp = nullptr;
    float* y = nullptr;
    unsigned long long* count = nullptr;
    double* loss = nullptr;
    int* status = nullptr;
    long long step = 0;
    std::string err;
};

namespace {

pct_status fail(pct_unet* n, pct_status s, const std::string& msg)
{
    if (n) n->err = msg;
    return s;
}

pct_status cuda_fail(pct_unet* n, cudaError_t e, const char* where)
{
    return fail(n, PCT_ERR_CUDA, std::string(where) + ": " + cudaGetErrorString(e));
}

#define UNET_CK(call, where)                              \
    do {                                                  \
        const cudaError_t e_ = (call);                    \
        if (e_ != cudaSuccess) return cuda_fail(n, e_, where); \
    } while (0)

void release(pct_unet* n)
{
    void* ptrs[] = {n->params, n->grads, n->adam_m, n->adam_v, n->wb, n->wt, n->input, n->tmp, n->y,
                    n->count, n->loss, n->status};
    for (void* p : ptrs)
        if (p) cudaFree(p);
    for (int l = 0; l < kLayers; ++l) {
        if (n->act[l]) cudaFree(n->act[l]);
        if (n->dz[l]) cudaFree(n->dz[l]);
    }
    for (int l = 0; l < 4; ++l)
        if (n->pool[l]) cudaFree(n->pool[l]);
    if (n->own_stream && n->stream) cudaStreamDestroy(n->stream);
}

pct_status emit_weights(pct_unet* n, cudaStream_t s)
{
    for (int l = 0; l < kLayers; ++l) {
        const LayerSpec& L = kSpec[l];
        emit_weights_kernel<<<grid_for(static_cast<long long>(L.cout) * 27 * L.cin, 256), 256, 0, s>>>(
            n->params + n->w_off[l], L.cin, L.cout, n->wb + n->wb_off[l], n->wt + n->wb_off[l]);
    }
    UNET_CK(cudaGetLastError(), "emit_weights_kernel");
    return PCT_OK;
}

const bf16* layer_input(pct_unet* n, int l)
{
    const LayerSpec& L = kSpec[l];
    if (L.input == -1) return n->input;
    if (L.input == kPoolInput) return n->pool[L.level];
    return n->act[L.input];
}

pct_status check_status(pct_unet* n, cudaStream_t s)
{
    int st = 0;
    UNET_CK(cudaMemcpyAsync(&st, n->status, sizeof(int), cudaMemcpyDeviceToHost, s), "status copy");
    UNET_CK(cudaStreamSynchronize(s), "synchronize");
    if (st) return fail(n, PCT_ERR_TIMEOUT, "a tensor-core pipeline wait expired");
    return PCT_OK;
}

// Forward pass: image = x0 + hull * network(x0, hull); all on stream s.
pct_status forward(pct_unet* n, const float* x0, const uint8_t* hull, float* image, cudaStream_t s)
{
    pack_input_kernel<<<grid_for(n->nv[0], 256), 256, 0, s>>>(x0, hull, n->nv[0], n->input);
    UNET_CK(cudaGetLastError(), "pack_input_kernel");
    for (int l = 0; l < kLayers; ++l) {
        const LayerSpec& L = kSpec[l];
        if (L.input == kPoolInput) {
            const int f = L.level - 1;  // pool the previous level's last encoder output
            const int src = 2 * f + 1;
            UNET_CK(pct::launch_kernel(true, avgpool_kernel, grid_for(n->nv[L.level] * (kSpec[src].cout / 8), 256), 256, s,
                                       n->act[src], n->nx[f], n->ny[f], n->nz[f], kSpec[src].cout, n->pool[L.level]),
                    "avgpool_kernel");
        }
        ConvFwdArgs a{};
        a.in = layer_input(n, l);
        a.cin = L.cin;
        a.up = L.up;
        a.weight = n->wb + n->wb_off[l];
        a.cout = L.cout;
        a.nx = n->nx[L.level];
        a.ny = n->ny[L.level];
        a.nz = n->nz[L.level];
        a.bias = n->params + n->b_off[l];
        a.residual = L.residual >= 0 ? n->act[L.residual] : nullptr;
        a.status = n->status;
        a.overlap = 1;
        if (l == kLayers - 1) {
            a.base = x0;
            a.hull = hull;
            a.image = image;
        } else {
            a.relu = 1;
            a.out = n->act[l];
        }
        UNET_CK(launch_conv_fwd(a, s), "conv3_slab_kernel");
    }
    return PCT_OK;
}

// Backward pass from n->dz[14] (dL/dy in channel 0): fills n->grads.
pct_status backward(pct_unet* n, cudaStream_t s)
{
    UNET_CK(cudaMemsetAsync(n->grads, 0, n->n_params * sizeof(float), s), "grad clear");
    for (int l = kLayers - 1; l >= 0; --l) {
        const LayerSpec& L = kSpec[l];
        const int nx = n->nx[L.level], ny = n->ny[L.level], nz = n->nz[L.level];
        // weights and bias
        ConvWgradArgs w{};
        w.in = layer_input(n, l);
        w.cin = L.cin;
        w.up = L.up;
        w.dz = n->dz[l];
        w.cout = L.cout;
        w.nx = nx;
        w.ny = ny;
        w.nz = nz;
        w.dw = n->grads + n->w_off[l];
        w.db = n->grads + n->b_off[l];
        w.status = n->status;
        UNET_CK(launch_conv_wgrad(w, s), "conv3_wgrad_slab_kernel");
        if (l == 0) break;
        // data gradient: conv of dz with the flipped, transposed weights
        ConvFwdArgs d{};
        d.cin = L.cout;
        d.cout = L.cin;
        d.in = n->dz[l];
        d.weight = n->wt + n->wb_off[l];
        d.nx = nx;
        d.ny = ny;
        d.nz = nz;
        d.status = n->status;
        d.overlap = 1;
        const bool into_tmp = L.up || L.input == kPoolInput;
        if (into_tmp) {
            d.out = n->tmp;  // gradient wrt the upsampled / pooled tensor
        } else {
            d.out = n->dz[L.input];
            d.mask = n->act[L.input];  // ReLU of the producing layer
        }
        UNET_CK(launch_conv_fwd(d, s), "conv3_slab_kernel (data gradient)");
        if (L.up) {
            const int src = L.input, cl = L.level + 1;
            upsum_mask_kernel<<<grid_for(n->nv[cl] * (L.cin / 8), 256), 256, 0, s>>>(
                n->tmp, n->act[src], n->nx[cl], n->ny[cl], n->nz[cl], L.cin, n->dz[src]);
            UNET_CK(cudaGetLastError(), "upsum_mask_kernel");
        } else if (L.input == kPoolInput) {
            const int f = L.level - 1, src = 2 * f + 1;
            // the decoder layer that adds act[src] as its residual
            int skip = -1;
            for (int k = 0; k < kLayers; ++k)
                if (kSpec[k].residual == src) skip = k;
            unpool_add_mask_kernel<<<grid_for(n->nv[f] * (L.cin / 8), 256), 256, 0, s>>>(
                n->tmp, n->dz[skip], n->act[src], n->nx[f], n->ny[f], n->nz[f], L.cin, n->dz[src]);
            UNET_CK(cudaGetLastError(), "unpool_add_mask_kernel");
        }
    }
    return PCT_OK;
}

pct_status loss_and_gradient(pct_unet* n, const float* x0, const uint8_t* hull, const float* target, double* loss_out,
                             cudaStream_t s)
{
    UNET_CK(cudaMemsetAsync(n->status, 0, sizeof(int), s), "status clear");
    pct_status st = forward(n, x0, hull, n->y, s);
    if (st != PCT_OK) return st;
    UNET_CK(cudaMemsetAsync(n->count, 0, sizeof(unsigned long long), s), "count clear");
    UNET_CK(cudaMemsetAsync(n->loss, 0, sizeof(double), s), "loss clear");
    count_kernel<<<grid_for(n->nv[0], 256), 256, 0, s>>>(hull, n->nv[0], n->count);
    loss_kernel<<<grid_for(n->nv[0], 256), 256, 0, s>>>(n->y, target, hull, n->nv[0], n->count, n->dz[kLayers - 1],
                                                       n->loss);
    UNET_CK(cudaGetLastError(), "loss_kernel");
    st = backward(n, s);
    if (st != PCT_OK) return st;
    if (loss_out) UNET_CK(cudaMemcpyAsync(loss_out, n->loss, sizeof(double), cudaMemcpyDeviceToHost, s), "loss copy");
    return check_status(n, s);
}

}  // namespace

extern "C" {

pct_status pct_unet_create(int columns, int rows, int slices, int64_t seed, int device, pct_unet** out)
{
    if (!out) return PCT_ERR_ARG;
    *out = nullptr;
    if (columns <= 0 || rows <= 0 || slices <= 0 || columns % 8 || rows % 8 || slices % 8) return PCT_ERR_ARG;
    pct_unet* n = new pct_unet();
    n->device = device;
    pct_status st = PCT_OK;
    auto ck = [&](cudaError_t e, const char* where) {
        if (e != cudaSuccess && st == PCT_OK) st = cuda_fail(n, e, where);
        return e == cudaSuccess;
    };
    if (ck(cudaSetDevice(device), "cudaSetDevice") && ck(cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking), "stream")) {
        n->own_stream = true;
        for (int l = 0; l < 4; ++l) {
            n->nx[l] = columns >> l;
            n->ny[l] = rows >> l;
            n->nz[l] = slices >> l;
            n->nv[l] = static_cast<long long>(n->nx[l]) * n->ny[l] * n->nz[l];
        }
        size_t off = 0, boff = 0;
        for (int l = 0; l < kLayers; ++l) {
            n->w_off[l] = off;
            off += static_cast<size_t>(kSpec[l].cout) * 27 * kSpec[l].cin;
            n->b_off[l] = off;
            off += kSpec[l].cout;
            n->wb_off[l] = boff;
            boff += static_cast<size_t>(kSpec[l].cout) * 27 * kSpec[l].cin;
        }
        n->n_params = off;
        // He-normal initial weights from a seeded generator; padding channels of the input layer,
        // and the whole output layer, start at zero (the untrained network returns x_0).
        std::vector<float> h(off, 0.f);
        std::mt19937_64 rng(static_cast<uint64_t>(seed));
        for (int l = 0; l < kLayers - 1; ++l) {
            const int fan_in = 27 * (l == 0 ? 2 : kSpec[l].cin);
            std::normal_distribution<float> nd(0.f, std::sqrt(2.f / fan_in));
            for (int co = 0; co < kSpec[l].cout; ++co)
                for (int t = 0; t < 27; ++t)
                    for (int ci = 0; ci < kSpec[l].cin; ++ci) {
                        const float w = nd(rng);
                        if (l != 0 || ci < 2) h[n->w_off[l] + (static_cast<size_t>(co) * 27 + t) * kSpec[l].cin + ci] = w;
                    }
        }
        const size_t pbytes = off * sizeof(float);
        ck(cudaMalloc(&n->params, pbytes), "cudaMalloc params");
        ck(cudaMalloc(&n->grads, pbytes), "cudaMalloc grads");
        ck(cudaMalloc(&n->adam_m, pbytes), "cudaMalloc adam");
        ck(cudaMalloc(&n->adam_v, pbytes), "cudaMalloc adam");
        ck(cudaMalloc(&n->wb, boff * sizeof(bf16)), "cudaMalloc weights");
        ck(cudaMalloc(&n->wt, boff * sizeof(bf16)), "cudaMalloc weights");
        ck(cudaMalloc(&n->input, n->nv[0] * 16 * sizeof(bf16)), "cudaMalloc input");
        for (int l = 0; l < kLayers; ++l) {
            const size_t bytes = n->nv[kSpec[l].level] * kSpec[l].cout * sizeof(bf16);
            ck(cudaMalloc(&n->act[l], bytes), "cudaMalloc activations");
            ck(cudaMalloc(&n->dz[l], bytes), "cudaMalloc gradients");
        }
        for (int l = 1; l < 4; ++l) ck(cudaMalloc(&n->pool[l], n->nv[l] * kSpec[2 * l].cin * sizeof(bf16)), "cudaMalloc pool");
        // largest data-gradient scratch: L0 x 32 (upsampled into d1a), L1 x 64, L2 x 128, pools
        size_t tmp = 0;
        for (int l = 0; l < kLayers; ++l)
            if (kSpec[l].up || kSpec[l].input == kPoolInput) {
                const size_t b = n->nv[kSpec[l].level] * kSpec[l].cin;
                if (b > tmp) tmp = b;
            }
        ck(cudaMalloc(&n->tmp, tmp * sizeof(bf16)), "cudaMalloc scratch");
        ck(cudaMalloc(&n->y, n->nv[0] * sizeof(float)), "cudaMalloc output");
        ck(cudaMalloc(&n->count, sizeof(unsigned long long)), "cudaMalloc");
        ck(cudaMalloc(&n->loss, sizeof(double)), "cudaMalloc");
        ck(cudaMalloc(&n->status, sizeof(int)), "cudaMalloc");
        if (st == PCT_OK) {
            ck(cudaMemcpyAsync(n->params, h.data(), pbytes, cudaMemcpyHostToDevice, n->stream), "params copy");
            ck(cudaMemsetAsync(n->adam_m, 0, pbytes, n->stream), "memset");
            ck(cudaMemsetAsync(n->adam_v, 0, pbytes, n->stream), "memset");
            ck(cudaMemsetAsync(n->status, 0, sizeof(int), n->stream), "memset");
            if (st == PCT_OK) st = emit_weights(n, n->stream);
            ck(cudaStreamSynchronize(n->stream), "synchronize");
        }
    }
    if (st != PCT_OK) {
        const cudaError_t e = cudaGetLastError();
        (void)e;
        release(n);
        delete n;
        return st;
    }
    *out = n;
    return PCT_OK;
}

pct_status pct_unet_destroy(pct_unet* n)
{
    if (!n) return PCT_OK;
    cudaSetDevice(n->device);
    if (n->stream) cudaStreamSynchronize(n->stream);
    release(n);
    delete n;
    return PCT_OK;
}

const char* pct_unet_last_error(const pct_unet* n) { return n ? n->err.c_str() : "null network"; }

pct_status pct_unet_param_count(const pct_unet* n, int64_t* count)
{
    if (!n || !count) return PCT_ERR_ARG;
    *count = static_cast<int64_t>(n->n_params);
    return PCT_OK;
}

pct_status pct_unet_get_params(pct_unet* n, float* host, int64_t count)
{
    if (!n || !host || count != static_cast<int64_t>(n->n_params)) return fail(n, PCT_ERR_ARG, "parameter count");
    UNET_CK(cudaSetDevice(n->device), "cudaSetDevice");
    UNET_CK(cudaMemcpyAsync(host, n->params, n->n_params * sizeof(float), cudaMemcpyDeviceToHost, n->stream), "copy");
    UNET_CK(cudaStreamSynchronize(n->stream), "synchronize");
    return PCT_OK;
}

pct_status pct_unet_set_params(pct_unet* n, const float* host, int64_t count)
{
    if (!n || !host || count != static_cast<int64_t>(n->n_params)) return fail(n, PCT_ERR_ARG, "parameter count");
    UNET_CK(cudaSetDevice(n->device), "cudaSetDevice");
    UNET_CK(cudaMemcpyAsync(n->params, host, n->n_params * sizeof(float), cudaMemcpyHostToDevice, n->stream), "copy");
    UNET_CK(cudaMemsetAsync(n->adam_m, 0, n->n_params * sizeof(float), n->stream), "memset");
    UNET_CK(cudaMemsetAsync(n->adam_v, 0, n->n_params * sizeof(float), n->stream), "memset");
    n->step = 0;
    const pct_status st = emit_weights(n, n->stream);
    if (st != PCT_OK) return st;
    UNET_CK(cudaStreamSynchronize(n->stream), "synchronize");
    return PCT_OK;
}

pct_status pct_unet_forward(pct_unet* n, const float* x0, const uint8_t* hull, float* image)
{
    if (!n || !x0 || !hull || !image) return fail(n, PCT_ERR_ARG, "null pointer");
    UNET_CK(cudaSetDevice(n->device), "cudaSetDevice");
    UNET_CK(cudaMemsetAsync(n->status, 0, sizeof(int), n->stream), "status clear");
    const pct_status st = forward(n, x0, hull, image, n->stream);
    if (st != PCT_OK) return st;
    return check_status(n, n->stream);
}

pct_status pct_unet_gradients(pct_unet* n, const float* x0, const uint8_t* hull, const float* target, float* grads_host,
                              double* loss)
{
    if (!n || !x0 || !hull || !target) return fail(n, PCT_ERR_ARG, "null pointer");
    UNET_CK(cudaSetDevice(n->device), "cudaSetDevice");
    const pct_status st = loss_and_gradient(n, x0, hull, target, loss, n->stream);
    if (st != PCT_OK) return st;
    if (grads_host) {
        UNET_CK(cudaMemcpyAsync(grads_host, n->grads, n->n_params * sizeof(float), cudaMemcpyDeviceToHost, n->stream),
                "gradient copy");
        UNET_CK(cudaStreamSynchronize(n->stream), "synchronize");
    }
    return PCT_OK;
}

pct_status pct_unet_train_step(pct_unet* n, const float* x0, const uint8_t* hull, const float* target, float lr,
                               double* loss)
{
    if (!n || !x0 || !hull || !target || !(lr > 0.f)) return fail(n, PCT_ERR_ARG, "invalid argument");
    UNET_CK(cudaSetDevice(n->device), "cudaSetDevice");
    pct_status st = loss_and_gradient(n, x0, hull, target, loss, n->stream);
    if (st != PCT_OK) return st;
    n->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float bc1 = 1.f - std::pow(b1, static_cast<float>(n->step));
    const float bc2 = 1.f - std::pow(b2, static_cast<float>(n->step));
    adam_kernel<<<grid_for(static_cast<long long>(n->n_params), 256), 256, 0, n->stream>>>(
        n->params, n->grads, n->adam_m, n->adam_v, static_cast<long long>(n->n_params), lr, b1, b2, 1e-8f, bc1, bc2);
    UNET_CK(cudaGetLastError(), "adam_kernel");
    st = emit_weights(n, n->stream);
    if (st != PCT_OK) return st;
    UNET_CK(cudaStreamSynchronize(n->stream), "synchronize");
    return PCT_OK;
}

pct_status pct_learned_initial_iterate(pct_ctx* ctx, pct_unet* n)
{
    if (!ctx || !n) return PCT_ERR_ARG;
    const pct::Geometry& g = ctx->geo;
    if (g.columns != n->nx[0] || g.rows != n->ny[0] || g.slices != n->nz[0]) {
        pct::context_set_error(ctx, "pct_learned_initial_iterate: network grid differs from the context's");
        return PCT_ERR_ARG;
    }
    const uint8_t* hull = pct::preproc_hull(ctx);
    if (!hull || !ctx->d_x) {
        pct::context_set_error(ctx, "pct_learned_initial_iterate: needs the hull and x_0 (run preprocessing first)");
        return PCT_ERR_STATE;
    }
    if (n->device != ctx->device) {
        pct::context_set_error(ctx, "pct_learned_initial_iterate: network and context on different devices");
        return PCT_ERR_ARG;
    }
    // image = x_0 + hull * network(x_0, hull) into the network's output buffer; it replaces the
    // context's image only if every voxel is finite, otherwise the FBP start x_0 is kept.
    cudaMemsetAsync(n->status, 0, sizeof(int), ctx->stream);
    pct_status st = forward(n, ctx->d_x, hull, n->y, ctx->stream);
    if (st == PCT_OK) {
        cudaMemsetAsync(n->count, 0, sizeof(unsigned long long), ctx->stream);
        nonfinite_kernel<<<grid_for(n->nv[0], 256), 256, 0, ctx->stream>>>(n->y, n->nv[0], n->count);
        unsigned long long bad = 0;
        cudaMemcpyAsync(&bad, n->count, sizeof(bad), cudaMemcpyDeviceToHost, ctx->stream);
        st = check_status(n, ctx->stream);
        if (st == PCT_OK && bad) st = fail(n, PCT_ERR_STATE, std::to_string(bad) + " non-finite voxels; the FBP start is kept");
        if (st == PCT_OK) {
            const cudaError_t e = cudaMemcpyAsync(ctx->d_x, n->y, n->nv[0] * sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream);
            if (e != cudaSuccess) st = cuda_fail(n, e, "image copy");
        }
    }
    if (st != PCT_OK) pct::context_set_error(ctx, ("pct_learned_initial_iterate: " + n->err).c_str());
    return st;
}

// ---------------------------------------------------------------- single convolutions --

}  // extern "C"

namespace {

// The status words of single convolutions: a fixed array on each device, a word claimed per call.
// (Allocated and freed per call they took 0.7 ms of a 0.1 ms convolution, and up to 16 ms next to another
// allocator's traffic: both wait for the device.)  More calls at once than words allocate theirs.
constexpr int kStatusWords = 64, kStatusDevices = 64;
__device__ int status_words[kStatusWords];
std::atomic<unsigned long long> status_claimed[kStatusDevices];

struct StatusWord {
    int* word = nullptr;
    StatusWord()
    {
        int dev = 0;
        void* base = nullptr;
        if (cudaGetDevice(&dev) != cudaSuccess) return;
        if (dev < kStatusDevices && cudaGetSymbolAddress(&base, status_words) == cudaSuccess) {
            unsigned long long have = status_claimed[dev].load();
            while (~have != 0) {
                const int free = __builtin_ctzll(~have);
                if (status_claimed[dev].compare_exchange_weak(have, have | 1ull << free)) {
                    word = static_cast<int*>(base) + free;
                    index_ = free;
                    device_ = dev;
                    return;
                }
            }
        }
        if (cudaMalloc(&word, sizeof(int)) != cudaSuccess) word = nullptr;
    }
    ~StatusWord()
    {
        if (index_ >= 0) status_claimed[device_].fetch_and(~(1ull << index_));
        else if (word) cudaFree(word);
    }
    StatusWord(const StatusWord&) = delete;
    StatusWord& operator=(const StatusWord&) = delete;

private:
    int index_ = -1, device_ = 0;
};

// Runs `launch` with a cleared status word on s and waits for it.
template <class Launch>
pct_status run_single(cudaStream_t s, const Launch& launch)
{
    StatusWord status;
    if (!status.word) return PCT_ERR_NOMEM;
    int h = 0;
    if (cudaMemsetAsync(status.word, 0, sizeof(int), s) != cudaSuccess || launch(status.word) != cudaSuccess ||
        cudaMemcpyAsync(&h, status.word, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess)
        h = -1;
    if (cudaStreamSynchronize(s) != cudaSuccess || h < 0) return PCT_ERR_CUDA;
    return h ? PCT_ERR_TIMEOUT : PCT_OK;
}

}  // namespace

extern "C" {

pct_status pct_conv3d_bf16(const uint16_t* in, int cin, int columns, int rows, int slices, int upsample,
                           const uint16_t* weight, int cout, const float* bias, const uint16_t* residual,
                           const uint16_t* mask, int relu, uint16_t* out, void* stream)
{
    if (!in || !weight || !out || !valid_channels(cin) || !valid_channels(cout) || columns <= 0 || rows <= 0 ||
        slices <= 0 || (upsample && (columns % 2 || rows % 2 || slices % 2)))
        return PCT_ERR_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    ConvFwdArgs a{};
    a.in = reinterpret_cast<const bf16*>(in);
    a.cin = cin;
    a.up = upsample ? 1 : 0;
    a.weight = reinterpret_cast<const bf16*>(weight);
    a.cout = cout;
    a.nx = columns;
    a.ny = rows;
    a.nz = slices;
    a.bias = bias;
    a.residual = reinterpret_cast<const bf16*>(residual);
    a.mask = reinterpret_cast<const bf16*>(mask);
    a.relu = relu;
    a.out = reinterpret_cast<bf16*>(out);
    return run_single(s, [&](int* status) {
        a.status = status;
        return launch_conv_fwd(a, s);
    });
}

pct_status pct_conv3d_bf16_wgrad(const uint16_t* in, int cin, int columns, int rows, int slices, int upsample,
                                 const uint16_t* dz, int cout, float* dweight, void* stream)
{
    if (!in || !dz || !dweight || !valid_channels(cin) || !valid_channels(cout) || columns <= 0 || rows <= 0 ||
        slices <= 0 || (upsample && (columns % 2 || rows % 2 || slices % 2)) ||
        static_cast<long long>(columns) * rows * slices > 0x7fffffffLL)
        return PCT_ERR_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    ConvWgradArgs a{};
    a.in = reinterpret_cast<const bf16*>(in);
    a.cin = cin;
    a.up = upsample ? 1 : 0;
    a.dz = reinterpret_cast<const bf16*>(dz);
    a.cout = cout;
    a.nx = columns;
    a.ny = rows;
    a.nz = slices;
    a.dw = dweight;
    return run_single(s, [&](int* status) {
        a.status = status;
        return launch_conv_wgrad(a, s);
    });
}

}  // extern "C"
