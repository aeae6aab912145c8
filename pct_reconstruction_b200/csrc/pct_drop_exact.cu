// pct_drop_exact.cu -- DROP block kernel and MLP-path kernel, exact (FP64, reference-rounding)
// mode.  Compiled with -fmad=false (see pct_mlp.cuh).
//
// drop_block_exact_kernel fuses the reference's calculate_x_update_GPU (B.cu:9321-9380) and
// DROP_block_update_GPU (B.cu:9522-9536): one thread per history computes the MLP voxel list,
// the sum of x over it, the DROP update value
//     upd = L * ((WEPL - L*sum_x) / (powf(L,2)*n)) * lambda        (rounded to float)
// and, when n >= MIN_MLP_LENGTH, scatters (upd, 1) into the interleaved accumulator
// acc[v] = {x_update[v], S[v]} with one 8-byte vector reduction per path entry
// (red.global.add.v2.f32) instead of the reference's two scalar atomics.
#include "pct_kernels.h"
#include "pct_mlp.cuh"

namespace pct {

namespace {

__global__ void __launch_bounds__(128) drop_block_exact_kernel(Geometry g, Tables tab, const StepConst* __restrict__ steps,
                                                               int kmax, const float* __restrict__ x, float2* __restrict__ acc,
                                                               HistorySoA h, long long begin, long long count,
                                                               unsigned long long* counters)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const long long id = begin + i;
    uint32_t path[kPathCap];
    const WalkResult r = mlp_walk_exact<true>(
        g, tab, steps, kmax, x, __ldg(h.first_MLP_voxel + id), __ldg(h.x_entry + id), __ldg(h.y_entry + id),
        __ldg(h.z_entry + id), __ldg(h.x_exit + id), __ldg(h.y_exit + id), __ldg(h.z_exit + id),
        __ldg(h.xy_entry_angle + id), __ldg(h.xz_entry_angle + id), __ldg(h.xy_exit_angle + id),
        __ldg(h.xz_exit_angle + id), [&](int j, uint32_t v) { path[j] = v; });
    if (r.flags) count_flags(r.flags, counters);
    if (r.n < g.min_mlp_length) return;
    const double a_i_dot_a_i = r.aia * r.n;
    const double a_i_dot_x_k = r.axk * r.chord;
    if (g.s_curve) {
        // S_CURVE_ON (B.cu:9530-9531): s(k) * L * ((WEPL - a_i_dot_x_k) / a_i_dot_a_i) * lambda per entry
        const double q = ((double)__ldg(h.WEPL + id) - a_i_dot_x_k) / a_i_dot_a_i;
        for (int j = 0; j < r.n; j++) {
            const uint32_t v = path[j];
            const float s = __ldg(g.s_curve + s_curve_index(g, j, r.n));
            if (v < (uint32_t)g.padded_voxels)
                atomicAdd(acc + v, make_float2((float)((((double)s * r.chord) * q) * g.lambda), 1.0f));
        }
        return;
    }
    const float upd = (float)(r.chord * (((double)__ldg(h.WEPL + id) - a_i_dot_x_k) / a_i_dot_a_i) * g.lambda);
    const float2 add = make_float2(upd, 1.0f);
    for (int j = 0; j < r.n; j++) {
        const uint32_t v = path[j];
        if (v < (uint32_t)g.padded_voxels) atomicAdd(acc + v, add);
    }
}

template <bool kMixed>
__global__ void __launch_bounds__(128) mlp_paths_kernel(Geometry g, Tables tab, const StepConst* __restrict__ steps,
                                                        int kmax, const float* __restrict__ x, HistorySoA h,
                                                        long long begin, long long count, int stride,
                                                        uint32_t* __restrict__ counts, uint32_t* __restrict__ voxels,
                                                        double* __restrict__ chord, double* __restrict__ a_dot_x,
                                                        unsigned long long* counters)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const long long id = begin + i;
    uint32_t* row = voxels ? voxels + i * (long long)stride : nullptr;
    auto emit = [&](int j, uint32_t v) {
        if (row && j < stride) row[j] = v;
    };
    WalkResult r;
    if constexpr (kMixed)
        r = mlp_walk_mixed<true>(g, tab, steps, kmax, x, h.first_MLP_voxel[id], h.x_entry[id], h.y_entry[id],
                                 h.z_entry[id], h.x_exit[id], h.y_exit[id], h.z_exit[id], h.xy_entry_angle[id],
                                 h.xz_entry_angle[id], h.xy_exit_angle[id], h.xz_exit_angle[id], emit);
    else
        r = mlp_walk_exact<true>(g, tab, steps, kmax, x, h.first_MLP_voxel[id], h.x_entry[id], h.y_entry[id],
                                 h.z_entry[id], h.x_exit[id], h.y_exit[id], h.z_exit[id], h.xy_entry_angle[id],
                                 h.xz_entry_angle[id], h.xy_exit_angle[id], h.xz_exit_angle[id], emit);
    if (r.flags) count_flags(r.flags, counters);
    if (r.n > stride && voxels) atomicAdd(counters + kCntPathOverflow, 1ull);
    if (counts) counts[i] = (uint32_t)r.n;
    if (chord) chord[i] = r.chord;
    if (a_dot_x) a_dot_x[i] = r.axk;
}

// Loop trips of the MLP walk per history (the number of MLP points find_MLP_path_GPU_tabulated
// computes, B.cu:9159-9255): the walk's own setup and loop condition (depth_2_go > MLP_U_STEP,
// carried by repeated subtraction), without the point algebra.  The measurement of the path
// kernel's FP64 work multiplies these by the operations of one point.
__global__ void __launch_bounds__(128) mlp_steps_kernel(Geometry g, Tables tab, int kmax, HistorySoA h, long long begin,
                                                        long long count, int* __restrict__ steps)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const long long id = begin + i;
    double xy_entry = h.xy_entry_angle[id], xy_exit = h.xy_exit_angle[id];
    unsigned flags = 0;
    const MlpStart m = mlp_start(g, tab, h.x_entry[id], h.y_entry[id], h.z_entry[id], h.x_exit[id], h.y_exit[id],
                                 h.z_exit[id], xy_entry, xy_exit, h.xz_entry_angle[id], h.xz_exit_angle[id], flags);
    double depth_2_go = m.depth_2_go;
    int k = 1;
    while (m.tables_ok && depth_2_go > g.mlp_u_step && k <= kmax) {
        depth_2_go -= g.mlp_u_step;
        k++;
    }
    steps[i] = k - 1;
}

// Exact and mixed-precision MLP points of the same steps side by side (the precision report):
// per history the largest |t_mixed - t_exact| and |v_mixed - v_exact| (cm) and the number of steps
// whose voxel differs, over the steps where the reference's Sigma_2 is well conditioned
// (1 - rho^2 > 1e-3); the other steps are counted in ill_posed.  Near the exit the tabulated Sigma_2 moments cancel to
// noise (u_2 enters the polynomials at its table grid point but the u_2 factors exactly), the
// determinant goes non-positive and the reference's point there is arbitrary in any precision.
__global__ void __launch_bounds__(128) mlp_precision_kernel(Geometry g, Tables tab, const StepConst* __restrict__ steps,
                                                            int kmax, HistorySoA h, long long begin, long long count,
                                                            double* __restrict__ dev_t, double* __restrict__ dev_v,
                                                            int* __restrict__ mismatched, int* __restrict__ ill_posed)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const long long id = begin + i;
    unsigned flags = 0;
    double xy_entry = h.xy_entry_angle[id], xy_exit = h.xy_exit_angle[id];
    MlpStart m = mlp_start(g, tab, h.x_entry[id], h.y_entry[id], h.z_entry[id], h.x_exit[id], h.y_exit[id],
                           h.z_exit[id], xy_entry, xy_exit, h.xz_entry_angle[id], h.xz_exit_angle[id], flags);
    const MlpHistoryF hf = mlp_history_f(m.h);
    const double s = g.mlp_u_step;
    double depth_2_go = m.depth_2_go, u_shifted = m.u_shifted, dt = 0.0, dv = 0.0;
    unsigned sigma_2_index = m.sigma_2_index;
    int bad = 0, ill = 0;
    for (int k = 1; m.tables_ok && depth_2_go > s && k <= kmax; k++) {
        double te, ve;
        float tm, vm;
        const StepConst& st = steps[k];
        mlp_point(m.h, st, tab.scattering_table, depth_2_go, sigma_2_index, te, ve);
        mlp_point_mixed(m.h, hf, st, tab.scattering_table, depth_2_go, sigma_2_index,
                        mixed_fp64_inverse(g, k, depth_2_go), tm, vm);
        u_shifted += s;
        // the reference's Sigma_2 determinant at this step (B.cu:9197)
        const MlpHistory& q = m.h;
        const double sigma_t2 = q.u_2_poly_3_12 - q.u_2_sq * st.p12 + q.two_u_2 * st.p23 - st.p34;
        const double sigma_t2_theta2 = q.u_2_poly_2_6 - q.u_2 * st.p12 + st.p23;
        const double sigma_theta2 = q.u_2_poly_1_2 - st.p12;
        // well posed: 1 - rho^2 of Sigma_2 above 1e-3 (its value for the scattering model is about 1/4)
        const double prod = sigma_t2 * sigma_theta2;
        if (sigma_theta2 > 0.0 && prod > 0.0 && prod - powf_square(sigma_t2_theta2) > 1e-3 * prod) {
            dt = fmax(dt, fabs((double)tm - te));
            dv = fmax(dv, fabs((double)vm - ve));
            if (mlp_voxel(g, m.h, u_shifted, te, ve) != mlp_voxel_mixed(g, hf, (float)u_shifted, tm, vm)) bad++;
        } else {
            ill++;
        }
        depth_2_go -= s;
        sigma_2_index -= g.sigma_index_step;
    }
    dev_t[i] = dt;
    dev_v[i] = dv;
    mismatched[i] = bad;
    ill_posed[i] = ill;
}

// ---- two-phase DROP iteration -------------------------------------------------------------
// Phase 1 (x-independent): every covered history's MLP voxel list is written to path storage.
// Phase 2 (per DROP block): gather x over the stored list, the DROP update, and the scatter.

// The path kernel's inputs in its processing order: dst[p] = src[perm[p]] (the ten geometry fields
// and the first voxel), with the path bound and the path-storage offset of the same history.
__global__ void gather_path_inputs_kernel(HistorySoA src, const int* __restrict__ perm, const int* __restrict__ bounds,
                                          const long long* __restrict__ offsets, long long n, HistorySoA dst,
                                          int* __restrict__ bounds_sorted, long long* __restrict__ offsets_sorted)
{
    const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const long long id = perm[p];
    dst.x_entry[p] = src.x_entry[id];
    dst.y_entry[p] = src.y_entry[id];
    dst.z_entry[p] = src.z_entry[id];
    dst.x_exit[p] = src.x_exit[id];
    dst.y_exit[p] = src.y_exit[id];
    dst.z_exit[p] = src.z_exit[id];
    dst.xy_entry_angle[p] = src.xy_entry_angle[id];
    dst.xz_entry_angle[p] = src.xz_entry_angle[id];
    dst.xy_exit_angle[p] = src.xy_exit_angle[id];
    dst.xz_exit_angle[p] = src.xz_exit_angle[id];
    dst.first_MLP_voxel[p] = src.first_MLP_voxel[id];
    bounds_sorted[p] = bounds[id];
    offsets_sorted[p] = offsets[id];
}

// Upper bound on the voxel-list length of each history (0 for histories the block launch does
// not cover): the loop runs at most u_2/MLP_U_STEP + 1 times and adds at most one entry per run.
// Rounded up to a multiple of kPathChunk entries so every history's slot starts on a 32-byte
// boundary and the path kernel writes whole sectors.
// The sorting key is the history's bucket of u_2 in the table of MLP weights (key_scale buckets per
// cm), so that histories of one bucket read the same rows; without a table (key_scale 0), the bound.
__global__ void path_bounds_kernel(Geometry g, Tables tab, HistorySoA h, long long n, long long block_size,
                                   int histories_per_block, double key_scale, int* __restrict__ bounds,
                                   int* __restrict__ keys)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long blk = i / block_size, pos = i - blk * block_size;
    long long hp = n - blk * block_size;
    if (hp > block_size) hp = block_size;
    const long long covered = histories_per_block > 0 ? (hp / histories_per_block) * histories_per_block : hp;
    int bound = 0, key = 0;
    if (pos < covered) {
        const double u_2 = mlp_u_extent(g, tab, h.x_entry[i], h.y_entry[i], h.x_exit[i], h.y_exit[i], h.xy_entry_angle[i]);
        const double q = u_2 / g.mlp_u_step;
        bound = (q >= 0 && q < (double)(kPathCap - 3)) ? (int)q + 3 : kPathCap;
        bound = (bound + kPathChunk - 1) / kPathChunk * kPathChunk;
        const double kq = u_2 * key_scale;
        key = key_scale <= 0.0 ? bound : (kq >= 0 && kq < (double)(kPathCap - 1)) ? (int)kq + 1 : kPathCap;
    }
    bounds[i] = bound;
    keys[i] = key;
}

// Launch shape of the table path kernel.  It is bound by instruction issue (about 80 instructions per
// point, 71% of the issue slots, load/store data stage 66%, FP64 pipe 4%) and takes 3.30 ms per 4M head
// histories, 0.263 ms per 600k of the small configuration; the walk that evaluated every point in
// double took 11.3 and 1.0 ms.  Resident 128-thread CTAs per SM (ms, 4M head): 6 3.55, 7 3.30, 8 3.43,
// 10 3.73: from 8 on the registers of the general points' set-up spill.
#ifndef PCT_PHASE1_MIN_BLOCKS
#define PCT_PHASE1_MIN_BLOCKS 7
#endif
// The path kernel of FP32 points keeps 8 CTAs (64 registers), as measured when it was tuned.
#ifndef PCT_PHASE1_MIXED_MIN_BLOCKS
#define PCT_PHASE1_MIXED_MIN_BLOCKS 8
#endif
// kThreads histories per CTA (PATH_CTA_THREADS), with the same resident threads per SM, hence the
// same register budget, at every size.  Position i of the processing order: its inputs at i (gathered
// into this order), its history id for the outputs.
template <int kThreads>
__global__ void __launch_bounds__(kThreads, PCT_PHASE1_MIN_BLOCKS * 128 / kThreads) mlp_phase1_table_kernel(
    const __grid_constant__ Geometry g, const __grid_constant__ Tables tab, const __grid_constant__ MlpTable tb,
    const StepConst* __restrict__ steps, int kmax, const __grid_constant__ HistorySoA h, const int* __restrict__ perm,
    long long count, const long long* __restrict__ offsets, long long offset_base, const int* __restrict__ bounds,
    uint32_t* __restrict__ paths, int* __restrict__ path_n, double* __restrict__ chord, unsigned long long* counters)
{
    __shared__ __align__(16) uint32_t stage[kThreads * kStageStride];
    const int i = blockIdx.x * kThreads + threadIdx.x;
    int cap = 0;
    uint32_t* out = nullptr;
    double* to_chord = nullptr;
    if (i < count) {
        cap = bounds[i];
        out = paths + (offsets[i] - offset_base);
        to_chord = chord + perm[i];
        if (cap <= 0) *to_chord = 0.0;  // not covered by its DROP block: no path
    }
    unsigned flags = 0;
    int n = mlp_walk_table(g, tab, tb, steps, kmax, h, i, cap,
                           (uint32_t)__cvta_generic_to_shared(stage + threadIdx.x * kStageStride), out, to_chord, &flags);
    if (i >= count) return;
    if (flags) count_flags(flags, counters);
    path_n[perm[i]] = n;
}

// Without a table: reference-order points.  Without the certain points' code in it, they take 10.11 ms for 3M head
// histories (11.04 with it, chosen at run time; 10.46 with 6 CTAs per SM, 10.22 with 8).
// kTryFast: a grid too large for the fixed-point positions.  The certain points need more registers than 7 CTAs
// have: the history's constants and its chord wait in shared memory, and the list leaves it in sectors of 8
// entries.  500k histories on 1100x1100x8 voxels: 1.83 ms; with the constants in registers and each entry stored
// by itself 2.22 (2.14 with 6 CTAs per SM, 2.23 with 5, 2.39 with 4).
template <int kThreads, bool kTryFast>
__global__ void __launch_bounds__(kThreads, 7 * 128 / kThreads) mlp_phase1_exact_kernel(
    Geometry g, Tables tab, const StepConst* __restrict__ steps, int kmax, HistorySoA h, const int* __restrict__ perm,
    long long count, const long long* __restrict__ offsets, long long offset_base, const int* __restrict__ bounds,
    uint32_t* __restrict__ paths, int* __restrict__ path_n, double* __restrict__ chord, unsigned long long* counters)
{
    constexpr int kPark = kTryFast ? kThreads * (int)sizeof(double) : 0;
    __shared__ double park[kTryFast ? (kHistoryFields + 1) * kThreads : 1];
    __shared__ uint32_t stage[kTryFast ? kThreads * (kPathChunk + 1) : 1];  // odd stride in words: no bank conflicts
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const long long id = perm[i];
    const int cap = bounds[i];
    if (cap <= 0) {
        path_n[id] = 0;
        chord[id] = 0.0;
        return;
    }
    uint32_t* out = paths + (offsets[i] - offset_base);  // 32-byte aligned, cap a multiple of 8
    uint32_t* mine = stage + (kTryFast ? threadIdx.x * (kPathChunk + 1) : 0);
    auto send = [&](int j0) {
        uint4* to = reinterpret_cast<uint4*>(out + j0);
        to[0] = make_uint4(mine[0], mine[1], mine[2], mine[3]);
        to[1] = make_uint4(mine[4], mine[5], mine[6], mine[7]);
    };
    const WalkResult r = mlp_walk_exact<false, kTryFast, kPark>(
        g, tab, steps, kmax, nullptr, __ldg(h.first_MLP_voxel + i), __ldg(h.x_entry + i), __ldg(h.y_entry + i),
        __ldg(h.z_entry + i), __ldg(h.x_exit + i), __ldg(h.y_exit + i), __ldg(h.z_exit + i),
        __ldg(h.xy_entry_angle + i), __ldg(h.xz_entry_angle + i), __ldg(h.xy_exit_angle + i),
        __ldg(h.xz_exit_angle + i), [&](int j, uint32_t v) {
            if (j >= cap) return;
            if (!kTryFast) {
                out[j] = v;
                return;
            }
            mine[j % kPathChunk] = v;
            if (j % kPathChunk == kPathChunk - 1) send(j - (kPathChunk - 1));
        }, (uint32_t)__cvta_generic_to_shared(park + (kTryFast ? threadIdx.x : 0)));
    unsigned flags = r.flags;
    int n = r.n;
    if (n > cap) {
        flags |= kFlagPathOverflow;
        n = cap;
    }
    if (kTryFast && n % kPathChunk) send(n - n % kPathChunk);  // the last sector, padded
    if (flags) count_flags(flags, counters);
    path_n[id] = n;
    chord[id] = r.chord;
}

// PRECISION MIXED or MIXED_COMPENSATED without a table.  With one, these modes take the table kernel
// too: its points are the exact ones and cost less (2M head histories 3.47 against 5.04 ms an iteration).
template <int kThreads>
__global__ void __launch_bounds__(kThreads, PCT_PHASE1_MIXED_MIN_BLOCKS * 128 / kThreads) mlp_phase1_mixed_kernel(
    Geometry g, Tables tab, const StepConst* __restrict__ steps, int kmax, HistorySoA h, const int* __restrict__ perm,
    long long count, const long long* __restrict__ offsets, long long offset_base, const int* __restrict__ bounds,
    uint32_t* __restrict__ paths, int* __restrict__ path_n, double* __restrict__ chord, unsigned long long* counters)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const long long id = perm[i];
    const int cap = bounds[i];
    if (cap <= 0) {
        path_n[id] = 0;
        chord[id] = 0.0;
        return;
    }
    uint32_t* out = paths + (offsets[i] - offset_base);
    const WalkResult r = mlp_walk_mixed<false>(
        g, tab, steps, kmax, nullptr, __ldg(h.first_MLP_voxel + i), __ldg(h.x_entry + i), __ldg(h.y_entry + i),
        __ldg(h.z_entry + i), __ldg(h.x_exit + i), __ldg(h.y_exit + i), __ldg(h.z_exit + i),
        __ldg(h.xy_entry_angle + i), __ldg(h.xz_entry_angle + i), __ldg(h.xy_exit_angle + i),
        __ldg(h.xz_exit_angle + i), [&](int j, uint32_t v) {
            if (j < cap) out[j] = v;
        });
    unsigned flags = r.flags;
    int n = r.n;
    if (n > cap) {
        flags |= kFlagPathOverflow;
        n = cap;
    }
    if (flags) count_flags(flags, counters);
    path_n[id] = n;
    chord[id] = r.chord;
}

// One warp per history.  Lane l holds entries l, l+32, ..., l+224 of the stored voxel list in
// registers: they are loaded once (eight independent loads in flight per lane), gathered for
// the sum of x, and reused for the scatter; longer lists stream their tail from memory twice.
//
// kAlgo selects the update: PCT_DROP (DROP_block_update_GPU B.cu:9522), PCT_ROBUSTA (a per-voxel
// perturbation Psi_j = (1 - x_j) ETA PSI_SIGN of the denominator, DROP_blocks_robust1 O.cu:7537)
// or PCT_ROBUSTB (the DROP update plus ||a||^2 per voxel into normA, DROP_blocks_robust2
// O.cu:7554).
//
// kMixed (PRECISION MIXED = 1 or MIXED_COMPENSATED = 2, PCT_DROP) runs the DROP arithmetic in FP32
// with compensation: each lane sums its entries of x with TwoSum (a float sum and its exact
// rounding error), the warp reduces the (sum, error) pairs with TwoSum, the residual WEPL - L*sum
// is formed from the exact product error (an FMA), and the update is a float expression of the
// float chord.  The scatter then adds (update, 1) to the float accumulator as the exact mode does.
// With 2 it instead returns each accumulator's old value, recomputes the float addition locally
// and adds its exact rounding error into a second per-voxel float array (comp), so a block's
// per-voxel partial sum is held as hi + lo and the image update applies (hi + lo) / S; that costs
// a returning atomic and a second reduction per entry.
//
// kSCurve (S_CURVE_ON, exact PCT_DROP only) scales the update of entry j by the S-curve table's
// s(k), k = s_curve_index(j, n), in the reference's order s * L * q * lambda (B.cu:9530-9531).
// Its launch bound asks for 6 CTAs per SM, which holds it to 40 registers without spills (48
// unbounded): the kernel is bound by the latency of its L2 reductions, so it keeps the warps per
// SM of the plain instantiations (39 registers, 6 CTAs).  A minimum of 0 leaves the others as
// they are (a minimum of 1 moves them to 48 registers).
//
// kMany: blocks of many histories, where warps that wait for the L2 are replaced by others rather than by
// loads ahead.  Measured, ms per iteration of 4M head histories in blocks of 60000 (2M for FP32 updates;
// 1M in blocks of 10000 / 3200 in brackets):
//   double updates: 4 entries in registers (32, 8 CTAs) 6.39, 8 entries 6.56 (2.603, 2.595 / 3.99, 3.79)
//   FP32 updates:   8 CTAs per SM 3.17, 6 CTAs 3.28 (2.463, 2.524 / 3.86, 3.70)
// Small blocks keep the entries that are loaded before the wait.  The lines: double updates from 256
// histories per SM (1M in blocks of 20000: 2.211 with 4 entries, 2.205 with 8), FP32 from 64.
constexpr int kManyDouble = 256, kManyFloat = 64;

// TwoSum (Knuth): s = RN(a + b) and the exact error e with a + b = s + e, six float operations.
__device__ __forceinline__ float two_sum(float a, float b, float& e)
{
    const float s = __fadd_rn(a, b);
    const float bp = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
    return s;
}

// x is read as ordinary memory: the image update before this kernel writes it while this kernel's CTAs are
// already there (they wait), and the read-only path wants data that no one writes while the kernel lives.
template <int kAlgo, bool kDet, int kMixed, bool kSCurve = false, bool kMany = false>
__global__ void __launch_bounds__(256, kSCurve ? 6 : kMany && kMixed ? 8 : 0) drop_phase2_kernel(Geometry g, const float* x, float2* __restrict__ acc,
                                                          float* __restrict__ normA, FixedAcc fx,
                                                          const float* __restrict__ WEPL,
                                                          const long long* __restrict__ offsets, long long offset_base,
                                                          const uint32_t* __restrict__ paths, const int* __restrict__ path_n,
                                                          const double* __restrict__ chord, long long begin, long long count)
{
    constexpr int kRegEntries = kMany && !kMixed ? 4 : 8;
    allow_dependent_launch();
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= count) return;
    // The voxel lists were written by the path kernel, which completed before the first block
    // kernel of this run started (a full dependency), so they are read before the wait.
    const long long id = begin + w;
    const int n = path_n[id];
    const uint32_t* p = paths + (offsets[id] - offset_base);
    const uint32_t npad = (uint32_t)g.padded_voxels;
    uint32_t v[kRegEntries];
#pragma unroll
    for (int m = 0; m < kRegEntries; m++) {
        const int j = lane + 32 * m;
        v[m] = j < n ? __ldg(p + j) : 0xffffffffu;
    }
    grid_dependency_wait();  // the previous block's image update has landed
    if constexpr (kMixed != 0 && kAlgo == PCT_DROP) {
        float hi = 0.0f, lo = 0.0f, e;
#pragma unroll
        for (int m = 0; m < kRegEntries; m++)
            if (v[m] < npad) {
                hi = two_sum(hi, x[v[m]], e);
                lo = __fadd_rn(lo, e);
            }
        for (int j = lane + 32 * kRegEntries; j < n; j += 32) {
            const uint32_t u = __ldg(p + j);
            if (u < npad) {
                hi = two_sum(hi, x[u], e);
                lo = __fadd_rn(lo, e);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float h2 = __shfl_xor_sync(0xffffffffu, hi, o), l2 = __shfl_xor_sync(0xffffffffu, lo, o);
            hi = two_sum(hi, h2, e);
            lo = __fadd_rn(__fadd_rn(lo, l2), e);
        }
        if (n < g.min_mlp_length) return;
        // residual = WEPL - L * (hi + lo) with the product's rounding error recovered by an FMA
        const float L = (float)chord[id];
        const float prod = __fmul_rn(L, hi);
        const float prod_err = __fmaf_rn(L, hi, -prod);
        const float residual =
            __fsub_rn(__fsub_rn(__fsub_rn(__ldg(WEPL + id), prod), prod_err), __fmul_rn(L, lo));
        const float a_i_dot_a_i = __fmul_rn(__fmul_rn(L, L), (float)n);
        const float upd = __fmul_rn(__fmul_rn(L, __fdiv_rn(residual, a_i_dot_a_i)), (float)g.lambda);
        auto put = [&](uint32_t u) {
            if (kDet) {
                atomicAdd(fx.sum + u, (unsigned long long)__double2ll_rn((double)upd * kFixedScale));
                atomicAdd(fx.cnt + u, 1u);
            } else if (kMixed == 2) {
                const float2 old = atomicAdd(acc + u, make_float2(upd, 1.0f));
                float err;
                two_sum(old.x, upd, err);
                if (err != 0.0f) atomicAdd(normA + u, err);
            } else {
                atomicAdd(acc + u, make_float2(upd, 1.0f));
            }
        };
#pragma unroll
        for (int m = 0; m < kRegEntries; m++)
            if (v[m] < npad) put(v[m]);
        for (int j = lane + 32 * kRegEntries; j < n; j += 32) {
            const uint32_t u = __ldg(p + j);
            if (u < npad) put(u);
        }
        return;
    }
    double sum = 0.0;
#pragma unroll
    for (int m = 0; m < kRegEntries; m++)
        if (v[m] < npad) sum += (double)x[v[m]];
    for (int j = lane + 32 * kRegEntries; j < n; j += 32) {
        const uint32_t u = __ldg(p + j);
        if (u < npad) sum += (double)x[u];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (n < g.min_mlp_length) return;
    const double L = chord[id];
    // one path entry's contribution: a float update and a count
    auto put = [&](uint32_t u, float upd) {
        if (kDet) {
            atomicAdd(fx.sum + u, (unsigned long long)__double2ll_rn((double)upd * kFixedScale));
            atomicAdd(fx.cnt + u, 1u);
        } else {
            atomicAdd(acc + u, make_float2(upd, 1.0f));
        }
    };
    if (kAlgo == PCT_DROP && kSCurve) {
        const double a_i_dot_a_i = powf_square(L) * n;
        const double a_i_dot_x_k = sum * L;
        const double q = ((double)__ldg(WEPL + id) - a_i_dot_x_k) / a_i_dot_a_i;
        auto scaled = [&](int j) {
            const double s = (double)__ldg(g.s_curve + s_curve_index(g, j, n));
            return (float)(((s * L) * q) * g.lambda);
        };
#pragma unroll
        for (int m = 0; m < kRegEntries; m++)
            if (v[m] < npad) put(v[m], scaled(lane + 32 * m));
        for (int j = lane + 32 * kRegEntries; j < n; j += 32) {
            const uint32_t u = __ldg(p + j);
            if (u < npad) put(u, scaled(j));
        }
    } else if (kAlgo == PCT_DROP) {
        const double a_i_dot_a_i = powf_square(L) * n;
        const double a_i_dot_x_k = sum * L;
        const float upd = (float)(L * (((double)__ldg(WEPL + id) - a_i_dot_x_k) / a_i_dot_a_i) * g.lambda);
#pragma unroll
        for (int m = 0; m < kRegEntries; m++)
            if (v[m] < npad) put(v[m], upd);
        for (int j = lane + 32 * kRegEntries; j < n; j += 32) {
            const uint32_t u = __ldg(p + j);
            if (u < npad) put(u, upd);
        }
    } else if (kAlgo == PCT_ROBUSTA) {
        // update_j = LAMBDA * residual / (<a,a> + Psi_j), Psi_j = ((1 - x_j) * ETA) * PSI_SIGN
        const double a_i_dot_a_i = L * L * n;
        const double residual = (double)__ldg(WEPL + id) - sum * L;
        auto add = [&](uint32_t u) {
            const double psi = ((1.0 - (double)x[u]) * g.eta) * g.psi_sign;
            put(u, (float)(g.lambda * (residual / (a_i_dot_a_i + psi))));
        };
#pragma unroll
        for (int m = 0; m < kRegEntries; m++)
            if (v[m] < npad) add(v[m]);
        for (int j = lane + 32 * kRegEntries; j < n; j += 32) {
            const uint32_t u = __ldg(p + j);
            if (u < npad) add(u);
        }
    } else {  // PCT_ROBUSTB: update = L * LAMBDA * residual / <a,a>; normA_j += L^2 (float atomics)
        const double a_i_dot_a_i = L * L * n;
        const float upd = (float)(L * g.lambda * (((double)__ldg(WEPL + id) - sum * L) / a_i_dot_a_i));
        const float2 add = make_float2(upd, 1.0f);
        const float l2 = (float)(L * L);
#pragma unroll
        for (int m = 0; m < kRegEntries; m++)
            if (v[m] < npad) {
                atomicAdd(acc + v[m], add);
                atomicAdd(normA + v[m], l2);
            }
        for (int j = lane + 32 * kRegEntries; j < n; j += 32) {
            const uint32_t u = __ldg(p + j);
            if (u < npad) {
                atomicAdd(acc + u, add);
                atomicAdd(normA + u, l2);
            }
        }
    }
}

// Per-step table (see pct_tables.h): the u_1 polynomials and Sigma_1I of loop iteration k,
// evaluated on the device like the reference's loop does (B.cu:9180-9195, powf on the device).
__global__ void build_step_table_kernel(Tables tab, unsigned sstep, unsigned pstep, int kmax, StepConst* steps)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > kmax) return;
    StepConst e{};
    if (k >= 1) {
        const unsigned pi1 = (unsigned)k * pstep, si1 = (unsigned)k * sstep;
        const double p12 = tab.poly_1_2[pi1];
        const double sigma_t1 = tab.poly_3_12[pi1], sigma_t1_theta1 = tab.poly_2_6[pi1], sigma_theta1 = p12;
        const double det1 = tab.scattering_table[si1] * (sigma_t1 * sigma_theta1 - powf_square(sigma_t1_theta1));
        e.p12 = p12;
        e.p23 = tab.poly_2_3[pi1];
        e.p34 = tab.poly_3_4[pi1];
        e.s1i0 = sigma_theta1 / det1;
        e.s1i1 = sigma_t1_theta1 / det1;
        e.s1i2 = sigma_t1 / det1;
        e.s1i0f = (float)e.s1i0;
        e.s1i1f = (float)e.s1i1;
        e.s1i2f = (float)e.s1i2;
    }
    steps[k] = e;
}

// ---- the table of MLP weights (pct_mlp.cuh, "Tabulated points") --------------------------------

// Rows of bucket b (m buckets per MLP step): the steps k of a walk with u_2 inside the bucket, those with
// u_2 - k s > s; and the rows of the buckets before it.
__host__ __device__ inline int table_row_count(int b, int m) { return b / m > 1 ? b / m - 1 : 0; }
__host__ __device__ inline long long table_first_row(int b, int m)
{
    const long long f = b / m;  // whole groups of m buckets before it; group i has max(0, i - 1) rows each
    return (f > 2 ? (f - 2) * (f - 1) / 2 : 0) * m + (long long)(b % m) * table_row_count(b, m);
}

// The weights B and C of step k for u_2 = grid point idx + delta and u_2^2 + epsilon, with Sigma_2's
// determinant scaled by 1 + eta: the formulas of mlp_point_rest solved for the weights, in double.
struct WeightNode {
    double B, C;
    double mag_num, mag_det;  // M(num) / |det| per unit of scale and M(det) / |det| (mlp_point_fast)
    double ratio;             // sigma_t2_theta2^2 / |determinant of the moments|
};
__device__ WeightNode weight_node(const Tables& tab, const StepConst& st, double s, int k, unsigned sstep, long long idx,
                                  double delta, double epsilon, double eta)
{
    const double u_2 = idx * kPolyTableStep + delta, d = u_2 - k * s;
    const double t2 = tab.poly_3_12[idx] - (u_2 * u_2 + epsilon) * st.p12 + 2.0 * u_2 * st.p23 - st.p34;
    const double tt = tab.poly_2_6[idx] - u_2 * st.p12 + st.p23;
    const double th = tab.poly_1_2[idx] - st.p12;
    const double mdet = t2 * th - tt * tt;
    // the walk's index: of its first depth u_2 - s, then sstep less a step (an entry off is in eta)
    long long is = llrint((u_2 - s) / kCoeffTableStep) - (long long)(k - 1) * sstep;
    if (is < 0) is = 0;  // log of 0: the row comes out unusable
    const double det2 = tab.scattering_table[is] * mdet * (1.0 + eta);
    const double S0 = th / det2, S1 = tt / det2, S2 = t2 / det2;
    const double c = S0 * d - S1, m0 = st.s1i0 + S0, m1 = c - st.s1i1, m3 = st.s1i2 + S2 + d * (c - S1);
    const double det = m0 * m3 - m1 * m1;
    const double aS0 = fabs(S0), aS1 = fabs(S1), aS2 = fabs(S2), Mc = aS0 * d + aS1, M0 = fabs(st.s1i0) + aS0,
                 M1 = Mc + fabs(st.s1i1), M3 = fabs(st.s1i2) + aS2 + d * (Mc + aS1);
    WeightNode w;
    w.B = (m3 * S0 - m1 * c) / det;
    w.C = -(m3 * S1 + m1 * (S2 - d * S1)) / det;
    w.mag_num = (M3 * (M0 + aS1) + M1 * (M1 + d * aS1 + aS2)) / fabs(det);
    w.mag_det = (M0 * M3 + M1 * M1) / fabs(det);
    w.ratio = tt * tt / fabs(mdet);
    return w;
}

// Quadratic through (z0, f0), (zp, fp), (zm, fm) as coefficients of 1, z, z^2.
__device__ void quadratic(double z0, double f0, double zp, double fp, double zm, double fm, double (&c)[3])
{
    const double p = (fp - f0) / (zp - z0), q = (fm - f0) / (zm - z0);
    c[2] = (p - q) / (zp - zm);
    c[1] = p - c[2] * (z0 + zp);
    c[0] = f0 - p * z0 + c[2] * z0 * zp;
}

// One CTA per bucket, one thread per step.  A row is kept while its bound is useful (kMaxErrB,
// kMaxErrC: a few thousandths of a voxel face's neighbourhood at head-scan deflections); the first
// row that is not ends the bucket's table.
constexpr float kMaxErrB = 2.0e-5f, kMaxErrC = 1.0e-4f, kMaxErrR = 1.0e-7f;
__global__ void __launch_bounds__(128) build_mlp_table_kernel(Tables tab, const StepConst* __restrict__ steps, double s,
                                                              unsigned sstep, int m, double width, float4* __restrict__ rows,
                                                              MlpBucket* __restrict__ bucket)
{
    const int b = blockIdx.x, count = table_row_count(b, m);
    const long long first = table_first_row(b, m);
    __shared__ float e_b[kPathCap], e_c[kPathCap];
    __shared__ int bad, max_r, max_b, max_c, all_b, all_c;
    if (threadIdx.x == 0) {
        bad = count + 1;
        max_r = max_b = max_c = all_b = all_c = 0;
    }
    __syncthreads();
    const double center = (b + 0.5) * width;
    const long long ic = llrint(center / kPolyTableStep);
    const double kappa = count > 0 ? steps[count].p12 / (2.0 * tab.poly_2_6[ic] * count) : 0.0;
    const double eps_max = 3.0e-7 * (b + 1) * width * (b + 1) * width;  // powf of the float u_2
    for (int k = 1 + threadIdx.x; k <= count; k += blockDim.x) {
        const StepConst st = steps[k];
        auto node = [&](double z, double delta, double eps, double eta, double& zeta) {
            const long long idx = llrint((center + 0.5 * z * width - delta) / kPolyTableStep);
            zeta = ((idx * kPolyTableStep + delta) / width - b) * 2.0 - 1.0;
            return weight_node(tab, st, s, k, sstep, idx, delta, eps, eta);
        };
        double z0, zp, zm, za, zb, qb[3], qc[3];
        const WeightNode n0 = node(0.0, 0.0, 0.0, 0.0, z0), np = node(0.8660254, 0.0, 0.0, 0.0, zp),
                         nm = node(-0.8660254, 0.0, 0.0, 0.0, zm), na = node(0.0, kSigmaUnit, 0.0, 0.0, za),
                         nb = node(0.0, -kSigmaUnit, 0.0, 0.0, zb);
        quadratic(z0, n0.B, zp, np.B, zm, nm.B, qb);
        quadratic(z0, n0.C, zp, np.C, zm, nm.C, qc);
        auto at = [](const double (&c)[3], double z) { return c[0] + z * (c[1] + z * c[2]); };
        const float4 rb = make_float4((float)qb[0], (float)qb[1], (float)qb[2],
                                      (float)(0.5 * ((na.B - at(qb, za)) - (nb.B - at(qb, zb)))));
        const float4 rc = make_float4((float)qc[0], (float)qc[1], (float)qc[2],
                                      (float)(0.5 * ((na.C - at(qc, za)) - (nb.C - at(qc, zb)))));
        rows[2 * (first + k - 1)] = rb;
        rows[2 * (first + k - 1) + 1] = rc;
        double err_b = 0.0, err_c = 0.0, finite = 0.0;  // finite: NaN once a value is not
        for (int i = 0; i < 81; i++) {
            const double delta = (i / 9 % 3 - 1) * kSigmaUnit, eps = (i / 27 - 1) * eps_max;
            double zeta;
            const WeightNode w = node((i % 9 - 4) * 0.25, delta, eps, 0.0, zeta);
            const float z = (float)zeta, sigma = (float)((delta + k * kappa * eps) * kInvSigmaUnit);
            err_b = fmax(err_b, fabs((double)table_weight(rb, z, sigma) - w.B));
            err_c = fmax(err_c, fabs((double)table_weight(rc, z, sigma) - w.C));
            finite += 0.0 * (w.B + w.C + w.mag_num + w.mag_det);
        }
        double det_b = 0.0, det_c = 0.0;
        for (int i = -1; i <= 1; i++) {
            double ze;
            const WeightNode w = node(i, 0.0, 0.0, 0.0, ze);
            const WeightNode we = node(i, 0.0, 0.0, 4.0e-7 * w.ratio + 6.0e-6 / (center + 0.5 * i * width - k * s), ze);
            det_b = fmax(det_b, fabs(we.B - w.B));
            det_c = fmax(det_c, fabs(we.C - w.C));
            finite += 0.0 * (we.B + we.C);
        }
        const float eb = (float)(2.0 * (err_b + det_b) + finite), ec = (float)(2.0 * (err_c + det_c));
        const float er = (float)(kBoundK * (n0.mag_num + 2.0 * n0.mag_det) * 2.0);
        e_b[k - 1] = eb;
        e_c[k - 1] = ec;
        if (!(eb < kMaxErrB && ec < kMaxErrC && er < kMaxErrR)) atomicMin(&bad, k);
        else {
            atomicMax(&max_r, __float_as_int(er));  // non-negative floats compare as integers
            atomicMax(&max_b, __float_as_int(fabsf(rb.x) + fabsf(rb.y) + fabsf(rb.z)));
            atomicMax(&max_c, __float_as_int(fabsf(rc.x) + fabsf(rc.y) + fabsf(rc.z)));
        }
    }
    __syncthreads();
    for (int k = 1 + threadIdx.x; k < bad; k += blockDim.x) {
        atomicMax(&all_b, __float_as_int(e_b[k - 1]));
        atomicMax(&all_c, __float_as_int(e_c[k - 1]));
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        MlpBucket o;
        o.row = (int)first;
        o.klast = bad - 1;
        o.err_b = __int_as_float(all_b);
        o.err_c = __int_as_float(all_c);
        o.err_r = __int_as_float(max_r);
        o.max_b = __int_as_float(max_b);
        o.max_c = __int_as_float(max_c);
        o.steps = count;
        o.kappa = kappa;
        bucket[b] = o;
    }
}

}  // namespace

MlpTableShape mlp_table_shape(const Geometry& g, int kmax)
{
    MlpTableShape t{};
    const double s = g.mlp_u_step;
    if (!g.exact_fast_points) return t;
    // positions: frac_bits fraction bits, the rest for the grid and its surroundings
    int extent = g.columns > g.rows ? g.columns : g.rows;
    if (g.slices > extent) extent = g.slices;
    int bits = 22;
    while (bits > 18 && (1LL << (31 - bits)) < extent + 24) bits--;
    const long long top = 1LL << (31 - bits);
    if (top < extent + 24 || top * (1 + g.columns + (long long)g.columns * g.rows) > 0x7fffffffLL) return t;
    t.frac_bits = bits;
    t.per_step = (int)ceil(s / 0.05 - 1e-9);
    if (t.per_step < 1) t.per_step = 1;
    t.width = s / t.per_step;
    // u_2 of a history inside the grid's cylinder, inside the tables
    double u_max = 1.5 * extent * fmax(g.voxel_width, g.voxel_height) + 0.5;
    if (u_max > kPolyTableRange - 0.5) u_max = kPolyTableRange - 0.5;
    t.buckets = (int)(u_max / t.width);
    if (t.buckets > kPathCap) t.buckets = kPathCap;
    while (t.buckets > 0 && table_row_count(t.buckets - 1, t.per_step) > kmax) t.buckets--;
    t.rows = table_first_row(t.buckets, t.per_step);
    t.t_max = (float)(kMaxOffset / ((double)(1u << (bits - kOffsetShift)) * g.inv_voxel_max));
    return t;
}

cudaError_t launch_build_mlp_table(const Tables& tab, const StepConst* steps, const Geometry& g, const MlpTableShape& shape,
                                   float4* rows, MlpBucket* bucket, cudaStream_t stream)
{
    if (shape.buckets <= 0) return cudaSuccess;
    build_mlp_table_kernel<<<shape.buckets, 128, 0, stream>>>(tab, steps, g.mlp_u_step, g.sigma_index_step,
                                                              shape.per_step, shape.width, rows, bucket);
    return cudaGetLastError();
}

cudaError_t launch_build_step_table(const Tables& tab, unsigned sstep, unsigned pstep, int kmax, StepConst* steps,
                                    cudaStream_t stream)
{
    const int threads = 128;
    build_step_table_kernel<<<(kmax + threads) / threads, threads, 0, stream>>>(tab, sstep, pstep, kmax, steps);
    return cudaGetLastError();
}

cudaError_t launch_path_bounds(const Geometry& g, const Tables& tab, const HistorySoA& h, long long n,
                               long long block_size, int histories_per_block, double key_scale, int* bounds, int* keys,
                               cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    const int threads = 256;
    path_bounds_kernel<<<(unsigned)((n + threads - 1) / threads), threads, 0, stream>>>(
        g, tab, h, n, block_size, histories_per_block, key_scale, bounds, keys);
    return cudaGetLastError();
}

cudaError_t launch_gather_path_inputs(const HistorySoA& src, const int* perm, const int* bounds,
                                      const long long* offsets, long long n, const HistorySoA& dst, int* bounds_sorted,
                                      long long* offsets_sorted, cudaStream_t stream)
{
    if (n <= 0) return cudaSuccess;
    const int threads = 256;
    gather_path_inputs_kernel<<<(unsigned)((n + threads - 1) / threads), threads, 0, stream>>>(
        src, perm, bounds, offsets, n, dst, bounds_sorted, offsets_sorted);
    return cudaGetLastError();
}

cudaError_t launch_mlp_phase1_exact(const Geometry& g, const Tables& tab, const MlpTable& tb, const StepConst* steps,
                                    int kmax,
                                    const HistorySoA& h, const int* perm, long long count, const long long* offsets,
                                    long long offset_base, const int* bounds, uint32_t* paths, int* path_n,
                                    double* chord, unsigned long long* counters, cudaStream_t stream)
{
    if (count <= 0) return cudaSuccess;
    cudaError_t e = cudaSuccess;
#define PCT_PHASE1(T)                                                                                             \
    do {                                                                                                          \
        const unsigned blocks = (unsigned)((count + (T) - 1) / (T));                                              \
        auto launch = [&](auto kernel, auto... first) {                                                           \
            e = launch_carved_kernel(false, g.carveout, kernel, blocks, T, stream, first..., steps, kmax, h, perm, count, \
                                     offsets, offset_base, bounds, paths, path_n, chord, counters);               \
        };                                                                                                        \
        if (tb.buckets > 0) launch(mlp_phase1_table_kernel<T>, g, tab, tb);                                       \
        else if (g.mixed_precision) launch(mlp_phase1_mixed_kernel<T>, g, tab);                                   \
        else if (g.exact_fast_points) launch(mlp_phase1_exact_kernel<T, true>, g, tab);                           \
        else launch(mlp_phase1_exact_kernel<T, false>, g, tab);                                                   \
    } while (0)
    if (g.path_cta_threads == 64) PCT_PHASE1(64);
    else if (g.path_cta_threads == 256) PCT_PHASE1(256);
    else PCT_PHASE1(128);
#undef PCT_PHASE1
    return e;
}

cudaError_t launch_drop_phase2(const Geometry& g, const float* x, float2* acc, float* normA, const FixedAcc& fx,
                               const float* WEPL, const long long* offsets, long long offset_base,
                               const uint32_t* paths, const int* path_n, const double* chord, long long begin,
                               long long count, cudaStream_t stream, bool pdl)
{
    if (count <= 0) return cudaSuccess;
    const int threads = 256;
    const unsigned blocks = (unsigned)((count * 32 + threads - 1) / threads);
    cudaError_t e = cudaSuccess;
#define PCT_PHASE2(ALGO, DET, MIXED, SC, MANY)                                                              \
    e = launch_carved_kernel(pdl, g.carveout, drop_phase2_kernel<ALGO, DET, MIXED, SC, MANY>, blocks, threads, stream, \
                             g, x, acc, normA, fx, WEPL, offsets, offset_base, paths, path_n, chord, begin, count)
    const bool many = count >= (long long)sm_count() * (g.mixed_precision ? kManyFloat : kManyDouble);
    if (g.projection_algorithm == PCT_ROBUSTA) {
        if (g.deterministic) PCT_PHASE2(PCT_ROBUSTA, true, 0, false, false);
        else PCT_PHASE2(PCT_ROBUSTA, false, 0, false, false);
    } else if (g.projection_algorithm == PCT_ROBUSTB) {
        PCT_PHASE2(PCT_ROBUSTB, false, 0, false, false);
    } else if (g.mixed_precision) {
        if (g.deterministic) PCT_PHASE2(PCT_DROP, true, 1, false, false);  // fixed-point sums need no compensation
        else if (g.compensated) PCT_PHASE2(PCT_DROP, false, 2, false, false);
        else if (many) PCT_PHASE2(PCT_DROP, false, 1, false, true);
        else PCT_PHASE2(PCT_DROP, false, 1, false, false);
    } else if (g.s_curve) {
        if (g.deterministic) PCT_PHASE2(PCT_DROP, true, 0, true, false);
        else PCT_PHASE2(PCT_DROP, false, 0, true, false);
    } else {
        if (g.deterministic) PCT_PHASE2(PCT_DROP, true, 0, false, false);
        else if (many) PCT_PHASE2(PCT_DROP, false, 0, false, true);
        else PCT_PHASE2(PCT_DROP, false, 0, false, false);
    }
#undef PCT_PHASE2
    return e;
}

// The carve-out, in percent of the largest shared memory an SM offers (228 KB on B200).  An SM runs CTAs of
// kernels with different carve-outs only after it has drained and been reconfigured, so the block chain's small
// kernels, interleaved with path-kernel chunks, would wait for whole SMs to empty: all have the same.
//  * With the table 7 path CTAs keep 10 KB of list staging each, the rest is L1 for the table rows and the
//    gathers.  Measured on B200 (ms per iteration; 4M head / 600k small / 2M head mixed): 25% (6 path CTAs)
//    6.68 / 1.450 / 3.36, 35% 6.38 / 1.461 / 3.16, 40% 6.39 / 1.459 / 3.15, 45% 6.43 / 1.468 / 3.17, 58%
//    6.50 / 1.477 / 3.19, 75% 6.64 / 1.513 / 3.26, each kernel's own 6.73 / 2.261 / 3.37.
//  * FP32 points (mixed precision without the table) keep no shared memory: the driver's choice, all of it L1
//    for their table gathers.  2M head: 4.91 so, 25% 4.97, 40% 5.04, 58% 5.26.
//  * Certain points without the table keep 20.5 KB for each of 7 CTAs, which 58% holds (57% gives 6 CTAs).
int iteration_carveout(const Geometry& g, bool table)
{
    if (table) return 40;
    if (g.mixed_precision) return -1;
    return g.exact_fast_points ? 58 : 40;
}

cudaError_t launch_drop_block_exact(const Geometry& g, const Tables& tab, const StepConst* steps, int kmax,
                                    const float* x, float2* acc, const HistorySoA& h, long long begin,
                                    long long count, unsigned long long* counters, cudaStream_t stream)
{
    if (count <= 0) return cudaSuccess;
    const int threads = 128;
    const long long blocks = (count + threads - 1) / threads;
    drop_block_exact_kernel<<<(unsigned)blocks, threads, 0, stream>>>(g, tab, steps, kmax, x, acc, h, begin, count,
                                                                      counters);
    return cudaGetLastError();
}

cudaError_t launch_mlp_paths_exact(const Geometry& g, const Tables& tab, const StepConst* steps, int kmax,
                                   const float* x, const HistorySoA& h, long long begin, long long count, int stride,
                                   uint32_t* counts, uint32_t* voxels, double* chord, double* a_dot_x,
                                   unsigned long long* counters, bool fp32_points, cudaStream_t stream)
{
    if (count <= 0) return cudaSuccess;
    const int threads = 128;
    const long long blocks = (count + threads - 1) / threads;
    if (fp32_points)
        mlp_paths_kernel<true><<<(unsigned)blocks, threads, 0, stream>>>(g, tab, steps, kmax, x, h, begin, count,
                                                                         stride, counts, voxels, chord, a_dot_x,
                                                                         counters);
    else
        mlp_paths_kernel<false><<<(unsigned)blocks, threads, 0, stream>>>(g, tab, steps, kmax, x, h, begin, count,
                                                                          stride, counts, voxels, chord, a_dot_x,
                                                                          counters);
    return cudaGetLastError();
}

cudaError_t launch_mlp_steps(const Geometry& g, const Tables& tab, int kmax, const HistorySoA& h, long long begin,
                             long long count, int* steps, cudaStream_t stream)
{
    if (count <= 0) return cudaSuccess;
    const int threads = 128;
    const long long blocks = (count + threads - 1) / threads;
    mlp_steps_kernel<<<(unsigned)blocks, threads, 0, stream>>>(g, tab, kmax, h, begin, count, steps);
    return cudaGetLastError();
}

cudaError_t launch_mlp_precision(const Geometry& g, const Tables& tab, const StepConst* steps, int kmax,
                                 const HistorySoA& h, long long begin, long long count, double* dev_t, double* dev_v,
                                 int* mismatched, int* ill_posed, cudaStream_t stream)
{
    if (count <= 0) return cudaSuccess;
    const int threads = 128;
    mlp_precision_kernel<<<(unsigned)((count + threads - 1) / threads), threads, 0, stream>>>(
        g, tab, steps, kmax, h, begin, count, dev_t, dev_v, mismatched, ill_posed);
    return cudaGetLastError();
}

}  // namespace pct
