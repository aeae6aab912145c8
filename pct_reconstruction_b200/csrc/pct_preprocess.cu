// pct_preprocess.cu -- the stages that turn tracker data into reconstruction histories and the
// initial image: recon-volume intersections, binning, statistical cuts, sinogram, FBP, hull
// detection, initial iterate and the hull-entry/exit (MLP endpoint) search.
//
// Each kernel restates one reference kernel (B.cu line cited at the kernel) in the same double and
// float operations -- including where the reference calls float functions on float operands
// (atan2 on float differences resolves to atan2f, abs on a float to fabsf) and where it calls
// powf on doubles -- so integer results (bins, survivors, hull voxels, first MLP voxels) come out
// identical.  This translation unit is compiled with -fmad=false.
//
// Design differences from the reference, all of which leave results unchanged:
//  * all histories are resident in HBM: no MAX_GPU_HISTORIES chunking, no host round trips;
//  * the host-side compactions (std::vector push_back loops, B.cu:5429-5450, 5892-5911,
//    8286-8294) are stable device compactions (prefix sum + scatter), so the history order -- and
//    with it the DROP block composition -- is the reference's;
//  * the filter, backprojection and median filter accumulate each output in one thread in the
//    reference's loop order, so they are deterministic (the reference's atomicAdds there each
//    touch one thread's own element);
//  * MSC edge detection runs out of place with the in-place kernel's condition (B.cu:6911-6956
//    reads neighbours that other blocks may already have overwritten; the result here is the
//    one that kernel gives when none has been);
//  * the hull voxel walks stop when an index leaves the grid on either side and after a bounded
//    number of steps: the reference's SC/MSC/SM walks (B.cu:6681-7099) only test the upper bounds
//    and would run forever (writing out of bounds) on a walk that misses its exit voxel towards
//    negative indices; such walks are counted (counter "wait_expired").
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "pct_context.h"

namespace pct {

namespace {

constexpr double kPi = 3.141592653589793;      // 4*atan(1.0)
constexpr double kPiOver4 = 0.7853981633974483;  // atan(1.0)
constexpr double kPiOver2 = 1.5707963267948966;  // 2*atan(1.0)

// Reference macro values derived from the configuration, by value for kernels.
struct PreGeom {
    int columns, rows, slices, num_voxels;
    double voxel_width, voxel_height, voxel_thickness;
    double R, H;  // RECON_CYL_RADIUS, RECON_CYL_HEIGHT
    int t_bins, v_bins, angular_bins, num_bins;
    double t_bin_size, v_bin_size, angular_bin_size;
    int sigmas_to_keep, sample_std_dev;
    int sinogram_filter;
    double source_radius, rsp_air, fbp_threshold;
    double sc_lower, sc_upper, msc_lower, msc_upper, sm_lower, sm_scale;
    int msc_diff_thresh;
    int fast_walks;  // EXACT_FAST_POINTS: voxel walks by crossing times where the order is certain
};

PreGeom make_pregeom(const pct_config& c)
{
    PreGeom g{};
    g.columns = c.COLUMNS;
    g.rows = c.ROWS;
    g.slices = c.SLICES;
    g.num_voxels = c.NUM_VOXELS;
    g.voxel_width = c.VOXEL_WIDTH;
    g.voxel_height = c.VOXEL_HEIGHT;
    g.voxel_thickness = c.VOXEL_THICKNESS;
    g.R = c.RECON_CYL_RADIUS;
    g.H = c.RECON_CYL_HEIGHT;
    g.t_bins = c.T_BINS;
    g.v_bins = c.V_BINS;
    g.angular_bins = c.ANGULAR_BINS;
    g.num_bins = c.NUM_BINS;
    g.t_bin_size = c.T_BIN_SIZE;
    g.v_bin_size = c.V_BIN_SIZE;
    g.angular_bin_size = c.ANGULAR_BIN_SIZE;
    g.sigmas_to_keep = c.SIGMAS_TO_KEEP;
    g.sample_std_dev = c.SAMPLE_STD_DEV ? 1 : 0;
    g.sinogram_filter = c.SINOGRAM_FILTER;
    g.source_radius = c.SOURCE_RADIUS;
    g.rsp_air = c.RSP_AIR;
    g.fbp_threshold = c.FBP_THRESHOLD;
    g.sc_lower = c.SC_LOWER_THRESHOLD;
    g.sc_upper = c.SC_UPPER_THRESHOLD;
    g.msc_lower = c.MSC_LOWER_THRESHOLD;
    g.msc_upper = c.MSC_UPPER_THRESHOLD;
    g.sm_lower = c.SM_LOWER_THRESHOLD;
    g.sm_scale = c.SM_SCALE_THRESHOLD;
    g.msc_diff_thresh = c.MSC_DIFF_THRESH;
    g.fast_walks = c.EXACT_FAST_POINTS ? 1 : 0;
    return g;
}

// Per-history geometry of one history set, structure of arrays.
enum GeomArray { kXE, kYE, kZE, kXO, kYO, kZO, kXYE, kXZE, kXYO, kXZO, kNumGeom };
const char* const kGeomNames[kNumGeom] = {"x_entry", "y_entry", "z_entry", "x_exit", "y_exit", "z_exit",
                                          "xy_entry_angle", "xz_entry_angle", "xy_exit_angle", "xz_exit_angle"};
struct GeomPtrs {
    float* a[kNumGeom];
};

// Tracker inputs (B.cu:4139-4766 arrays after the mm->cm conversion).
enum TrackerArray { kTIn1, kTIn2, kTOut1, kTOut2, kUIn1, kUIn2, kUOut1, kUOut2, kVIn1, kVIn2, kVOut1, kVOut2, kNumTracker };
const char* const kTrackerNames[kNumTracker] = {"t_in_1", "t_in_2", "t_out_1", "t_out_2", "u_in_1", "u_in_2",
                                                "u_out_1", "u_out_2", "v_in_1", "v_in_2", "v_out_1", "v_out_2"};
struct TrackerPtrs {
    const float* a[kNumTracker];
};
static_assert(kTrackerSlots == kNumTracker + 2, "tracker slots: coordinates, WEPL, angle");

}  // namespace

// Device arrays of the preprocessing stages.
struct Preproc {
    long long n_raw = 0, cap_raw = 0;
    float* tracker[kNumTracker] = {};
    float* gantry_angle = nullptr;   // degrees
    int integer_angles = 0;
    float* raw_geom[kNumGeom] = {};  // intersections output
    float* raw_wepl = nullptr;
    uint8_t* missed = nullptr;
    int* raw_bin_num = nullptr;
    uint8_t* keep = nullptr;
    // current history vectors (compacted after binning, after cuts, after reconstruction cuts)
    long long n_vec = 0, cap_vec = 0;
    float* vec_geom[kNumGeom] = {};
    float* vec_wepl = nullptr;
    int* vec_bin_num = nullptr;
    uint32_t* vec_first_voxel = nullptr;
    // compaction scratch
    float* tmp_geom[kNumGeom] = {};
    float* tmp_wepl = nullptr;
    int* tmp_bin_num = nullptr;
    int* flags = nullptr;
    long long* offsets = nullptr;
    long long* scan_tmp = nullptr;
    long long cap_scratch = 0;
    // bins
    int* bin_counts = nullptr;
    float *mean_WEPL = nullptr, *mean_rel_ut_angle = nullptr, *mean_rel_uv_angle = nullptr;
    float *stddev_WEPL = nullptr, *stddev_rel_ut_angle = nullptr, *stddev_rel_uv_angle = nullptr;
    float *sinogram = nullptr, *sinogram_filtered = nullptr;
    double* fbp_tables = nullptr;
    // images
    float *FBP_image = nullptr, *FBP_median = nullptr;
    uint8_t *FBP_hull = nullptr, *SC_hull = nullptr, *hull = nullptr;
    int *MSC_counts = nullptr, *SM_counts = nullptr, *SM_differences = nullptr, *SM_thresholds = nullptr;
    int* edge_tmp = nullptr;
    unsigned* walk_hist = nullptr;  // bucket-sort scratch of the walk order
    int* hull_starts = nullptr;     // the hull walk's ranges of histories
    uint32_t* hull_bits = nullptr;  // hull, one bit per voxel (for the endpoint walks)
    bool hull_ready = false;
};

void preproc_release(Preproc* p)
{
    if (!p) return;
    for (int k = 0; k < kNumTracker; k++) cudaFree(p->tracker[k]);
    for (int k = 0; k < kNumGeom; k++) {
        cudaFree(p->raw_geom[k]);
        cudaFree(p->vec_geom[k]);
        cudaFree(p->tmp_geom[k]);
    }
    void* ptrs[] = {p->gantry_angle, p->raw_wepl, p->missed, p->raw_bin_num, p->keep, p->vec_wepl, p->vec_bin_num,
                    p->vec_first_voxel, p->tmp_wepl, p->tmp_bin_num, p->flags, p->offsets, p->scan_tmp,
                    p->bin_counts, p->mean_WEPL, p->mean_rel_ut_angle, p->mean_rel_uv_angle, p->stddev_WEPL,
                    p->stddev_rel_ut_angle, p->stddev_rel_uv_angle, p->sinogram, p->sinogram_filtered,
                    p->FBP_image, p->FBP_median, p->FBP_hull, p->SC_hull, p->hull, p->MSC_counts, p->SM_counts,
                    p->SM_differences, p->SM_thresholds, p->edge_tmp, p->walk_hist, p->hull_starts, p->hull_bits, p->fbp_tables};
    for (void* q : ptrs) cudaFree(q);
    delete p;
}

namespace {

// ------------------------------------------------------------------------------------------
// Device helpers
// ------------------------------------------------------------------------------------------

// calculate_intercepts (B.cu:5286-5372).  The intercept stays at its initial value when the
// line misses the circle (the reference leaves it unassigned).
__device__ bool calculate_intercepts(double R, double u, double t, double ut_angle, double& u_intercept,
                                     double& t_intercept)
{
    const bool entry_in_cone = ((ut_angle > kPiOver4) && (ut_angle < 3 * kPiOver4)) ||
                               ((ut_angle > 5 * kPiOver4) && (ut_angle < 7 * kPiOver4));
    double u_temp;
    if (entry_in_cone) {
        u_temp = u;
        u = -t;
        t = u_temp;
        ut_angle += kPiOver2;
    }
    const double m = tan(ut_angle);
    const double b_in = t - m * u;
    const double a = 1 + powf((float)m, 2.0f);
    const double b = 2 * m * b_in;
    const double c = __fsub_rn(powf((float)b_in, 2.0f), powf((float)R, 2.0f));
    const double entry_discriminant = powf((float)b, 2.0f) - (4 * a * c);
    const bool intersected = (entry_discriminant > 0);
    if (intersected) {
        const double u_intercept_1 = (sqrt(entry_discriminant) - b) / (2 * a);
        const double u_intercept_2 = (sqrt(entry_discriminant) + b) / (2 * a);
        const double t_intercept_1 = m * u_intercept_1 + b_in;
        const double t_intercept_2 = m * u_intercept_2 - b_in;
        const double squared_distance_1 =
            __fadd_rn(powf((float)(u_intercept_1 - u), 2.0f), powf((float)(t_intercept_1 - t), 2.0f));
        const double squared_distance_2 =
            __fadd_rn(powf((float)(u_intercept_2 + u), 2.0f), powf((float)(t_intercept_2 + t), 2.0f));
        u_intercept = u_intercept_1 * (squared_distance_1 <= squared_distance_2) -
                      u_intercept_2 * (squared_distance_1 > squared_distance_2);
        t_intercept = t_intercept_1 * (squared_distance_1 <= squared_distance_2) -
                      t_intercept_2 * (squared_distance_1 > squared_distance_2);
    }
    if (entry_in_cone) {
        u_temp = u_intercept;
        u_intercept = t_intercept;
        t_intercept = -u_temp;
    }
    return intersected;
}

// recon_volume_intersections_GPU / _exact_angles (B.cu:4890-5153): outputs are stored as float and
// later read back as float, as the reference does.
__global__ void intersections_kernel(PreGeom g, long long n, TrackerPtrs T, const float* __restrict__ angle_deg,
                                     int integer_angles, GeomPtrs out, uint8_t* __restrict__ missed)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float t_in_1 = T.a[kTIn1][i], t_in_2 = T.a[kTIn2][i], t_out_1 = T.a[kTOut1][i], t_out_2 = T.a[kTOut2][i];
    const float u_in_1 = T.a[kUIn1][i], u_in_2 = T.a[kUIn2][i], u_out_1 = T.a[kUOut1][i], u_out_2 = T.a[kUOut2][i];
    const float v_in_1 = T.a[kVIn1][i], v_in_2 = T.a[kVIn2][i], v_out_1 = T.a[kVOut1][i], v_out_2 = T.a[kVOut2][i];
    const double ANGLE_TO_RADIANS = (kPi / 180.0);
    const double rotation_angle_radians =
        integer_angles ? (int)angle_deg[i] * ANGLE_TO_RADIANS : angle_deg[i] * ANGLE_TO_RADIANS;
    const double HALF_H = g.H * 0.5;

    const double ut_entry_angle = atan2f(__fsub_rn(t_in_2, t_in_1), __fsub_rn(u_in_2, u_in_1));
    double u_entry = 0.0, t_entry = 0.0;
    bool entered = calculate_intercepts(g.R, u_in_2, t_in_2, ut_entry_angle, u_entry, t_entry);
    const float xy_entry_angle = (float)(ut_entry_angle + rotation_angle_radians);
    float x_entry = (float)((cos(rotation_angle_radians) * u_entry) - (sin(rotation_angle_radians) * t_entry));
    float y_entry = (float)((sin(rotation_angle_radians) * u_entry) + (cos(rotation_angle_radians) * t_entry));

    const double ut_exit_angle = atan2f(__fsub_rn(t_out_2, t_out_1), __fsub_rn(u_out_2, u_out_1));
    double u_exit = 0.0, t_exit = 0.0;
    bool exited = calculate_intercepts(g.R, u_out_1, t_out_1, ut_exit_angle, u_exit, t_exit);
    const float xy_exit_angle = (float)(ut_exit_angle + rotation_angle_radians);
    float x_exit = (float)((cos(rotation_angle_radians) * u_exit) - (sin(rotation_angle_radians) * t_exit));
    float y_exit = (float)((sin(rotation_angle_radians) * u_exit) + (cos(rotation_angle_radians) * t_exit));

    const double uv_entry_slope = __fdiv_rn(__fsub_rn(v_in_2, v_in_1), __fsub_rn(u_in_2, u_in_1));
    const double uv_exit_slope = __fdiv_rn(__fsub_rn(v_out_2, v_out_1), __fsub_rn(u_out_2, u_out_1));
    const float xz_entry_angle = atan2f(__fsub_rn(v_in_2, v_in_1), __fsub_rn(u_in_2, u_in_1));
    const float xz_exit_angle = atan2f(__fsub_rn(v_out_2, v_out_1), __fsub_rn(u_out_2, u_out_1));

    u_entry = (cos(rotation_angle_radians) * x_entry) + (sin(rotation_angle_radians) * y_entry);
    u_exit = (cos(rotation_angle_radians) * x_exit) + (sin(rotation_angle_radians) * y_exit);
    float z_entry = (float)(v_in_2 + uv_entry_slope * (u_entry - u_in_2));
    float z_exit = (float)(v_out_1 - uv_exit_slope * (u_out_1 - u_exit));

    if (entered && exited) {
        if ((fabsf(z_entry) < HALF_H) && (fabsf(z_exit) > HALF_H)) {
            const double recon_cyl_fraction =
                fabs((((z_exit >= 0) - (z_exit < 0)) * g.H * 0.5 - z_entry) / (double)__fsub_rn(z_exit, z_entry));
            x_exit = (float)(x_entry + recon_cyl_fraction * __fsub_rn(x_exit, x_entry));
            y_exit = (float)(y_entry + recon_cyl_fraction * __fsub_rn(y_exit, y_entry));
            z_exit = (float)(((z_exit >= 0) - (z_exit < 0)) * g.H * 0.5);
        } else if (fabsf(z_entry) > HALF_H) {
            entered = false;
            exited = false;
        }
        if ((fabsf(z_entry) > HALF_H) && (fabsf(z_exit) < HALF_H)) {
            const double recon_cyl_fraction =
                fabs((((z_exit >= 0) - (z_exit < 0)) * g.H * 0.5 - z_exit) / (double)__fsub_rn(z_exit, z_entry));
            x_entry = (float)(x_exit + recon_cyl_fraction * __fsub_rn(x_exit, x_entry));
            y_entry = (float)(y_exit + recon_cyl_fraction * __fsub_rn(y_exit, y_entry));
            z_entry = (float)(((z_entry >= 0) - (z_entry < 0)) * g.H * 0.5);
        }
        if ((fabsf(__fsub_rn(t_out_1, t_in_2)) > 5) || (fabsf(__fsub_rn(v_out_1, v_in_2)) > 5)) {
            entered = false;
            exited = false;
        }
    }
    out.a[kXE][i] = x_entry;
    out.a[kYE][i] = y_entry;
    out.a[kZE][i] = z_entry;
    out.a[kXO][i] = x_exit;
    out.a[kYO][i] = y_exit;
    out.a[kZO][i] = z_exit;
    out.a[kXYE][i] = xy_entry_angle;
    out.a[kXZE][i] = xz_entry_angle;
    out.a[kXYO][i] = xy_exit_angle;
    out.a[kXZO][i] = xz_exit_angle;
    missed[i] = (!entered || !exited) ? 1 : 0;
}

// rel angle of a history, wrapped as B.cu:5528-5537 does
__device__ __forceinline__ double rel_angle(float exit_angle, float entry_angle)
{
    double a = __fsub_rn(exit_angle, entry_angle);
    if (a > kPi) a -= 2 * kPi;
    if (a < -kPi) a += 2 * kPi;
    return a;
}

// binning_GPU (B.cu:5482-5553); bin_num keeps its 0 default when t/v fall outside (B.cu:5380).
__global__ void binning_kernel(PreGeom g, long long n, GeomPtrs G, const float* __restrict__ WEPL,
                               const uint8_t* __restrict__ missed, int* __restrict__ bin_num, int* bin_counts,
                               float* mean_WEPL, float* mean_ut, float* mean_uv)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float xe = G.a[kXE][i], ye = G.a[kYE][i], ze = G.a[kZE][i];
    const float xo = G.a[kXO][i], yo = G.a[kYO][i], zo = G.a[kZO][i];
    const double x_midpath = __fdiv_rn(__fadd_rn(xe, xo), 2.0f);
    const double y_midpath = __fdiv_rn(__fadd_rn(ye, yo), 2.0f);
    const double z_midpath = __fdiv_rn(__fadd_rn(ze, zo), 2.0f);
    double path_angle = atan2f(__fsub_rn(yo, ye), __fsub_rn(xo, xe));
    if (path_angle < 0) path_angle += 2 * kPi;
    const double RADIANS_TO_ANGLE = (180.0 / kPi), ANGLE_TO_RADIANS = (kPi / 180.0);
    const int angle_bin = int((path_angle * RADIANS_TO_ANGLE / g.angular_bin_size) + 0.5) % g.angular_bins;
    const double angle = angle_bin * g.angular_bin_size * ANGLE_TO_RADIANS;
    const double t = y_midpath * cos(angle) - x_midpath * sin(angle);
    const int t_bin = int((t / g.t_bin_size) + g.t_bins / 2);
    const double v = z_midpath;
    const int v_bin = int((v / g.v_bin_size) + g.v_bins / 2);
    int bin = 0;
    if ((t_bin >= 0) && (v_bin >= 0) && (t_bin < g.t_bins) && (v_bin < g.v_bins)) {
        bin = t_bin + angle_bin * g.t_bins + v_bin * g.t_bins * g.angular_bins;
        if (!missed[i]) {
            const double rel_ut_angle = rel_angle(G.a[kXYO][i], G.a[kXYE][i]);
            const double rel_uv_angle = rel_angle(G.a[kXZO][i], G.a[kXZE][i]);
            atomicAdd(&bin_counts[bin], 1);
            atomicAdd(&mean_WEPL[bin], WEPL[i]);
            atomicAdd(&mean_ut[bin], (float)rel_ut_angle);
            atomicAdd(&mean_uv[bin], (float)rel_uv_angle);
        }
    }
    bin_num[i] = bin;
}

// calculate_means_GPU (B.cu:5644)
__global__ void means_kernel(int nb, const int* __restrict__ bin_counts, float* mean_WEPL, float* mean_ut, float* mean_uv)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const int c = bin_counts[b];
    if (c > 0) {
        mean_WEPL[b] = __fdiv_rn(mean_WEPL[b], (float)c);
        mean_ut[b] = __fdiv_rn(mean_ut[b], (float)c);
        mean_uv[b] = __fdiv_rn(mean_uv[b], (float)c);
    }
}

// sum_squared_deviations_GPU (B.cu:5689)
__global__ void sum_sq_dev_kernel(long long n, const int* __restrict__ bin_num, const float* __restrict__ WEPL,
                                  GeomPtrs G, const float* __restrict__ mean_WEPL, const float* __restrict__ mean_ut,
                                  const float* __restrict__ mean_uv, float* sd_WEPL, float* sd_ut, float* sd_uv)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = bin_num[i];
    const double rel_ut_angle = rel_angle(G.a[kXYO][i], G.a[kXYE][i]);
    const double rel_uv_angle = rel_angle(G.a[kXZO][i], G.a[kXZE][i]);
    const double WEPL_difference = __fsub_rn(WEPL[i], mean_WEPL[b]);
    const double rel_ut_angle_difference = rel_ut_angle - mean_ut[b];
    const double rel_uv_angle_difference = rel_uv_angle - mean_uv[b];
    atomicAdd(&sd_WEPL[b], powf((float)WEPL_difference, 2.0f));
    atomicAdd(&sd_ut[b], powf((float)rel_ut_angle_difference, 2.0f));
    atomicAdd(&sd_uv[b], powf((float)rel_uv_angle_difference, 2.0f));
}

// calculate_standard_deviations_GPU (B.cu:5737); also zeroes bin_counts (B.cu:5748-5749)
__global__ void stddev_kernel(int nb, int sample, int* bin_counts, float* sd_WEPL, float* sd_ut, float* sd_uv)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const int c = bin_counts[b];
    if (c > 1) {
        const float d = (float)(c - sample);
        sd_WEPL[b] = sqrtf(__fdiv_rn(sd_WEPL[b], d));
        sd_ut[b] = sqrtf(__fdiv_rn(sd_ut[b], d));
        sd_uv[b] = sqrtf(__fdiv_rn(sd_uv[b], d));
    }
    bin_counts[b] = 0;
}

// statistical_cuts_GPU (B.cu:5937-5971): flags survivors, accumulates counts and WEPL sums
__global__ void cuts_kernel(PreGeom g, long long n, const int* __restrict__ bin_num, const float* __restrict__ WEPL,
                            GeomPtrs G, const float* __restrict__ mean_WEPL, const float* __restrict__ mean_ut,
                            const float* __restrict__ mean_uv, const float* __restrict__ sd_WEPL,
                            const float* __restrict__ sd_ut, const float* __restrict__ sd_uv, int* bin_counts,
                            float* sinogram, int* __restrict__ keep)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int b = bin_num[i];
    const double rel_ut_angle = rel_angle(G.a[kXYO][i], G.a[kXYE][i]);
    const double rel_uv_angle = rel_angle(G.a[kXZO][i], G.a[kXZE][i]);
    const bool passed_ut_cut = (fabs(rel_ut_angle - mean_ut[b]) < (double)__fmul_rn((float)g.sigmas_to_keep, sd_ut[b]));
    const bool passed_uv_cut = (fabs(rel_uv_angle - mean_uv[b]) < (double)__fmul_rn((float)g.sigmas_to_keep, sd_uv[b]));
    const bool passed_WEPL_cut = (fabsf(__fsub_rn(mean_WEPL[b], WEPL[i])) <= __fmul_rn((float)g.sigmas_to_keep, sd_WEPL[b]));
    const bool failed = !passed_ut_cut || !passed_uv_cut || !passed_WEPL_cut;
    if (!failed) {
        atomicAdd(&bin_counts[b], 1);
        atomicAdd(&sinogram[b], WEPL[i]);
    }
    keep[i] = failed ? 0 : 1;
}

// construct_sinogram_GPU (B.cu:6073)
__global__ void sinogram_kernel(int nb, const int* __restrict__ bin_counts, float* sinogram)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    const int c = bin_counts[b];
    if (c > 0) sinogram[b] = __fdiv_rn(sinogram[b], (float)c);
}

// What the filter and the backprojection need of the configuration alone, evaluated with the
// reference's expressions: the filter's value at each separation, its scale factor at each (v, t)
// bin, and the cosine and sine of each angle bin.
struct FbpTables {
    double* filter;  // [t_bins]
    double* scale;   // [v_bins][t_bins]
    double* trig;    // [angular_bins][2]
};
__global__ void fbp_tables_kernel(PreGeom g, FbpTables tab)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < g.t_bins) {  // symmetric in the separation
        const int t_bin_sep = i;
        // RAM_LAK_TAU = 2/ROOT_TWO * T_BIN_SIZE, ROOT_TWO = sqrtf(2.0): a float quotient
        const double ram_lak_tau = (double)__fdiv_rn(2.0f, sqrtf(2.0f)) * g.t_bin_size;
        double filtered;
        if (g.sinogram_filter == PCT_RAM_LAK) {
            if (t_bin_sep == 0) filtered = 1.0 / (4.0 * pow(ram_lak_tau, 2.0));
            else if (t_bin_sep % 2 == 0) filtered = 0;
            else filtered = -1.0 / (pow(ram_lak_tau * kPi * t_bin_sep, 2.0));
        } else {
            filtered = 1.0 / ((g.t_bin_size * kPi * g.t_bin_size * kPi) * (1.0 - (4 * t_bin_sep * t_bin_sep)));
        }
        tab.filter[i] = filtered;
    }
    if (i < g.t_bins * g.v_bins) {
        const int v_bin = i / g.t_bins, t_bin_ref = i - v_bin * g.t_bins;
        const double v = (v_bin - g.v_bins / 2 + 0.5) * g.v_bin_size;
        const double t = (t_bin_ref - g.t_bins / 2 + 0.5) * g.t_bin_size;
        tab.scale[i] = g.source_radius / sqrt(g.source_radius * g.source_radius + t * t + v * v);
    }
    if (i < g.angular_bins) {
        const double bin_angle = i * (g.angular_bin_size * (kPi / 180.0));
        tab.trig[2 * i] = cos(bin_angle);
        tab.trig[2 * i + 1] = sin(bin_angle);
    }
}

// filter_GPU (B.cu:6206-6240): every output sums its strip in the reference's order; each term is rounded
// to float as atomicAdd(float*, double) rounds it.  The reference leaves the filter value unset for
// UNFILTERED; here it passes the sinogram through.
// A CTA takes kFilterStrips angle bins of one v bin, which share the scale factors and, per thread, the
// filter values; the strips' bins times T_BIN_SIZE wait in shared memory.  It is bound by the two double
// products and the conversion of each of the NUM_BINS x T_BINS terms.  On the head scan (350 x 90 x 36
// bins) one thread per output that evaluated each term in full, a square root and two divisions,
// took 1.21 ms; this takes 0.14.
constexpr int kFilterStrips = 6, kFilterTile = 256;
__global__ void __launch_bounds__(128) filter_kernel(PreGeom g, FbpTables tab, const float* __restrict__ sinogram,
                                                     float* __restrict__ filtered_out)
{
    __shared__ double term[kFilterTile][kFilterStrips], scale[kFilterTile];
    const int t_blocks = (g.t_bins + blockDim.x - 1) / blockDim.x, groups = (g.angular_bins + kFilterStrips - 1) / kFilterStrips;
    const int t_bin = (blockIdx.x % t_blocks) * blockDim.x + threadIdx.x;
    const int v_bin = blockIdx.x / t_blocks / groups, first = blockIdx.x / t_blocks % groups * kFilterStrips;
    const long long base = ((long long)v_bin * g.angular_bins + first) * g.t_bins;
    const int strips = min(kFilterStrips, g.angular_bins - first);
    if (g.sinogram_filter == PCT_UNFILTERED) {
        if (t_bin < g.t_bins)
            for (int j = 0; j < strips; j++) filtered_out[base + (long long)j * g.t_bins + t_bin] = sinogram[base + (long long)j * g.t_bins + t_bin];
        return;
    }
    float acc[kFilterStrips];
#pragma unroll
    for (int j = 0; j < kFilterStrips; j++) acc[j] = 0.0f;
    for (int r0 = 0; r0 < g.t_bins; r0 += kFilterTile) {
        const int here = min(kFilterTile, g.t_bins - r0);
        __syncthreads();
        for (int k = threadIdx.x; k < here; k += blockDim.x) {
            scale[k] = tab.scale[(long long)v_bin * g.t_bins + r0 + k];
#pragma unroll
            for (int j = 0; j < kFilterStrips; j++)
                term[k][j] = j < strips ? g.t_bin_size * sinogram[base + (long long)j * g.t_bins + r0 + k] : 0.0;
        }
        __syncthreads();
        if (t_bin < g.t_bins)
#pragma unroll 4
            for (int k = 0; k < here; k++) {
                const double f = __ldg(tab.filter + abs(t_bin - (r0 + k))), sc = scale[k];
#pragma unroll
                for (int j = 0; j < kFilterStrips; j++) acc[j] = __fadd_rn(acc[j], (float)(term[k][j] * f * sc));
            }
    }
    if (t_bin < g.t_bins)
#pragma unroll
        for (int j = 0; j < kFilterStrips; j++)
            if (j < strips) filtered_out[base + (long long)j * g.t_bins + t_bin] = acc[j];
}

// voxel_2_3D_voxels_GPU (B.cu:11117-11133): the reference's loops stop at "> 0", so an index that
// is an exact multiple of COLUMNS*ROWS (or COLUMNS) is decomposed one step short; kept as is.
__device__ __forceinline__ void voxel_2_3D_voxels(const PreGeom& g, int voxel, int& vx, int& vy, int& vz)
{
    const int CR = g.columns * g.rows;
    vz = voxel > 0 ? (voxel - 1) / CR : 0;
    voxel -= vz * CR;
    vy = voxel > 0 ? (voxel - 1) / g.columns : 0;
    voxel -= vy * g.columns;
    vx = voxel;
}

__device__ __forceinline__ double voxel_2_position(int voxel_i, double size, int num_i, int progression)
{
    const double zero_voxel = (num_i - 1) / 2.0;
    return progression * (voxel_i - zero_voxel) * size;
}

// backprojection_GPU2 (B.cu:6340-6479): angles summed in order.  A thread takes kBackSlices slices of a
// column: u, t and everything across the detector depend only on the column and the angle.  Bound by
// double arithmetic and conversions.  On 200x200x32 voxels and 90 angles: 1.37 ms with a thread per voxel
// that evaluated each angle's cosine and sine and five divisions, 0.81 ms with two slices and the cosines
// from a table, 0.63 ms with quotient() for the divisions.  Four slices take 0.59 ms there but 0.22
// instead of 0.15 ms on 128x128x16, where they leave SMs without work.
constexpr int kBackSlices = 2;

// a / b from b's correctly rounded reciprocal r: two steps of q + (a - q b) r from q = a r.  The first
// leaves q within one unit in the last place, and from such a q the second gives the correctly rounded
// quotient (Markstein, IBM J. Res. Dev. 34, 1990).  For a zero or well inside the range of double; the sign of
// a zero is lost.  pct_selftest_quotient compares it with the division.
__device__ __forceinline__ double quotient(double a, double b, double r)
{
    double q = a * r;
    q = __fma_rn(__fma_rn(-q, b, a), r, q);
    return __fma_rn(__fma_rn(-q, b, a), r, q);
}

// quotient(a, b, 1/b) against a / b over n pairs of the backprojection's ranges: a heights, distances and positions
// up to 2^8 with exponents down to 2^-40, whole eighths, and zero; b ranges, bin sizes, and mantissas of all ones
// and near ones.
__global__ void quotient_check_kernel(long long n, unsigned long long seed, unsigned long long* mismatches)
{
    const long long stride = (long long)gridDim.x * blockDim.x;
    unsigned long long local = 0, state = seed;
    auto next = [&](unsigned long long counter) {  // splitmix64
        unsigned long long z = state + counter * 0x9e3779b97f4a7c15ull;
        z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
        z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
        return z ^ (z >> 31);
    };
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const unsigned long long ra = next(2 * i + 1), rb = next(2 * i + 2), mantissa = 0xfffffffffffffull;
        double a = __longlong_as_double((long long)((983 + (ra >> 52) % 48) << 52 | (ra & mantissa)));
        double b = __longlong_as_double((long long)((1013 + (rb >> 52) % 20) << 52 | (rb & mantissa)));  // 2^-10 to 2^10
        const int kind = (int)(i & 7);
        if (kind == 1) b = __longlong_as_double(__double_as_longlong(b) | (long long)mantissa);
        if (kind == 2) b = __longlong_as_double((__double_as_longlong(b) & ~(long long)mantissa) | (long long)(rb >> 40 & 15));
        if (kind == 3) b = __longlong_as_double(__double_as_longlong(b) | (long long)(mantissa & ~15ull));
        if (kind == 4) a = (double)((long long)(ra & 4095) - 2048) * 0.125;
        if (kind == 5) b = (double)(1 + (rb & 1023)) * 0.05;
        if (kind == 6) a = b * (double)(1 + (ra & 255));  // whole and nearly whole quotients
        if (i & 8) a = -a;
        if (quotient(a, b, __drcp_rn(b)) != a / b) local++;
    }
    if (local) atomicAdd(mismatches, local);
}

template <bool kRegular>
__device__ __forceinline__ void backproject(const PreGeom& g, const double* __restrict__ trig,
                                            const float* __restrict__ sinogram_filtered, double x, double y, const double* z,
                                            float* acc)
{
    const double ANGLE_TO_RADIANS = (kPi / 180.0);
    const double delta = g.angular_bin_size * ANGLE_TO_RADIANS;
    const int T = g.t_bins, V = g.v_bins, A = g.angular_bins;
    const double t_size_inv = __drcp_rn(g.t_bin_size), v_size_inv = __drcp_rn(g.v_bin_size), T_half = T / 2.0, V_half = V / 2.0;
#pragma unroll
    for (int k = 0; k < kBackSlices; k++) acc[k] = 0.0f;
    for (int angle_bin = 0; angle_bin < A; angle_bin++) {
        const double c = __ldg(trig + 2 * angle_bin), sn = __ldg(trig + 2 * angle_bin + 1);
        const double u = x * c + y * sn;
        const double t = y * c - x * sn;
        const double range = g.source_radius + u, range_inv = __drcp_rn(range);
        const double across_t = t - u * (kRegular ? quotient(t, range, range_inv) : t / range);
        const double detector_number_t = (kRegular ? quotient(across_t, g.t_bin_size, t_size_inv) : across_t / g.t_bin_size) + T_half;
        const int t_bin = __double2int_rd(detector_number_t);
        const double eta = detector_number_t - t_bin, eta_1 = 1 - eta;
        const double scale_factor = powf((float)(kRegular ? quotient(g.source_radius, range, range_inv) : g.source_radius / range), 2.0f);
        const bool t_in = t_bin > -1 && t_bin < T - 1, t_low = t_bin == -1, t_high = t_bin == T - 1;
#pragma unroll
        for (int k = 0; k < kBackSlices; k++) {
            const double v = z[k];
            const double across = v - u * (kRegular ? quotient(v, range, range_inv) : v / range);
            const double detector_number_v = (kRegular ? quotient(across, g.v_bin_size, v_size_inv) : across / g.v_bin_size) + V_half;
            const int v_bin = __double2int_rd(detector_number_v);
            const double epsilon = detector_number_v - v_bin, epsilon_1 = 1 - epsilon;
            const long long bin11 = ((long long)v_bin * A + angle_bin) * T + t_bin;
            const long long bin12 = bin11 + 1;
            const long long bin21 = bin11 + (long long)A * T;
            const long long bin22 = bin21 + 1;
            const bool v_in = v_bin > -1 && v_bin < V - 1, v_low = v_bin == -1, v_high = v_bin == V - 1;
            float xterm = 0.0f;
            if (t_in) {
                if (v_in) {
                    xterm = (float)(sinogram_filtered[bin11] * eta_1 * epsilon_1 + sinogram_filtered[bin12] * eta * epsilon_1 +
                                    sinogram_filtered[bin21] * eta_1 * epsilon + sinogram_filtered[bin22] * eta * epsilon);
                } else if (v_low) {
                    xterm = (float)(sinogram_filtered[bin21] * eta_1 * epsilon + sinogram_filtered[bin22] * eta * epsilon);
                } else if (v_high) {
                    xterm = (float)(sinogram_filtered[bin11] * eta_1 * epsilon_1 + sinogram_filtered[bin12] * eta * epsilon_1);
                }
            } else if (t_low) {
                if (v_in) {
                    xterm = (float)(sinogram_filtered[bin12] * eta * epsilon_1 + sinogram_filtered[bin22] * eta * epsilon);
                } else if (v_low) {
                    xterm = (float)(sinogram_filtered[bin22] * eta * epsilon);
                } else if (v_high) {
                    xterm = (float)(sinogram_filtered[bin12] * eta * epsilon_1);
                }
            } else if (t_high) {
                if (v_in) {
                    xterm = (float)(sinogram_filtered[bin11] * eta_1 * epsilon_1 + sinogram_filtered[bin21] * eta_1 * epsilon);
                } else if (v_low) {
                    xterm = (float)(sinogram_filtered[bin21] * eta_1 * epsilon);
                } else if (v_high) {
                    xterm = (float)(sinogram_filtered[bin11] * eta_1 * epsilon_1);
                }
            }
            acc[k] = __fadd_rn(acc[k], (float)(xterm * delta * scale_factor));
        }
    }
}

__global__ void __launch_bounds__(128) backprojection_kernel(PreGeom g, const double* __restrict__ trig,
                                                             const float* __restrict__ sinogram_filtered,
                                                             float* __restrict__ FBP)
{
    const int slab = g.columns * g.rows;
    const int blocks = (slab + blockDim.x - 1) / blockDim.x;  // of a group of slices
    const int in_slab = (blockIdx.x % blocks) * blockDim.x + threadIdx.x, s0 = blockIdx.x / blocks * kBackSlices;
    if (in_slab >= slab) return;
    const int count = min(kBackSlices, g.slices - s0);
    // u is at most R, so that range and the heights on the detector are far from the limits of double
    const bool regular = g.source_radius > 2 * g.R && g.source_radius < 1e9 && g.v_bin_size > 1e-9 && g.v_bin_size < 1e9 &&
                         g.t_bin_size > 1e-9 && g.t_bin_size < 1e9 && g.voxel_width > 1e-9 && g.voxel_height > 1e-9 &&
                         g.voxel_thickness > 1e-9 && g.voxel_thickness < 1e9;
    double x = 0.0, y = 0.0, z[kBackSlices];
    float acc[kBackSlices];
    // the voxel at the slab's start takes another column in slice 0 than in the others (voxel_2_3D_voxels):
    // slices one by one there
    const int step = in_slab == 0 ? 1 : kBackSlices;
    for (int s = 0; s < count; s += step) {
        const int here = min(step, count - s);
#pragma unroll
        for (int k = 0; k < kBackSlices; k++) {
            int vx, vy, vz;  // (the last slice again where there are no more)
            voxel_2_3D_voxels(g, in_slab + (s0 + s + min(k, here - 1)) * slab, vx, vy, vz);
            if (k == 0) {
                x = voxel_2_position(vx, g.voxel_width, g.columns, 1);
                y = voxel_2_position(vy, g.voxel_height, g.rows, -1);
            }
            z[k] = voxel_2_position(vz, g.voxel_thickness, g.slices, -1);
        }
        if ((x * x + y * y) > (g.R * g.R)) {
            for (int k = 0; k < here; k++) FBP[in_slab + (long long)(s0 + s + k) * slab] = (float)g.rsp_air;
        } else {
            if (regular) backproject<true>(g, trig, sinogram_filtered, x, y, z, acc);
            else backproject<false>(g, trig, sinogram_filtered, x, y, z, acc);
#pragma unroll
            for (int k = 0; k < kBackSlices; k++)
                if (k < here) FBP[in_slab + (long long)(s0 + s + k) * slab] = acc[k];
        }
    }
}

// median_filter_2D (B.cu:7482-7521): (2r+1)^2 neighbourhood per slice, the element at index
// n/2 of the sorted values; voxels within r of a slice edge stay 0.

// The element of rank `middle` by counting: the value with fewer than middle+1 smaller elements and at
// least middle+1 elements <= it (the first such one if there are several, the first value if none).
__device__ float median_by_counting(const PreGeom& g, int radius, const float* __restrict__ in, int col, int row)
{
    const int side = 2 * radius + 1, count = side * side, middle = count / 2;
    float vals[225];  // radius <= 7
    int k = 0;
    for (int c = col - radius; c <= col + radius; c++)
        for (int r = row - radius; r <= row + radius; r++) vals[k++] = in[c + r * g.columns];
    float result = vals[0];
    for (int a = 0; a < count; a++) {
        int less = 0, less_eq = 0;
        for (int b = 0; b < count; b++) {
            less += vals[b] < vals[a];
            less_eq += vals[b] <= vals[a];
        }
        if (less <= middle && middle < less_eq) {
            result = vals[a];
            break;
        }
    }
    return result;
}

// kRadius 1, 2, 3: the median of the 2n+1 values by discarding extremes: of n + 2 values the smallest and
// the largest cannot be the median, so they are replaced by the next value until three are left; the
// values stay in registers.  Radius 0 stands for any other, by counting, as do neighbourhoods with
// a NaN or an infinity and zero medians.  Bound by the exchanges (about 1050 minima and maxima at radius
// 3): 0.077 ms on 200x200x32 voxels, 0.64 ms by counting.
template <int kRadius>
__global__ void __launch_bounds__(128) median_kernel(PreGeom g, int radius, const float* __restrict__ in, float* __restrict__ out)
{
    const long long voxel = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (voxel >= g.num_voxels) return;
    const int CR = g.columns * g.rows;
    const int slice = (int)(voxel / CR), rem = (int)(voxel % CR), row = rem / g.columns, col = rem % g.columns;
    if (col < radius || col >= g.columns - radius || row < radius || row >= g.rows - radius) {
        out[voxel] = 0.0f;
        return;
    }
    const float* plane = in + (long long)slice * CR;
    if constexpr (kRadius > 0) {
        constexpr int side = 2 * kRadius + 1, count = side * side, held = count / 2 + 2;
        const float* corner = plane + (col - kRadius) + (row - kRadius) * g.columns;
        auto value = [&](int k) { return __ldg(corner + k % side + k / side * g.columns); };
        float v[held], finite = 0.0f;
#pragma unroll
        for (int k = 0; k < held; k++) {
            v[k] = value(k);
            finite = __fmaf_rn(v[k], 0.0f, finite);
        }
#pragma unroll
        for (int n = held; n >= 3; n--) {  // v[0 .. n): smallest to the front, largest to the back
#pragma unroll
            for (int k = 0; k < n / 2; k++) {
                const float a = v[k], b = v[n - 1 - k];
                v[k] = fminf(a, b);
                v[n - 1 - k] = fmaxf(a, b);
            }
#pragma unroll
            for (int k = 1; k < (n + 1) / 2; k++) {
                const float a = v[0], b = v[k];
                v[0] = fminf(a, b);
                v[k] = fmaxf(a, b);
            }
#pragma unroll
            for (int k = n / 2; k < n - 1; k++) {
                const float a = v[k], b = v[n - 1];
                v[k] = fminf(a, b);
                v[n - 1] = fmaxf(a, b);
            }
            if (n > 3) {  // drop both, take the next value
                v[0] = value(count - n + 3);
                finite = __fmaf_rn(v[0], 0.0f, finite);
            }
        }
        if (finite == 0.0f && v[1] != 0.0f) {  // (zeros of both signs compare equal)
            out[voxel] = v[1];
            return;
        }
    }
    out[voxel] = median_by_counting(g, radius, plane, col, row);
}

// FBP_image_2_hull_GPU (B.cu:6592)
__global__ void fbp_hull_kernel(PreGeom g, const float* __restrict__ FBP, uint8_t* __restrict__ hull)
{
    const long long voxel = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (voxel >= g.num_voxels) return;
    const int rem = (int)(voxel % ((long long)g.columns * g.rows)), row = rem / g.columns, column = rem % g.columns;
    const double x = -g.R + (column + 0.5) * g.voxel_width;
    const double y = g.R - (row + 0.5) * g.voxel_height;
    const double d_squared = __fadd_rn(powf((float)x, 2.0f), powf((float)y, 2.0f));
    hull[voxel] = (FBP[voxel] > g.fbp_threshold && (d_squared < powf((float)g.R, 2.0f))) ? 1 : 0;
}

// initialize_hull_GPU (B.cu:6659): 1 inside the reconstruction cylinder
template <class T>
__global__ void init_hull_kernel(PreGeom g, T* __restrict__ hull)
{
    const long long voxel = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (voxel >= g.num_voxels) return;
    const int rem = (int)(voxel % ((long long)g.columns * g.rows)), row = rem / g.columns, column = rem % g.columns;
    const double x = (column - g.columns / 2 + 0.5) * g.voxel_width;
    const double y = (g.rows / 2 - row - 0.5) * g.voxel_height;
    hull[voxel] = (__fadd_rn(powf((float)x, 2.0f), powf((float)y, 2.0f)) < powf((float)g.R, 2.0f)) ? 1 : 0;
}

// ---- straight-line voxel walks (B.cu:11313-11462) ----
__device__ __forceinline__ int calculate_voxel(double zero, double pos, double size)
{
    const double q = fabs(pos - zero) / size;
    return q < 2147483647.0 ? (int)q : 2147483647;
}
__device__ __forceinline__ double edge_coordinate(double zero, int voxel_entered, double size, int inc, int step)
{
    const int on_edge = (step == inc) ? voxel_entered : voxel_entered + 1;
    return zero + (inc * on_edge * size);
}
__device__ __forceinline__ double distance_remaining(double zero, double pos, int inc, int step, double size, int voxel)
{
    const int next_voxel = voxel + inc * step;
    return fabs(edge_coordinate(zero, next_voxel, size, inc, step) - pos);
}
__device__ __forceinline__ double corresponding_coordinate(double m, double x, double x0, double y0) { return m * (x - x0) + y0; }

struct WalkState {
    double x, y, z, x_to_go, y_to_go, z_to_go;
    int vx, vy, vz, voxel;
};

// take_3D_step_GPU (B.cu:11392-11460) with X_INCREASING_DIRECTION = RIGHT, Y/Z = DOWN
__device__ void take_3D_step(const PreGeom& g, int xd, int yd, int zd, double dy_dx, double dz_dx, double dz_dy,
                             double dx_dy, double dx_dz, double dy_dz, double x0, double y0, double z0, WalkState& w)
{
    const double X0 = -g.R, Y0 = g.R, Z0 = g.H / 2;
    const double x_extension = fabs(dz_dx) * w.x_to_go;
    const double y_extension = fabs(dz_dy) * w.y_to_go;
    if ((w.z_to_go <= x_extension) && (w.z_to_go <= y_extension)) {
        w.vz -= zd;
        w.z = edge_coordinate(Z0, w.vz, g.voxel_thickness, -1, zd);
        w.x = corresponding_coordinate(dx_dz, w.z, z0, x0);
        w.y = corresponding_coordinate(dy_dz, w.z, z0, y0);
        w.x_to_go = distance_remaining(X0, w.x, 1, xd, g.voxel_width, w.vx);
        w.y_to_go = distance_remaining(Y0, w.y, -1, yd, g.voxel_height, w.vy);
        w.z_to_go = g.voxel_thickness;
    } else if (x_extension <= y_extension) {
        w.vx += xd;
        w.x = edge_coordinate(X0, w.vx, g.voxel_width, 1, xd);
        w.y = corresponding_coordinate(dy_dx, w.x, x0, y0);
        w.z = corresponding_coordinate(dz_dx, w.x, x0, z0);
        w.x_to_go = g.voxel_width;
        w.y_to_go = distance_remaining(Y0, w.y, -1, yd, g.voxel_height, w.vy);
        w.z_to_go = distance_remaining(Z0, w.z, -1, zd, g.voxel_thickness, w.vz);
    } else {
        w.vy -= yd;
        w.y = edge_coordinate(Y0, w.vy, g.voxel_height, -1, yd);
        w.x = corresponding_coordinate(dx_dy, w.y, y0, x0);
        w.z = corresponding_coordinate(dz_dy, w.y, y0, z0);
        w.x_to_go = distance_remaining(X0, w.x, 1, xd, g.voxel_width, w.vx);
        w.y_to_go = g.voxel_height;
        w.z_to_go = distance_remaining(Z0, w.z, -1, zd, g.voxel_thickness, w.vz);
    }
    if (w.x_to_go == 0) {
        w.x_to_go = g.voxel_width;
        w.vx += xd;
    }
    if (w.y_to_go == 0) {
        w.y_to_go = g.voxel_height;
        w.vy -= yd;
    }
    if (w.z_to_go == 0) {
        w.z_to_go = g.voxel_thickness;
        w.vz -= zd;
    }
    w.vz = max(w.vz, 0);
    w.voxel = w.vx + w.vy * g.columns + w.vz * g.columns * g.rows;
}

// take_2D_step_GPU (B.cu:11346-11390)
__device__ void take_2D_step(const PreGeom& g, int xd, int yd, double dy_dx, double dx_dy, double x0, double y0, WalkState& w)
{
    const double X0 = -g.R, Y0 = g.R;
    const double y_extension = fabs(dx_dy) * w.y_to_go;
    if (w.x_to_go <= y_extension) {
        w.vx += xd;
        w.x = edge_coordinate(X0, w.vx, g.voxel_width, 1, xd);
        w.y = corresponding_coordinate(dy_dx, w.x, x0, y0);
        w.x_to_go = g.voxel_width;
        w.y_to_go = distance_remaining(Y0, w.y, -1, yd, g.voxel_height, w.vy);
    } else {
        w.vy -= yd;
        w.y = edge_coordinate(Y0, w.vy, g.voxel_height, -1, yd);
        w.x = corresponding_coordinate(dx_dy, w.y, y0, x0);
        w.x_to_go = distance_remaining(X0, w.x, 1, xd, g.voxel_width, w.vx);
        w.y_to_go = g.voxel_height;
    }
    if (w.x_to_go == 0) {
        w.x_to_go = g.voxel_width;
        w.vx += xd;
    }
    if (w.y_to_go == 0) {
        w.y_to_go = g.voxel_height;
        w.vy -= yd;
    }
    w.vz = max(w.vz, 0);
    w.voxel = w.vx + w.vy * g.columns + w.vz * g.columns * g.rows;
}

// ---- voxel walks by crossing times --------------------------------------------------------------
// A step of the reference's walk is about 40 double operations, three ways: it moves to the nearest
// voxel face, computes the other two coordinates there, and their distances to the next faces.  Which
// face is nearest depends only on the line's crossing times with the three families of planes, which
// are arithmetic sequences.  So the walk carries the next crossing time of each axis as a 32-bit fixed
// point number and steps on the smallest one: an addition and a voxel index increment.
//  * A step is taken this way only when the smallest time leads the others by more than the reference's
//    coordinates can be off: its slopes are float quotients (or powf and tanf values), so a coordinate is
//    off by that relative error times the distance travelled.
//  * Otherwise the state the reference has at this point is set up again from the last face crossed (every
//    coordinate it keeps follows from that face and the line) and the reference's own step decides: one
//    warp step in 200.
//  * All lanes of a warp stay in one loop, which they leave together; a lane that needs the reference's
//    step waits for that.
// The voxels visited are the reference's either way (EXACT_FAST_POINTS = 0 takes every step by the
// reference's code).  On the head scan the end points of 3.3M histories took 5.74 ms with the reference's
// steps and take 2.53 ms, half of it the walks' setup (trigonometry, divisions), half the steps; a warp's
// walks differ in length, so 12 of its 32 lanes step on average.
enum WalkAxis { kAxisX = 0, kAxisY = 1, kAxisZ = 2, kAxisNone = 3 };
struct WalkLine {
    double x0, y0, z0;
    int xd, yd, zd;
};
struct WalkSlopes {
    double dy_dx, dz_dx, dz_dy, dx_dy, dx_dz, dy_dz;
};

// The coordinates on the face last crossed (the assignments of take_3D_step's three cases).
__device__ __forceinline__ void face_position(const PreGeom& g, const WalkLine& l, const WalkSlopes& m, int axis, WalkState& w)
{
    if (axis == kAxisX) {
        w.x = edge_coordinate(-g.R, w.vx, g.voxel_width, 1, l.xd);
        w.y = corresponding_coordinate(m.dy_dx, w.x, l.x0, l.y0);
        w.z = corresponding_coordinate(m.dz_dx, w.x, l.x0, l.z0);
    } else if (axis == kAxisY) {
        w.y = edge_coordinate(g.R, w.vy, g.voxel_height, -1, l.yd);
        w.x = corresponding_coordinate(m.dx_dy, w.y, l.y0, l.x0);
        w.z = corresponding_coordinate(m.dz_dy, w.y, l.y0, l.z0);
    } else if (axis == kAxisZ) {
        w.z = edge_coordinate(g.H / 2, w.vz, g.voxel_thickness, -1, l.zd);
        w.x = corresponding_coordinate(m.dx_dz, w.z, l.z0, l.x0);
        w.y = corresponding_coordinate(m.dy_dz, w.z, l.z0, l.y0);
    } else {
        w.x = l.x0;
        w.y = l.y0;
        w.z = l.z0;
    }
}

__device__ __forceinline__ void face_distances(const PreGeom& g, const WalkLine& l, int axis, WalkState& w)
{
    w.x_to_go = axis == kAxisX ? g.voxel_width : distance_remaining(-g.R, w.x, 1, l.xd, g.voxel_width, w.vx);
    w.y_to_go = axis == kAxisY ? g.voxel_height : distance_remaining(g.R, w.y, -1, l.yd, g.voxel_height, w.vy);
    w.z_to_go = axis == kAxisZ ? g.voxel_thickness : distance_remaining(g.H / 2, w.z, -1, l.zd, g.voxel_thickness, w.vz);
}

__device__ __forceinline__ bool walk_outside(const PreGeom& g, const WalkState& w)
{
    return w.vx >= g.columns || w.vy >= g.rows || w.vz >= g.slices || w.vx < 0 || w.vy < 0 || w.vz < 0;
}

struct CrossingTimes {
    unsigned tx, ty, tz, bx, by, bz;  // next crossings and their spacing
    int ix, iy, iz;                   // voxel index increments
    unsigned stop;         // from here on a crossing may leave the grid
    unsigned lead;         // by which a crossing decides
    int exit_axis;         // the crossing that leaves the grid (kAxisNone: through its top)
    bool above;            // more than half of the way lies beyond the grid's top, where every step is the reference's
};

// w: the walk's initial state; |dx|, |dy|, |dz|: the line's direction.  `error`: how far the reference's
// crossing times can be off, relative to the walk's length (its slopes' relative errors); to that come the roundings of its coordinates (1e-13 cm) and of the fixed point
// (half a unit of 2^-30 of the walk per crossing).  False where the line is too close to a coordinate
// plane for the times to be of use.
__device__ __forceinline__ bool crossing_times(const PreGeom& g, const WalkLine& l, const WalkState& w, double dx, double dy,
                                               double dz, double error, CrossingTimes& c)
{
    if (!g.fast_walks || l.xd == 0 || l.yd == 0 || l.zd == 0 || !(dx > 1e-9) || !(dy > 1e-9) || !(dz > 1e-9) ||
        !(error < 0.05) || !(dx < 1e9 && dy < 1e9 && dz < 1e9))
        return false;
    if (g.columns < 2 || g.rows < 2) return false;  // index increments tell the axes
    // a start beyond the grid's zero corner has the mirrored index: its first planes lie behind it
    if (w.x < -g.R || w.y > g.R || w.z > g.H / 2) return false;
    const double rx = 1.0 / dx, ry = 1.0 / dy, rz = 1.0 / dz;
    const double tx = w.x_to_go * rx, ty = w.y_to_go * ry, tz = w.z_to_go * rz;
    const double bx = g.voxel_width * rx, by = g.voxel_height * ry, bz = g.voxel_thickness * rz;
    // planes before the one that leaves the grid (columns grow with x; rows and slices fall with y and z)
    const int nx = l.xd > 0 ? g.columns - 1 - w.vx : w.vx;
    const int ny = l.yd > 0 ? w.vy : g.rows - 1 - w.vy;
    const int nz = l.zd > 0 ? w.vz : g.slices - 1 - w.vz;
    const double ex = tx + nx * bx, ey = ty + ny * by, ez = tz + nz * bz, end = fmin(fmin(ex, ey), ez);
    if (!(end > 0.0) || !(end < 1e12)) return false;
    const double unit = 1073741824.0 / end;  // 2^30
    auto fixed = [&](double t) { return (unsigned)fmin(t * unit + 0.5, 1.6e9); };
    c.tx = fixed(tx);
    c.ty = fixed(ty);
    c.tz = fixed(tz);
    c.bx = fixed(bx);
    c.by = fixed(by);
    c.bz = fixed(bz);
    c.ix = l.xd;
    c.iy = -l.yd * g.columns;
    c.iz = -l.zd * g.columns * g.rows;
    const double roundings = 1.0e-13 * fmax(fmax(rx, ry), rz) * unit + max(max(nx, ny), nz) + 8.0;
    c.lead = (unsigned)fmin(roundings + error * 1073741824.0, 1.0e9);
    if (c.lead > min(min(c.bx, c.by), c.bz) / 8) return false;  // also tells the last crossing from the one before
    const double leave = 1073741824.0 - 2.0 * c.lead;
    c.stop = leave > 0.0 ? (unsigned)leave : 0u;
    c.above = l.zd > 0 && end < 0.5 * fmin(ex, ey);
    c.exit_axis = ex == end ? kAxisX : ey == end ? kAxisY : l.zd > 0 ? kAxisNone : kAxisZ;
    return true;
}

// Walks from w (inside the grid, `done` false) until visit, called for every voxel entered, returns
// true, or the walk leaves the grid, or more than max_steps steps have been taken (limit is then set).
// All lanes of the warp call it; those with done set do nothing.  Leaves the last voxel in w.vx, w.vy,
// w.vz, w.voxel, and returns the axis last crossed, kAxisNone if w.x, w.y, w.z are those of the last
// voxel.  `slopes` gives the line's slopes, only where a step needs them.
// visit(voxel, step, timed) is also called without a step (step = false), with any voxel of the grid, and
// returns false then; timed tells the steps by crossing times, which never enter a voxel twice.
enum WalkMode { kReferenceWalk, kTimedWalk, kMixedWalk };
// kMode: every step the reference's, lane by lane (kReferenceWalk); by crossing times in the lanes that can
// (kMixedWalk); kTimedWalk: by crossing times in the warps all of whose lanes can, and stay below the grid's top
// for half of their way or more.  A lane without crossing times walks alone while the rest of its warp waits,
// and then waits itself, where with all lanes in step the reference's steps take twice the time of the others.
template <WalkMode kMode, class Slopes, class Visit>
__device__ __forceinline__ int walk_3D(const PreGeom& g, const WalkLine& l, const CrossingTimes& times, bool fast, bool done,
                                       const Slopes& slopes, const Visit& visit, int max_steps, WalkState& w, bool& limit)
{
    limit = false;
    if (kMode == kReferenceWalk || (kMode == kTimedWalk && __any_sync(0xffffffffu, !done && (!fast || times.above)))) {
        if (done) return kAxisNone;
        const WalkSlopes m = slopes();
        for (int steps = 0; !done;) {
            take_3D_step(g, l.xd, l.yd, l.zd, m.dy_dx, m.dz_dx, m.dz_dy, m.dx_dy, m.dx_dz, m.dy_dz, l.x0, l.y0, l.z0, w);
            done = walk_outside(g, w) || visit(w.voxel, true, false);
            if (!done && ++steps > max_steps) {
                limit = true;
                done = true;
            }
        }
        return kAxisNone;
    }
    CrossingTimes c = times;
    const int vx0 = w.vx, vy0 = w.vy, vz0 = w.vz;
    int voxel = w.voxel, before = voxel, extra = 0;  // before: the last step; extra: steps that did not move one index
    bool left = false;
    const bool walked = !done;
    if (done) voxel = before = 0;  // any index that may be looked at
    // a step that is not certain leaves its lane as it is, and so does every step after it, until the
    // reference's step below has been taken; a lane that is done has stop = 0
    if (done || !fast) c.stop = 0;
    auto last_axis = [&]() {
        const int d = voxel - before;
        return d == 0 ? kAxisNone : d == c.ix ? kAxisX : d == c.iy ? kAxisY : kAxisZ;
    };
    for (;;) {
        bool stuck;
        do {
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const unsigned t = min(min(c.tx, c.ty), c.tz), far = t + c.lead;
                const bool px = c.tx <= far, py = c.ty <= far, pz = c.tz <= far;
                const bool go = !((px && py) || (px && pz) || (py && pz) || t >= c.stop);
                if (go) before = voxel;
                if (go && px) {
                    c.tx += c.bx;
                    voxel += c.ix;
                }
                if (go && py) {
                    c.ty += c.by;
                    voxel += c.iy;
                }
                if (go && pz) {
                    c.tz += c.bz;
                    voxel += c.iz;
                }
                if (visit(voxel, go, true)) {
                    done = true;
                    c.stop = 0;
                }
                stuck = !go && !done;
            }
        } while (!__any_sync(0xffffffffu, stuck) && __any_sync(0xffffffffu, !done));
        if (stuck && fast) {
            // a crossing that is certain and leaves the grid (not through its top) ends the walk here
            const unsigned t = min(min(c.tx, c.ty), c.tz), far = t + c.lead;
            const bool px = c.tx <= far, py = c.ty <= far, pz = c.tz <= far;
            if (px + py + pz == 1 && (px ? kAxisX : py ? kAxisY : kAxisZ) == c.exit_axis && far >= 1073741824u) {
                left = done = true;
                c.stop = 0;
                stuck = false;
            }
        }
        if (stuck) {
            const WalkSlopes m = slopes();
            const int slab = g.columns * g.rows;
            w.vz = voxel / slab;
            w.vy = (voxel - w.vz * slab) / g.columns;
            w.vx = voxel - w.vz * slab - w.vy * g.columns;
            int axis = last_axis(), moved;
            face_position(g, l, m, axis, w);
            face_distances(g, l, axis, w);
            do {
                // near the grid's end every step is the reference's: beyond its top the slice index is
                // clamped, and the coordinates no longer follow from the last face
                if (min(min(c.tx, c.ty), c.tz) >= c.stop) fast = false;
                const int vx = w.vx, vy = w.vy, vz = w.vz;
                take_3D_step(g, l.xd, l.yd, l.zd, m.dy_dx, m.dz_dx, m.dz_dy, m.dx_dy, m.dx_dz, m.dy_dz, l.x0, l.y0, l.z0, w);
                left = walk_outside(g, w);
                voxel = w.voxel;
                if (w.vx != vx) c.tx += c.bx;
                if (w.vy != vy) c.ty += c.by;
                if (w.vz != vz) c.tz += c.bz;
                moved = (w.vx != vx) + (w.vy != vy) + (w.vz != vz);
                axis = w.vx != vx ? kAxisX : w.vy != vy ? kAxisY : kAxisZ;
                done = left || visit(voxel, true, false);
                extra += 1 - moved;
                if (!done && abs(w.vx - vx0) + abs(w.vy - vy0) + abs(w.vz - vz0) + extra > max_steps) {
                    limit = true;
                    done = true;
                }
                // a step across one face can be set up again from that face, one across an edge cannot
            } while (!done && (moved != 1 || !fast));
            before = done ? voxel : voxel - (axis == kAxisX ? c.ix : axis == kAxisY ? c.iy : c.iz);
            if (done || !fast) c.stop = 0;
        }
        __syncwarp();
        if (!__any_sync(0xffffffffu, !done)) break;
    }
    if (walked && !left) {
        const int slab = g.columns * g.rows;
        w.vz = voxel / slab;
        w.vy = (voxel - w.vz * slab) / g.columns;
        w.vx = voxel - w.vz * slab - w.vy * g.columns;
        w.voxel = voxel;
    }
    return last_axis();
}

// Processing order of the voxel walks.  A history's walk lengths depend on where its line crosses
// the grid: its distance t from the z axis and its direction (the chord for the hull walk, the gap
// to the hull for the endpoint walks), and one thread walks one history, so neighbouring threads
// should have similar lines.  The key is t in kWalkT buckets of the cylinder radius, times the
// line's direction (mod pi) in dir_buckets buckets: measured on a 20M-proton head scan, direction
// buckets shorten the endpoint walks (38.2 -> 31.2 ms; t alone 33.8) but not the hull walks, which
// run entry to exit (23.0 -> 21.5 ms with t alone, 23.7 with 32 directions).  The order changes no
// result (integer counts, per-history endpoints).
constexpr int kWalkT = 32, kWalkDir = 32;
__global__ void walk_order_key_kernel(long long n, const float* __restrict__ xe, const float* __restrict__ ye,
                                      const float* __restrict__ xo, const float* __restrict__ yo, float R,
                                      int dir_buckets, int* __restrict__ key)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float dx = xo[i] - xe[i], dy = yo[i] - ye[i];
    const float len = sqrtf(dx * dx + dy * dy);
    const float t = len > 0.f ? fabsf(xe[i] * yo[i] - xo[i] * ye[i]) / len : 0.f;
    int kt = (int)(t / R * kWalkT);
    kt = kt < 0 ? 0 : (kt >= kWalkT ? kWalkT - 1 : kt);
    float a = atan2f(dy, dx);
    if (a < 0.f) a += 3.14159265f;  // direction mod pi
    int ka = (int)(a / 3.14159265f * dir_buckets);
    ka = ka < 0 ? 0 : (ka >= dir_buckets ? dir_buckets - 1 : ka);
    key[i] = kt * dir_buckets + ka;
}

// SC_GPU / MSC_GPU / SM_GPU (B.cu:6681-7099) in one pass.  The three reference kernels walk the
// same straight line from the entry to the exit voxel and differ only in their WEPL window and in
// what they do at each voxel: SC carves (writes 0), MSC and SM count.  Here each history walks once
// and applies every hull whose window (and *_ON switch) it satisfies, so the voxel sequence each
// hull sees is the one its own kernel would walk.
enum HullMask { kHullSC = 1, kHullMSC = 2, kHullSM = 4 };
struct HullImages {
    uint8_t* sc;  // null where the hull is off
    int *msc, *sm;
};

__device__ __forceinline__ int hull_mask(const PreGeom& g, const HullImages& im, float wepl)
{
    const bool sc = im.sc && (wepl <= g.sc_upper) && (wepl >= g.sc_lower);
    const bool msc = im.msc && (wepl <= g.msc_upper) && (wepl >= g.msc_lower);
    const bool sm = im.sm && (wepl >= g.sm_lower);
    return (sc ? kHullSC : 0) | (msc ? kHullMSC : 0) | (sm ? kHullSM : 0);
}

__device__ __forceinline__ void hull_mark(const HullImages& im, int mask, int voxel, int count)
{
    if (mask & kHullSC) im.sc[voxel] = 0;
    if (mask & kHullMSC) atomicAdd(im.msc + voxel, count);
    if (mask & kHullSM) atomicAdd(im.sm + voxel, count);
}

// The walk of history i, by all lanes of a warp (have = false: without one); count(voxel, timed) is called
// for every voxel but the last.
template <WalkMode kMode, class Count>
__device__ __forceinline__ void hull_walk(const PreGeom& g, bool have, long long i, const GeomPtrs& G, const Count& count,
                                          unsigned long long* counters)
{
    float xe = 0, ye = 0, ze = 0, xo = 0, yo = 0, zo = 0;
    if (have) {
        xe = G.a[kXE][i];
        ye = G.a[kYE][i];
        ze = G.a[kZE][i];
        xo = G.a[kXO][i];
        yo = G.a[kYO][i];
        zo = G.a[kZO][i];
    }
    bool done = !have;
    const double X0 = -g.R, Y0 = g.R, Z0 = g.H / 2;
    const WalkLine l{xe, ye, ze, (xe <= xo) - (xe >= xo), (ye <= yo) - (ye >= yo), (ze <= zo) - (ze >= zo)};
    WalkState w;
    w.x = xe;
    w.y = ye;
    w.z = ze;
    w.vx = calculate_voxel(X0, xe, g.voxel_width);
    w.vy = calculate_voxel(Y0, ye, g.voxel_height);
    w.vz = calculate_voxel(Z0, ze, g.voxel_thickness);
    w.voxel = w.vx + w.vy * g.columns + w.vz * g.columns * g.rows;
    face_distances(g, l, kAxisNone, w);
    const float dx = __fsub_rn(xo, xe), dy = __fsub_rn(yo, ye), dz = __fsub_rn(zo, ze);
    auto slopes = [&]() {
        return WalkSlopes{(double)__fdiv_rn(dy, dx), (double)__fdiv_rn(dz, dx), (double)__fdiv_rn(dz, dy),
                          (double)__fdiv_rn(dx, dy), (double)__fdiv_rn(dx, dz), (double)__fdiv_rn(dy, dz)};
    };
    const int voxel_out = calculate_voxel(X0, xo, g.voxel_width) + calculate_voxel(Y0, yo, g.voxel_height) * g.columns +
                          calculate_voxel(Z0, zo, g.voxel_thickness) * g.columns * g.rows;
    auto mark = [&](int voxel, bool step, bool timed) {
        const bool end = step && voxel == voxel_out;
        if (step && !end) count(voxel, timed);
        return end;
    };
    if (!done) done = walk_outside(g, w) || mark(w.voxel, true, true);
    const int max_steps = 4 * (g.columns + g.rows + g.slices) + 16;
    // the slopes are float quotients of dx, dy and dz, 2^-24 off each; a comparison involves up to four
    CrossingTimes times{};
    const bool flat = l.zd == 0;
    const bool fast = kMode != kReferenceWalk && !done && !flat && crossing_times(g, l, w, fabs((double)dx), fabs((double)dy), fabs((double)dz),
                                                                 5.0e-7, times);
    bool limit;
    walk_3D<kMode>(g, l, times, fast, done || flat, slopes, mark, max_steps, w, limit);
    if (flat && !done) {
        const WalkSlopes m = slopes();
        int steps = 0;
        while (!done) {
            take_2D_step(g, l.xd, l.yd, m.dy_dx, m.dx_dy, xe, ye, w);
            done = (w.voxel == voxel_out) || walk_outside(g, w);
            if (!done) mark(w.voxel, true, false);
            if (++steps > max_steps) {
                limit = true;
                break;
            }
        }
    }
    if (limit) atomicAdd(counters + kCntWaitExpired, 1ull);
}

// One thread per history, every mark an atomic on its image: bound by the L2's atomics, 155 G/s.
template <WalkMode kMode>
__global__ void __launch_bounds__(128) hull_walks_kernel(PreGeom g, long long n, const int* __restrict__ order, GeomPtrs G,
                                                         const float* __restrict__ WEPL, const uint8_t* __restrict__ missed,
                                                         HullImages im, unsigned long long* counters)
{
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long i = k < n ? order[k] : 0;
    const int mask = k < n && !missed[i] ? hull_mask(g, im, WEPL[i]) : 0;
    hull_walk<kMode>(g, mask != 0, i, G, [&](int voxel, bool) { hull_mark(im, mask, voxel, 1); }, counters);
}

// The same with the marks counted in shared memory.  All histories of one mask mark the same voxels in
// the same images, so one 16-bit count per voxel serves them; a CTA counts those of a window of as many
// slices as shared memory holds and adds the window to the images when the mask or the window
// changes.  The histories are sorted by (mask, first slice they touch, distance from the axis); a CTA
// takes a contiguous range of them, and the ranges cost the same by the chords' lengths.  Marks
// outside the window, and those of the reference's own steps, go to the images directly.
// On the head scan (4M histories, 650M marks, windows of two slices) 1.61 ms against 4.21 ms with every
// mark in L2, bound by the walks' instructions; before the steps were shortened 768 threads took 1.75 ms,
// 512 1.97 and 1024 (which spill) 1.74.
// The line lies where the windows win with any number of marks.  Order and walks of 300k / 600k / 1.2M histories,
// us, windows and (every mark in L2): 200x200x32 voxels with all histories marked 362 / 455 / 753 (498 / 966 / 1877),
// a third of them 132 / 174 / 250 (213 / 394 / 768), almost none 29 / 32 / 40 (24 / 36 / 60); 128x128x16 227 / 309 / 489
// (467 / 873 / 1741), 121 / 164 / 219 (221 / 446 / 803), 27 / 29 / 37 (24 / 36 / 60); 316x316x8, a window of one slice, 512 /
// 825 / 1574 (817 / 1565 / 2998), 246 / 326 / 468 (406 / 683 / 1370), 27 / 29 / 37 (25 / 37 / 60).  From 262,144 on, the
// preprocessing of a 300,000-proton scan of a cylinder that fills the grid takes 1066 us where it takes 1037.
constexpr long long kHullWindowMin = 1 << 19;
constexpr int kHullKeys = 4096, kHullThreads = 768, kHullWindow = 200 * 1024;
// histories between two additions of the window: a timed step enters a voxel once, so counts stay below 2^16
constexpr int kHullFlush = 65000;

struct HullPlan {
    int window;     // slices of a window (0: one does not fit)
    int first;      // window starts: 0 .. first - 1
    int distances;  // buckets of the distance from the axis
};
HullPlan hull_plan(const PreGeom& g)
{
    HullPlan p{};
    const long long fit = kHullWindow / (2LL * g.columns * g.rows);
    p.window = (int)(fit < g.slices ? fit : g.slices);
    p.first = g.slices - p.window + 1;
    p.distances = kHullKeys / (8 * p.first);
    if (p.distances > 32) p.distances = 32;
    if (p.distances == 0) p.window = 0;
    return p;
}

__global__ void hull_key_kernel(PreGeom g, HullPlan plan, long long n, GeomPtrs G, const float* __restrict__ WEPL,
                                const uint8_t* __restrict__ missed, HullImages im, int* __restrict__ key)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int mask = !missed[i] ? hull_mask(g, im, WEPL[i]) : 0;
    if (mask == 0) {
        key[i] = 0;
        return;
    }
    const float xe = G.a[kXE][i], ye = G.a[kYE][i], xo = G.a[kXO][i], yo = G.a[kYO][i];
    const float dx = xo - xe, dy = yo - ye, len = sqrtf(dx * dx + dy * dy);
    const float t = len > 0.f ? fabsf(xe * yo - xo * ye) / len : 0.f;
    const int kt = (int)fminf(t / (float)g.R * plan.distances, (float)(plan.distances - 1));
    const int z = min(calculate_voxel(g.H / 2, G.a[kZE][i], g.voxel_thickness), calculate_voxel(g.H / 2, G.a[kZO][i], g.voxel_thickness));
    key[i] = (mask * plan.first + max(0, min(z, plan.first - 1))) * plan.distances + max(kt, 0);
}

// starts[b]: where CTA b's range begins.  hist: histories of each key, in descending order of the keys.
__global__ void __launch_bounds__(1024) hull_ranges_kernel(PreGeom g, HullPlan plan, const unsigned* __restrict__ hist, int blocks,
                                                           int* __restrict__ starts)
{
    __shared__ unsigned long long cost[1024];
    __shared__ unsigned count[1024];
    const int keys = 8 * plan.first * plan.distances, none = plan.first * plan.distances, per = (keys + 1023) / 1024;
    auto weight = [&](int key) {  // of a history: its setup and its steps
        const double t = (key % plan.distances + 0.5) / plan.distances;
        return key < none ? 0u : (unsigned)(60.0 + 2.5 * g.R * sqrt(1.0 - t * t) / g.voxel_width);
    };
    unsigned long long own_cost = 0;
    unsigned own = 0;
    for (int j = 0; j < per; j++) {
        const int key = keys - 1 - ((int)threadIdx.x * per + j);
        if (key < 0) break;
        own += hist[key];
        own_cost += (unsigned long long)hist[key] * weight(key);
    }
    cost[threadIdx.x] = own_cost;
    count[threadIdx.x] = own;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        const unsigned long long c = threadIdx.x >= o ? cost[threadIdx.x - o] : 0;
        const unsigned m = threadIdx.x >= o ? count[threadIdx.x - o] : 0;
        __syncthreads();
        cost[threadIdx.x] += c;
        count[threadIdx.x] += m;
        __syncthreads();
    }
    const unsigned long long total = cost[1023];
    for (int b = threadIdx.x; b <= blocks; b += 1024) {
        const unsigned long long target = total / blocks * b + total % blocks * b / blocks;
        int lo = 0, hi = 1023;  // the first thread whose keys reach the target
        while (lo < hi) {
            const int mid = (lo + hi) / 2;
            if (cost[mid] >= target) hi = mid;
            else lo = mid + 1;
        }
        unsigned long long c = lo ? cost[lo - 1] : 0;
        unsigned position = lo ? count[lo - 1] : 0;
        for (int j = 0; j < per; j++) {
            const int key = keys - 1 - (lo * per + j);
            if (key < none) break;
            const unsigned long long here = (unsigned long long)hist[key] * weight(key);
            if (c + here >= target) {
                position += (unsigned)((target - c) / weight(key));
                break;
            }
            c += here;
            position += hist[key];
        }
        starts[b] = (int)position;
    }
}

__global__ void __launch_bounds__(kHullThreads, 1)
    hull_window_kernel(PreGeom g, HullPlan plan, const int* __restrict__ order, const int* __restrict__ key,
                       const unsigned* __restrict__ bucket_end, const int* __restrict__ starts, GeomPtrs G, HullImages im,
                       unsigned long long* counters)
{
    extern __shared__ unsigned window[];
    __shared__ int next;
    const int lane = threadIdx.x & 31, slab = g.columns * g.rows, voxels = plan.window * slab, words = (voxels + 1) / 2;
    for (int k = threadIdx.x; k < words; k += blockDim.x) window[k] = 0;
    const int end = starts[blockIdx.x + 1];
    for (int p = starts[blockIdx.x]; p < end;) {
        const int group = key[order[p]] / plan.distances, mask = group / plan.first;
        const int base = (group - mask * plan.first) * slab;
        const int last = min(min(end, (int)bucket_end[group * plan.distances]), p + kHullFlush);
        if (threadIdx.x == 0) next = p;
        __syncthreads();
        for (;;) {
            int first;
            if (lane == 0) first = atomicAdd(&next, 32);
            first = __shfl_sync(0xffffffffu, first, 0);
            if (first >= last) break;
            const bool have = first + lane < last;
            hull_walk<kMixedWalk>(g, have, have ? order[first + lane] : 0, G,
                      [&](int voxel, bool timed) {
                          const unsigned local = (unsigned)(voxel - base);
                          if (timed && local < (unsigned)voxels) atomicAdd(window + (local >> 1), (local & 1) ? 0x10000u : 1u);
                          else hull_mark(im, mask, voxel, 1);
                      },
                      counters);
        }
        __syncthreads();
        for (int k = threadIdx.x; k < words; k += blockDim.x) {
            const unsigned both = window[k];
            if (both == 0) continue;
            window[k] = 0;
            if (both & 0xffffu) hull_mark(im, mask, base + 2 * k, both & 0xffffu);
            if (both >> 16) hull_mark(im, mask, base + 2 * k + 1, both >> 16);
        }
        p = last;
    }
}

// MSC_edge_detection_GPU (B.cu:6911-6956), out of place: 3x3 maximum difference over the
// interior, threshold on the difference or the count, then the cylinder mask.
__global__ void msc_edge_kernel(PreGeom g, const int* __restrict__ counts, int* __restrict__ out)
{
    const long long voxel = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (voxel >= g.num_voxels) return;
    const long long CR = (long long)g.columns * g.rows;
    const int slice = (int)(voxel / CR), rem = (int)(voxel % CR), row = rem / g.columns, column = rem % g.columns;
    const float x = (float)((column - g.columns / 2 + 0.5) * g.voxel_width);
    const float y = (float)((g.rows / 2 - row - 0.5) * g.voxel_height);
    int max_difference = 0;
    if ((row != 0) && (row != g.rows - 1) && (column != 0) && (column != g.columns - 1)) {
        for (int r = row - 1; r <= row + 1; r++)
            for (int c = column - 1; c <= column + 1; c++) {
                const int difference = counts[voxel] - counts[c + r * g.columns + slice * CR];
                if (difference > max_difference) max_difference = difference;
            }
    }
    int result = (max_difference > g.msc_diff_thresh || counts[voxel] > g.msc_diff_thresh) ? 0 : 1;
    const double half = (g.voxel_width > g.voxel_height ? g.voxel_width : g.voxel_height) / 2;
    if (__fadd_rn(powf(x, 2.0f), powf(y, 2.0f)) >= powf((float)(g.R - half), 2.0f)) result = 0;
    out[voxel] = result;
}

// carve_differences (B.cu:6616-6634): interior 3x3 maximum difference
__global__ void carve_differences_kernel(PreGeom g, const int* __restrict__ image, int* __restrict__ diff)
{
    const long long voxel = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (voxel >= g.num_voxels) return;
    const long long CR = (long long)g.columns * g.rows;
    const int slice = (int)(voxel / CR), rem = (int)(voxel % CR), row = rem / g.columns, column = rem % g.columns;
    int max_difference = 0;
    if ((row != 0) && (row != g.rows - 1) && (column != 0) && (column != g.columns - 1)) {
        for (int r = row - 1; r <= row + 1; r++)
            for (int c = column - 1; c <= column + 1; c++) {
                const int difference = image[voxel] - image[c + r * g.columns + slice * CR];
                if (difference > max_difference) max_difference = difference;
            }
        diff[voxel] = max_difference;
    } else {
        diff[voxel] = 0;
    }
}

// SM_edge_detection's host threshold search (B.cu:7118-7133): per slice, the count at the first
// voxel (in index order) holding the slice's largest positive difference; 0 if none is positive.
// One 256-thread CTA per slice; the winner is the smallest index among maximal differences.
__global__ void sm_threshold_kernel(PreGeom g, const int* __restrict__ diff, const int* __restrict__ counts,
                                    int* __restrict__ thresholds)
{
    const int slice = blockIdx.x;
    const long long CR = (long long)g.columns * g.rows;
    const long long base = slice * CR;
    int best = 0;
    long long best_idx = -1;
    for (long long p = threadIdx.x; p < CR; p += blockDim.x) {
        const int d = diff[base + p];
        if (d > best) {  // within a thread indices increase, so the first maximum is kept
            best = d;
            best_idx = p;
        }
    }
    __shared__ int s_best[256];
    __shared__ long long s_idx[256];
    s_best[threadIdx.x] = best;
    s_idx[threadIdx.x] = best_idx;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            const int b2 = s_best[threadIdx.x + o];
            const long long i2 = s_idx[threadIdx.x + o];
            if (b2 > s_best[threadIdx.x] || (b2 == s_best[threadIdx.x] && b2 > 0 && i2 >= 0 &&
                                              (s_idx[threadIdx.x] < 0 || i2 < s_idx[threadIdx.x]))) {
                s_best[threadIdx.x] = b2;
                s_idx[threadIdx.x] = i2;
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) thresholds[slice] = s_idx[0] >= 0 ? counts[base + s_idx[0]] : 0;
}

// SM_edge_detection_GPU (B.cu:7160-7175)
__global__ void sm_edge_kernel(PreGeom g, int* __restrict__ counts, const int* __restrict__ thresholds)
{
    const long long voxel = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (voxel >= g.num_voxels) return;
    const long long CR = (long long)g.columns * g.rows;
    const int slice = (int)(voxel / CR), rem = (int)(voxel % CR), row = rem / g.columns, column = rem % g.columns;
    const float x = (float)((column - g.columns / 2 + 0.5) * g.voxel_width);
    const float y = (float)((g.rows / 2 - row - 0.5) * g.voxel_height);
    int v = (counts[voxel] > g.sm_scale * thresholds[slice]) ? 1 : 0;
    const double half = (g.voxel_width > g.voxel_height ? g.voxel_width : g.voxel_height) / 2;
    if (__fadd_rn(powf(x, 2.0f), powf(y, 2.0f)) >= powf((float)(g.R - half), 2.0f)) v = 0;
    counts[voxel] = v;
}

__global__ void counts_to_hull_kernel(long long n, const int* __restrict__ counts, uint8_t* __restrict__ hull)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) hull[i] = counts[i] == 1 ? 1 : 0;
}

// initial_iterate_generate_hybrid (B.cu:8582-8591): x = FBP where the hull is set, else 0
__global__ void hybrid_kernel(long long n, const uint8_t* __restrict__ hull, const float* __restrict__ fbp, float* __restrict__ x)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = hull[i] ? fbp[i] : 0.0f;
}

// The hull as bits: 160 KB for 1.28 million voxels, which stay in L1 where the bytes did not.
__global__ void hull_bits_kernel(long long words, long long n, const uint8_t* __restrict__ hull, uint32_t* __restrict__ bits)
{
    const long long word = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (word >= words) return;  // whole warps: a warp writes one word
    const long long v = word * 32 + (threadIdx.x & 31);
    const unsigned b = __ballot_sync(0xffffffffu, v < n && hull[v] == 1);
    if ((threadIdx.x & 31) == 0) bits[word] = b;
}

// find_MLP_endpoints_GPU (B.cu:7581-7773): walk from the cylinder point along the straight line
// (angle + PI when leaving) until the first hull voxel or the image edge.  All lanes of a warp call it;
// lanes without a history (have = false) walk nothing.
template <WalkMode kMode>
__device__ __forceinline__ bool find_endpoint(const PreGeom& g, const uint32_t* __restrict__ bits, bool have, double x_start,
                                              double y_start, double z_start, double xy_angle, double xz_angle,
                                              double& x_object, double& y_object, double& z_object, int& voxel_x,
                                              int& voxel_y, int& voxel_z, bool entering)
{
    if (!entering) xy_angle += kPi;
    WalkLine l{x_start, y_start, z_start, 0, 0, 0};
    l.xd = (cos(xy_angle) >= 0) - (cos(xy_angle) <= 0);
    l.yd = (sin(xy_angle) >= 0) - (sin(xy_angle) <= 0);
    l.zd = (sin(xz_angle) >= 0) - (sin(xz_angle) <= 0);
    if (l.xd < 0) l.zd *= -1;
    WalkState w;
    w.x = x_start;
    w.y = y_start;
    w.z = z_start;
    w.vx = calculate_voxel(-g.R, x_start, g.voxel_width);
    w.vy = calculate_voxel(g.R, y_start, g.voxel_height);
    w.vz = calculate_voxel(g.H / 2, z_start, g.voxel_thickness);
    w.voxel = w.vx + (w.vy + w.vz * g.rows) * g.columns;
    face_distances(g, l, kAxisNone, w);
    const double tan_xy = tan(xy_angle), tan_xz = tan(xz_angle);
    auto slopes = [&]() {
        return WalkSlopes{tan_xy, tan_xz, tan_xz / tan_xy, (double)powf((float)tan_xy, -1.0f),
                          (double)powf((float)tan_xz, -1.0f), tanf((float)xy_angle) / tan_xz};
    };
    bool hit_hull = false;
    auto visit = [&](int voxel, bool step, bool) {
        const bool hit = step && ((__ldg(bits + (voxel >> 5)) >> (voxel & 31)) & 1u);
        hit_hull = hit_hull || hit;
        return hit;
    };
    bool done = !have || walk_outside(g, w);
    if (!done) done = visit(w.voxel, true, false);
    // every pass moves one index monotonically, so the walk leaves the grid within this bound
    const int max_steps = 2 * (g.columns + g.rows + g.slices) + 16;
    // slopes: tan in double, powf of a float within 4 units in the last place (5.4e-7 with the float's own
    // rounding), and for y after a z crossing tanf (4 units) of the angle as a float, whose rounding
    // changes the tangent by 2 / |sin 2 angle| = tan + 1 / tan times that
    const double a_xy = fabs(tan_xy), a_xz = fabs(tan_xz), scale = 1.0 / fmax(fmax(a_xy, a_xz), 1.0);
    CrossingTimes times{};
    const bool flat = l.zd == 0;
    const double turn = 1.2e-7 * fabs(xy_angle) + 1.0e-7;
    // an elevation beyond a right angle moves z against its own direction: left to the reference's steps
    const bool forward = (tan_xy > 0) == (l.xd * l.yd > 0) && (tan_xz > 0) == (l.xd * l.zd > 0);
    const bool fast = kMode != kReferenceWalk && !done && !flat && forward && crossing_times(g, l, w, scale, a_xy * scale, a_xz * scale,
                                                       2.4e-6 + turn * (a_xy + 1.0 / a_xy), times);
    bool limit;
    int axis = walk_3D<kMode>(g, l, times, fast, done || flat, slopes, visit, max_steps - 1, w, limit);
    if (flat && !done) {
        // the reference's 2D loop of this walk (B.cu:7718-7752) keeps its slice index and its start height
        const double delta_yx = fabs(tan_xy);
        const WalkSlopes m = slopes();
        int steps = 0;
        while (!done && steps++ < max_steps) {
            const double y_extension = w.y_to_go / delta_yx;
            if (w.x_to_go <= y_extension) {
                w.vx += l.xd;
                w.x = edge_coordinate(-g.R, w.vx, g.voxel_width, 1, l.xd);
                w.y = corresponding_coordinate(m.dy_dx, w.x, x_start, y_start);
                w.x_to_go = g.voxel_width;
                w.y_to_go = distance_remaining(g.R, w.y, -1, l.yd, g.voxel_height, w.vy);
            } else {
                w.vy -= l.yd;
                // the reference passes Z_INCREASING_DIRECTION here (B.cu:7736); it equals Y's
                w.y = edge_coordinate(g.R, w.vy, g.voxel_height, -1, l.yd);
                w.x = corresponding_coordinate(m.dx_dy, w.y, y_start, x_start);
                w.x_to_go = distance_remaining(-g.R, w.x, 1, l.xd, g.voxel_width, w.vx);
                w.y_to_go = g.voxel_height;
            }
            if (w.x_to_go == 0) {
                w.x_to_go = g.voxel_width;
                w.vx += l.xd;
            }
            if (w.y_to_go == 0) {
                w.y_to_go = g.voxel_height;
                w.vy -= l.yd;
            }
            w.voxel = w.vx + w.vy * g.columns + w.vz * g.columns * g.rows;
            done = walk_outside(g, w);
            if (!done) done = visit(w.voxel, true, false);
        }
        axis = kAxisNone;
    } else if (hit_hull && axis != kAxisNone) {
        face_position(g, l, slopes(), axis, w);  // where the reference's step left x, y and z
    }
    voxel_x = w.vx;
    voxel_y = w.vy;
    voxel_z = w.vz;
    if (hit_hull) {
        x_object = w.x;
        y_object = w.y;
        z_object = w.z;
    }
    return hit_hull;
}

// collect_MLP_endpoints_GPU_nobool (B.cu:7819-7854).  Six CTAs per SM: 2.53 ms for 3.3M histories, five
// 2.63 ms (before the steps were shortened: six 3.20 ms, four 4.26, eight, which spill, 3.34).
template <WalkMode kMode>
__global__ void __launch_bounds__(128, 6) endpoints_kernel(PreGeom g, long long n, const int* __restrict__ order,
                                                           const uint32_t* __restrict__ hull_bits, GeomPtrs G,
                                                           uint32_t* __restrict__ first_voxel, int* __restrict__ keep)
{
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool have = k < n;
    const long long i = have ? order[k] : 0;
    float p[kNumGeom];
#pragma unroll
    for (int a = 0; a < kNumGeom; a++) p[a] = have ? G.a[a][i] : 0.5f;
    int vx = 0, vy = 0, vz = 0, vx2 = 0, vy2 = 0, vz2 = 0;
    double xin = 0, yin = 0, zin = 0, xout = 0, yout = 0, zout = 0;
    const bool entered =
        find_endpoint<kMode>(g, hull_bits, have, p[kXE], p[kYE], p[kZE], p[kXYE], p[kXZE], xin, yin, zin, vx, vy, vz, true);
    const bool exited = find_endpoint<kMode>(g, hull_bits, have && entered, p[kXO], p[kYO], p[kZO], p[kXYO], p[kXZO], xout, yout,
                                      zout, vx2, vy2, vz2, false);
    if (!have) return;
    if (entered && exited) {
        first_voxel[i] = (uint32_t)(vx + g.columns * vy + g.rows * g.columns * vz);
        G.a[kXE][i] = (float)xin;
        G.a[kYE][i] = (float)yin;
        G.a[kZE][i] = (float)zin;
        G.a[kXO][i] = (float)xout;
        G.a[kYO][i] = (float)yout;
        G.a[kZO][i] = (float)zout;
        keep[i] = 1;
    } else {
        first_voxel[i] = (uint32_t)g.num_voxels;
        keep[i] = 0;
    }
}

// stable compaction of the history vectors: out[offsets[i]] = in[i] where keep[i]
struct CompactArrays {
    const float* in_f[kNumGeom + 1];
    float* out_f[kNumGeom + 1];
    const int* in_i[2];
    int* out_i[2];
    int nf, ni;
};
__global__ void compact_kernel(long long n, const int* __restrict__ keep, const long long* __restrict__ offsets, CompactArrays c)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !keep[i]) return;
    const long long o = offsets[i];
    for (int k = 0; k < c.nf; k++) c.out_f[k][o] = c.in_f[k][i];
    for (int k = 0; k < c.ni; k++) c.out_i[k][o] = c.in_i[k][i];
}

__global__ void u8_to_int_kernel(long long n, const uint8_t* __restrict__ in, int invert, int* __restrict__ out)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = invert ? !in[i] : in[i];
}

unsigned grid_for(long long n, int threads) { return (unsigned)((n + threads - 1) / threads); }

}  // namespace

}  // namespace pct

// ==========================================================================================
// C ABI
// ==========================================================================================

using pct::Preproc;

namespace {

pct_status fail(pct_ctx* ctx, pct_status st, const std::string& what, cudaError_t e = cudaSuccess)
{
    if (ctx) {
        ctx->last_error = what;
        if (e != cudaSuccess) ctx->last_error += " -> " + pct::cuda_error_string(e);
    }
    return st;
}

#define PRE_TRY(expr, what)                                             \
    do {                                                                \
        cudaError_t _e = (expr);                                        \
        if (_e != cudaSuccess) return fail(ctx, PCT_ERR_CUDA, what, _e); \
    } while (0)

template <class T>
cudaError_t alloc(T*& p, long long n)
{
    cudaFree(p);
    p = nullptr;
    return cudaMalloc(&p, sizeof(T) * (size_t)(n > 0 ? n : 1));
}

Preproc* pre_of(pct_ctx* ctx)
{
    if (!ctx->pre) ctx->pre = new Preproc();
    return ctx->pre;
}

pct::GeomPtrs geom_ptrs(float* const a[pct::kNumGeom])
{
    pct::GeomPtrs g;
    for (int k = 0; k < pct::kNumGeom; k++) g.a[k] = a[k];
    return g;
}

// bins and images, sized once per context
pct_status ensure_fixed(pct_ctx* ctx, Preproc* p)
{
    if (p->bin_counts) return PCT_OK;
    const long long nb = ctx->cfg.NUM_BINS, nv = ctx->cfg.NUM_VOXELS;
    cudaError_t e = alloc(p->bin_counts, nb);
    float** fb[] = {&p->mean_WEPL, &p->mean_rel_ut_angle, &p->mean_rel_uv_angle, &p->stddev_WEPL, &p->stddev_rel_ut_angle,
                    &p->stddev_rel_uv_angle, &p->sinogram, &p->sinogram_filtered};
    for (float** q : fb)
        if (e == cudaSuccess) e = alloc(*q, nb);
    if (e == cudaSuccess) e = alloc(p->FBP_image, nv);
    if (e == cudaSuccess) e = alloc(p->FBP_median, nv);
    if (e == cudaSuccess) e = alloc(p->FBP_hull, nv);
    if (e == cudaSuccess) e = alloc(p->SC_hull, nv);
    if (e == cudaSuccess) e = alloc(p->hull, nv);
    if (e == cudaSuccess) e = alloc(p->MSC_counts, nv);
    if (e == cudaSuccess) e = alloc(p->SM_counts, nv);
    if (e == cudaSuccess) e = alloc(p->SM_differences, nv);
    if (e == cudaSuccess) e = alloc(p->edge_tmp, nv);
    if (e == cudaSuccess) e = alloc(p->walk_hist, 2 * pct::kHullKeys);
    if (e == cudaSuccess) e = alloc(p->hull_starts, pct::sm_count() + 1);
    if (e == cudaSuccess) e = alloc(p->hull_bits, (nv + 31) / 32);
    if (e == cudaSuccess) e = alloc(p->SM_thresholds, ctx->cfg.SLICES);
    const long long bins_tv = (long long)ctx->cfg.T_BINS * ctx->cfg.V_BINS;
    if (e == cudaSuccess) e = alloc(p->fbp_tables, ctx->cfg.T_BINS + bins_tv + 2LL * ctx->cfg.ANGULAR_BINS);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(ctx, PCT_ERR_NOMEM, "preprocessing arrays", e);
    }
    return PCT_OK;
}

pct_status ensure_scratch(pct_ctx* ctx, Preproc* p, long long n)
{
    if (n <= p->cap_scratch) return PCT_OK;
    cudaError_t e = alloc(p->flags, n);
    if (e == cudaSuccess) e = alloc(p->offsets, n + 1);
    if (e == cudaSuccess) e = alloc(p->scan_tmp, pct::scan_tile_scratch_elems(n));
    for (int k = 0; k < pct::kNumGeom && e == cudaSuccess; k++) e = alloc(p->tmp_geom[k], n);
    if (e == cudaSuccess) e = alloc(p->tmp_wepl, n);
    if (e == cudaSuccess) e = alloc(p->tmp_bin_num, n);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return fail(ctx, PCT_ERR_NOMEM, "compaction scratch", e);
    }
    p->cap_scratch = n;
    return PCT_OK;
}

// Walk order of n histories by the key above: keys in the compaction's int scratch, the order in
// the offsets array (both idle while the walks run).  Returns the order (device), or null if a
// launch failed.  Needs ensure_scratch(n).
int* walk_order(pct_ctx* ctx, Preproc* p, long long n, float* const geom[pct::kNumGeom], int dir_buckets)
{
    cudaStream_t s = ctx->stream;
    int* key = p->tmp_bin_num;
    int* order = reinterpret_cast<int*>(p->offsets);
    pct::walk_order_key_kernel<<<pct::grid_for(n, 256), 256, 0, s>>>(n, geom[pct::kXE], geom[pct::kYE], geom[pct::kXO],
                                                                     geom[pct::kYO], (float)ctx->cfg.RECON_CYL_RADIUS,
                                                                     dir_buckets, key);
    if (cudaGetLastError() != cudaSuccess) return nullptr;
    if (pct::bucket_sort_by_key(key, 0, n, pct::kWalkT * dir_buckets, p->walk_hist, order, s) != cudaSuccess)
        return nullptr;
    ctx->launches += 4;
    return order;
}

// Stable compaction of the current vectors by p->flags (1 = keep); returns the new length.
pct_status compact_vectors(pct_ctx* ctx, Preproc* p, long long n, long long* kept)
{
    cudaStream_t s = ctx->stream;
    PRE_TRY(pct::exclusive_scan_i32_to_i64(p->flags, n, p->offsets, p->scan_tmp, s), "compaction scan");
    long long total = 0;
    PRE_TRY(cudaMemcpyAsync(&total, p->offsets + n, sizeof(long long), cudaMemcpyDeviceToHost, s), "compaction count");
    pct::CompactArrays c{};
    int nf = 0;
    for (int k = 0; k < pct::kNumGeom; k++) {
        c.in_f[nf] = p->vec_geom[k];
        c.out_f[nf++] = p->tmp_geom[k];
    }
    c.in_f[nf] = p->vec_wepl;
    c.out_f[nf++] = p->tmp_wepl;
    c.nf = nf;
    c.in_i[0] = p->vec_bin_num;
    c.out_i[0] = p->tmp_bin_num;
    c.ni = 1;
    if (n > 0) pct::compact_kernel<<<pct::grid_for(n, 256), 256, 0, s>>>(n, p->flags, p->offsets, c);
    PRE_TRY(cudaGetLastError(), "compaction kernel");
    PRE_TRY(cudaStreamSynchronize(s), "compaction sync");
    for (int k = 0; k < pct::kNumGeom; k++) std::swap(p->vec_geom[k], p->tmp_geom[k]);
    std::swap(p->vec_wepl, p->tmp_wepl);
    std::swap(p->vec_bin_num, p->tmp_bin_num);
    p->n_vec = total;
    *kept = total;
    ctx->launches += 4;
    return PCT_OK;
}

}  // namespace

namespace pct {

// Device tracker arrays for n histories: dst[0..11] in the order of kTrackerNames, dst[12] WEPL,
// dst[13] the projection angle (degrees).  Grows the arrays when n exceeds their capacity.
pct_status preproc_reserve_tracker(pct_ctx* ctx, long long n, float* dst[kTrackerSlots])
{
    if (!ctx || n < 0 || n > 0x7fffffffLL) return PCT_ERR_ARG;
    cudaSetDevice(ctx->device);
    Preproc* p = pre_of(ctx);
    if (n > p->cap_raw) {
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < kNumTracker && e == cudaSuccess; k++) e = alloc(p->tracker[k], n);
        for (int k = 0; k < kNumGeom && e == cudaSuccess; k++) e = alloc(p->raw_geom[k], n);
        if (e == cudaSuccess) e = alloc(p->gantry_angle, n);
        if (e == cudaSuccess) e = alloc(p->raw_wepl, n);
        if (e == cudaSuccess) e = alloc(p->missed, n);
        if (e == cudaSuccess) e = alloc(p->raw_bin_num, n);
        if (e != cudaSuccess) {
            cudaGetLastError();
            p->cap_raw = 0;
            return fail(ctx, PCT_ERR_NOMEM, "tracker arrays", e);
        }
        p->cap_raw = n;
    }
    for (int k = 0; k < kNumTracker; k++) dst[k] = p->tracker[k];
    dst[kNumTracker] = p->raw_wepl;
    dst[kNumTracker + 1] = p->gantry_angle;
    return PCT_OK;
}

const uint8_t* preproc_hull(pct_ctx* ctx)
{
    return (ctx && ctx->pre && ctx->pre->hull_ready) ? ctx->pre->hull : nullptr;
}

// The tracker arrays hold n histories: reset the stage state.
void preproc_tracker_loaded(pct_ctx* ctx, long long n, int integer_angles)
{
    Preproc* p = pre_of(ctx);
    p->n_raw = n;
    p->integer_angles = integer_angles ? 1 : 0;
    p->n_vec = 0;
    p->hull_ready = false;
}

}  // namespace pct

extern "C" pct_status pct_load_tracker_data(pct_ctx* ctx, const pct_tracker_data* t, int64_t n, pct_memory where,
                                            int integer_angles)
{
    if (!ctx || !t || n < 0 || n > 0x7fffffffLL) return PCT_ERR_ARG;
    const float* src[pct::kTrackerSlots] = {t->t_in_1,  t->t_in_2,  t->t_out_1, t->t_out_2, t->u_in_1,
                                            t->u_in_2,  t->u_out_1, t->u_out_2, t->v_in_1,  t->v_in_2,
                                            t->v_out_1, t->v_out_2, t->WEPL,    t->gantry_angle};
    if (n > 0)
        for (const float* q : src)
            if (!q) return fail(ctx, PCT_ERR_ARG, "pct_load_tracker_data: NULL array");
    float* dst[pct::kTrackerSlots];
    pct_status st = pct::preproc_reserve_tracker(ctx, n, dst);
    if (st != PCT_OK) return st;
    const cudaMemcpyKind kind = where == PCT_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
    for (int k = 0; k < pct::kTrackerSlots && n > 0; k++)
        PRE_TRY(cudaMemcpyAsync(dst[k], src[k], sizeof(float) * n, kind, ctx->stream), "tracker copy");
    if (where == PCT_HOST) PRE_TRY(cudaStreamSynchronize(ctx->stream), "tracker sync");
    pct::preproc_tracker_loaded(ctx, n, integer_angles);
    return PCT_OK;
}

extern "C" pct_status pct_recon_volume_intersections(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    const pct::PreGeom g = pct::make_pregeom(ctx->cfg);
    pct::TrackerPtrs T;
    for (int k = 0; k < pct::kNumTracker; k++) T.a[k] = p->tracker[k];
    if (p->n_raw > 0)
        pct::intersections_kernel<<<pct::grid_for(p->n_raw, 256), 256, 0, ctx->stream>>>(
            g, p->n_raw, T, p->gantry_angle, p->integer_angles, geom_ptrs(p->raw_geom), p->missed);
    PRE_TRY(cudaGetLastError(), "intersections kernel");
    ctx->launches += 1;
    return PCT_OK;
}

extern "C" pct_status pct_binning(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    pct_status st = ensure_fixed(ctx, p);
    if (st != PCT_OK) return st;
    const long long n = p->n_raw, nb = ctx->cfg.NUM_BINS;
    cudaStream_t s = ctx->stream;
    PRE_TRY(cudaMemsetAsync(p->bin_counts, 0, sizeof(int) * nb, s), "bins clear");
    PRE_TRY(cudaMemsetAsync(p->mean_WEPL, 0, sizeof(float) * nb, s), "bins clear");
    PRE_TRY(cudaMemsetAsync(p->mean_rel_ut_angle, 0, sizeof(float) * nb, s), "bins clear");
    PRE_TRY(cudaMemsetAsync(p->mean_rel_uv_angle, 0, sizeof(float) * nb, s), "bins clear");
    PRE_TRY(cudaMemsetAsync(p->sinogram, 0, sizeof(float) * nb, s), "bins clear");
    const pct::PreGeom g = pct::make_pregeom(ctx->cfg);
    if (n > 0)
        pct::binning_kernel<<<pct::grid_for(n, 256), 256, 0, s>>>(g, n, geom_ptrs(p->raw_geom), p->raw_wepl, p->missed,
                                                                   p->raw_bin_num, p->bin_counts, p->mean_WEPL,
                                                                   p->mean_rel_ut_angle, p->mean_rel_uv_angle);
    PRE_TRY(cudaGetLastError(), "binning kernel");
    ctx->launches += 1;
    // the reference keeps histories that hit the volume with bin_num >= 0 (always, since bin_num
    // defaults to 0) in the history vectors, in order (B.cu:5429-5450)
    if (n > p->cap_vec) {
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < pct::kNumGeom && e == cudaSuccess; k++) e = alloc(p->vec_geom[k], n);
        if (e == cudaSuccess) e = alloc(p->vec_wepl, n);
        if (e == cudaSuccess) e = alloc(p->vec_bin_num, n);
        if (e == cudaSuccess) e = alloc(p->vec_first_voxel, n);
        if (e != cudaSuccess) {
            cudaGetLastError();
            p->cap_vec = 0;
            return fail(ctx, PCT_ERR_NOMEM, "history vectors", e);
        }
        p->cap_vec = n;
    }
    st = ensure_scratch(ctx, p, n);
    if (st != PCT_OK) return st;
    for (int k = 0; k < pct::kNumGeom; k++)
        PRE_TRY(cudaMemcpyAsync(p->vec_geom[k], p->raw_geom[k], sizeof(float) * n, cudaMemcpyDeviceToDevice, s), "copy");
    PRE_TRY(cudaMemcpyAsync(p->vec_wepl, p->raw_wepl, sizeof(float) * n, cudaMemcpyDeviceToDevice, s), "copy");
    PRE_TRY(cudaMemcpyAsync(p->vec_bin_num, p->raw_bin_num, sizeof(int) * n, cudaMemcpyDeviceToDevice, s), "copy");
    if (n > 0) pct::u8_to_int_kernel<<<pct::grid_for(n, 256), 256, 0, s>>>(n, p->missed, 1, p->flags);
    PRE_TRY(cudaGetLastError(), "keep flags");
    long long kept = 0;
    return compact_vectors(ctx, p, n, &kept);
}

extern "C" pct_status pct_hull_detection(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    pct_status st = ensure_fixed(ctx, p);
    if (st != PCT_OK) return st;
    const pct::PreGeom g = pct::make_pregeom(ctx->cfg);
    const long long nv = ctx->cfg.NUM_VOXELS, n = p->n_raw;
    cudaStream_t s = ctx->stream;
    // hull_initializations / initialize_hull_GPU (B.cu:6636-6669)
    pct::init_hull_kernel<uint8_t><<<pct::grid_for(nv, 256), 256, 0, s>>>(g, p->SC_hull);
    pct::init_hull_kernel<int><<<pct::grid_for(nv, 256), 256, 0, s>>>(g, p->MSC_counts);
    pct::init_hull_kernel<int><<<pct::grid_for(nv, 256), 256, 0, s>>>(g, p->SM_counts);
    ctx->launches += 3;
    if (n > 0) {
        const pct::GeomPtrs G = geom_ptrs(p->raw_geom);
        if (ctx->cfg.SC_ON || ctx->cfg.MSC_ON || ctx->cfg.SM_ON) {
            st = ensure_scratch(ctx, p, n);
            if (st != PCT_OK) return st;
            const pct::HullImages im{ctx->cfg.SC_ON ? p->SC_hull : nullptr, ctx->cfg.MSC_ON ? p->MSC_counts : nullptr,
                                     ctx->cfg.SM_ON ? p->SM_counts : nullptr};
            const pct::HullPlan plan = pct::hull_plan(g);
            if (plan.window > 0 && n >= pct::kHullWindowMin) {
                const int keys = 8 * plan.first * plan.distances, blocks = pct::sm_count();
                const size_t shared = 4 * ((size_t)plan.window * g.columns * g.rows / 2 + 1);
                int *key = p->tmp_bin_num, *order = reinterpret_cast<int*>(p->offsets);
                pct::hull_key_kernel<<<pct::grid_for(n, 256), 256, 0, s>>>(g, plan, n, G, p->raw_wepl, p->missed, im, key);
                PRE_TRY(pct::bucket_sort_by_key(key, 0, n, keys, p->walk_hist, order, s), "walk order");
                PRE_TRY(cudaFuncSetAttribute(pct::hull_window_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, pct::kHullWindow + 4),
                        "hull window");
                pct::hull_ranges_kernel<<<1, 1024, 0, s>>>(g, plan, p->walk_hist, blocks, p->hull_starts);
                pct::hull_window_kernel<<<blocks, pct::kHullThreads, shared, s>>>(g, plan, order, key, p->walk_hist + keys,
                                                                                  p->hull_starts, G, im, ctx->d_counters);
                ctx->launches += 6;
            } else {
                int* order = walk_order(ctx, p, n, p->raw_geom, 1);
                if (!order) return fail(ctx, PCT_ERR_CUDA, "walk order", cudaGetLastError());
                const auto kernel = g.fast_walks ? pct::hull_walks_kernel<pct::kMixedWalk> : pct::hull_walks_kernel<pct::kReferenceWalk>;
                kernel<<<pct::grid_for(n, 128), 128, 0, s>>>(g, n, order, G, p->raw_wepl, p->missed, im, ctx->d_counters);
                ctx->launches += 1;
            }
        }
    }
    PRE_TRY(cudaGetLastError(), "hull walk kernels");
    return PCT_OK;
}

extern "C" pct_status pct_calculate_means(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre || !ctx->pre->bin_counts) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    const int nb = ctx->cfg.NUM_BINS;
    pct::means_kernel<<<pct::grid_for(nb, 256), 256, 0, ctx->stream>>>(nb, p->bin_counts, p->mean_WEPL, p->mean_rel_ut_angle,
                                                                     p->mean_rel_uv_angle);
    PRE_TRY(cudaGetLastError(), "means kernel");
    ctx->launches += 1;
    return PCT_OK;
}

extern "C" pct_status pct_sum_squared_deviations(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre || !ctx->pre->bin_counts) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    const long long nb = ctx->cfg.NUM_BINS, n = p->n_vec;
    cudaStream_t s = ctx->stream;
    PRE_TRY(cudaMemsetAsync(p->stddev_WEPL, 0, sizeof(float) * nb, s), "clear");
    PRE_TRY(cudaMemsetAsync(p->stddev_rel_ut_angle, 0, sizeof(float) * nb, s), "clear");
    PRE_TRY(cudaMemsetAsync(p->stddev_rel_uv_angle, 0, sizeof(float) * nb, s), "clear");
    if (n > 0)
        pct::sum_sq_dev_kernel<<<pct::grid_for(n, 256), 256, 0, s>>>(n, p->vec_bin_num, p->vec_wepl, geom_ptrs(p->vec_geom),
                                                                     p->mean_WEPL, p->mean_rel_ut_angle, p->mean_rel_uv_angle,
                                                                     p->stddev_WEPL, p->stddev_rel_ut_angle, p->stddev_rel_uv_angle);
    PRE_TRY(cudaGetLastError(), "sum of squared deviations kernel");
    ctx->launches += 1;
    return PCT_OK;
}

extern "C" pct_status pct_calculate_standard_deviations(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre || !ctx->pre->bin_counts) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    const int nb = ctx->cfg.NUM_BINS;
    pct::stddev_kernel<<<pct::grid_for(nb, 256), 256, 0, ctx->stream>>>(nb, ctx->cfg.SAMPLE_STD_DEV ? 1 : 0, p->bin_counts,
                                                                      p->stddev_WEPL, p->stddev_rel_ut_angle,
                                                                      p->stddev_rel_uv_angle);
    PRE_TRY(cudaGetLastError(), "standard deviations kernel");
    ctx->launches += 1;
    return PCT_OK;
}

extern "C" pct_status pct_statistical_cuts(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre || !ctx->pre->bin_counts) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    const long long n = p->n_vec;
    cudaStream_t s = ctx->stream;
    PRE_TRY(cudaMemsetAsync(p->sinogram, 0, sizeof(float) * ctx->cfg.NUM_BINS, s), "sinogram clear");
    const pct::PreGeom g = pct::make_pregeom(ctx->cfg);
    if (n > 0)
        pct::cuts_kernel<<<pct::grid_for(n, 256), 256, 0, s>>>(g, n, p->vec_bin_num, p->vec_wepl, geom_ptrs(p->vec_geom),
                                                               p->mean_WEPL, p->mean_rel_ut_angle, p->mean_rel_uv_angle,
                                                               p->stddev_WEPL, p->stddev_rel_ut_angle, p->stddev_rel_uv_angle,
                                                               p->bin_counts, p->sinogram, p->flags);
    PRE_TRY(cudaGetLastError(), "cuts kernel");
    ctx->launches += 1;
    long long kept = 0;
    return compact_vectors(ctx, p, n, &kept);
}

extern "C" pct_status pct_construct_sinogram(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre || !ctx->pre->bin_counts) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    const int nb = ctx->cfg.NUM_BINS;
    pct::sinogram_kernel<<<pct::grid_for(nb, 256), 256, 0, ctx->stream>>>(nb, p->bin_counts, p->sinogram);
    PRE_TRY(cudaGetLastError(), "sinogram kernel");
    ctx->launches += 1;
    return PCT_OK;
}

extern "C" pct_status pct_FBP(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre || !ctx->pre->bin_counts) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    const pct::PreGeom g = pct::make_pregeom(ctx->cfg);
    const long long nv = ctx->cfg.NUM_VOXELS;
    cudaStream_t s = ctx->stream;
    const pct::FbpTables tab{p->fbp_tables, p->fbp_tables + g.t_bins, p->fbp_tables + g.t_bins + (long long)g.t_bins * g.v_bins};
    const long long most = (long long)g.t_bins * g.v_bins > g.angular_bins ? (long long)g.t_bins * g.v_bins : g.angular_bins;
    pct::fbp_tables_kernel<<<pct::grid_for(most, 256), 256, 0, s>>>(g, tab);
    const long long strips = (long long)pct::grid_for(g.t_bins, 128) * pct::grid_for(g.angular_bins, pct::kFilterStrips) * g.v_bins;
    pct::filter_kernel<<<(unsigned)strips, 128, 0, s>>>(g, tab, p->sinogram, p->sinogram_filtered);
    const long long columns = (long long)pct::grid_for((long long)g.columns * g.rows, 128) * pct::grid_for(g.slices, pct::kBackSlices);
    pct::backprojection_kernel<<<(unsigned)columns, 128, 0, s>>>(g, tab.trig, p->sinogram_filtered, p->FBP_image);
    ctx->launches += 3;
    const int r = ctx->cfg.FBP_MED_FILTER_RADIUS;
    if (ctx->cfg.MEDIAN_FILTER_FBP && r > 0) {
        if (r > 7) return fail(ctx, PCT_ERR_ARG, "FBP_MED_FILTER_RADIUS above 7 is not supported");
        const auto median = r == 1 ? pct::median_kernel<1> : r == 2 ? pct::median_kernel<2> : r == 3 ? pct::median_kernel<3> : pct::median_kernel<0>;
        median<<<pct::grid_for(nv, 128), 128, 0, s>>>(g, r, p->FBP_image, p->FBP_median);
        ctx->launches += 1;
    } else {
        PRE_TRY(cudaMemcpyAsync(p->FBP_median, p->FBP_image, sizeof(float) * nv, cudaMemcpyDeviceToDevice, s), "copy");
    }
    // FBP_image_2_hull thresholds the unfiltered FBP image (B.cu:6163-6164, 6592)
    if (ctx->cfg.ENDPOINTS_HULL == PCT_FBP_HULL) {
        pct::fbp_hull_kernel<<<pct::grid_for(nv, 256), 256, 0, s>>>(g, p->FBP_image, p->FBP_hull);
        ctx->launches += 1;
    }
    PRE_TRY(cudaGetLastError(), "FBP kernels");
    return PCT_OK;
}

extern "C" pct_status pct_hull_detection_finish(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre || !ctx->pre->bin_counts) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    const pct::PreGeom g = pct::make_pregeom(ctx->cfg);
    const long long nv = ctx->cfg.NUM_VOXELS;
    cudaStream_t s = ctx->stream;
    if (ctx->cfg.MSC_ON) {  // MSC_edge_detection (B.cu:6902), out of place
        pct::msc_edge_kernel<<<pct::grid_for(nv, 256), 256, 0, s>>>(g, p->MSC_counts, p->edge_tmp);
        PRE_TRY(cudaMemcpyAsync(p->MSC_counts, p->edge_tmp, sizeof(int) * nv, cudaMemcpyDeviceToDevice, s), "copy");
        ctx->launches += 1;
    }
    if (ctx->cfg.SM_ON) {  // SM_edge_detection (B.cu:7100)
        pct::carve_differences_kernel<<<pct::grid_for(nv, 256), 256, 0, s>>>(g, p->SM_counts, p->SM_differences);
        pct::sm_threshold_kernel<<<ctx->cfg.SLICES, 256, 0, s>>>(g, p->SM_differences, p->SM_counts, p->SM_thresholds);
        pct::sm_edge_kernel<<<pct::grid_for(nv, 256), 256, 0, s>>>(g, p->SM_counts, p->SM_thresholds);
        ctx->launches += 3;
    }
    PRE_TRY(cudaGetLastError(), "hull finish kernels");
    return PCT_OK;
}

extern "C" pct_status pct_hull_selection(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre || !ctx->pre->bin_counts) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    const long long nv = ctx->cfg.NUM_VOXELS;
    cudaStream_t s = ctx->stream;
    switch (ctx->cfg.ENDPOINTS_HULL) {  // hull_selection (B.cu:7351-7393)
        case PCT_SC_HULL:
            PRE_TRY(cudaMemcpyAsync(p->hull, p->SC_hull, nv, cudaMemcpyDeviceToDevice, s), "hull copy");
            break;
        case PCT_MSC_HULL:
            pct::counts_to_hull_kernel<<<pct::grid_for(nv, 256), 256, 0, s>>>(nv, p->MSC_counts, p->hull);
            ctx->launches += 1;
            break;
        case PCT_SM_HULL:
            pct::counts_to_hull_kernel<<<pct::grid_for(nv, 256), 256, 0, s>>>(nv, p->SM_counts, p->hull);
            ctx->launches += 1;
            break;
        default:
            PRE_TRY(cudaMemcpyAsync(p->hull, p->FBP_hull, nv, cudaMemcpyDeviceToDevice, s), "hull copy");
    }
    PRE_TRY(cudaGetLastError(), "hull selection");
    p->hull_ready = true;
    return PCT_OK;
}

extern "C" pct_status pct_define_initial_iterate(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre || !ctx->pre->hull_ready) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    const long long nv = ctx->cfg.NUM_VOXELS;
    pct::hybrid_kernel<<<pct::grid_for(nv, 256), 256, 0, ctx->stream>>>(nv, p->hull, p->FBP_median, ctx->d_x);
    PRE_TRY(cudaGetLastError(), "initial iterate");
    ctx->launches += 1;
    return PCT_OK;
}

extern "C" pct_status pct_reconstruction_cuts(pct_ctx* ctx)
{
    if (!ctx || !ctx->pre || !ctx->pre->hull_ready) return PCT_ERR_STATE;
    Preproc* p = ctx->pre;
    cudaSetDevice(ctx->device);
    const long long n = p->n_vec;
    cudaStream_t s = ctx->stream;
    const pct::PreGeom g = pct::make_pregeom(ctx->cfg);
    if (n > 0) {
        int* order = walk_order(ctx, p, n, p->vec_geom, pct::kWalkDir);
        if (!order) return fail(ctx, PCT_ERR_CUDA, "walk order", cudaGetLastError());
        const long long words = (ctx->cfg.NUM_VOXELS + 31LL) / 32;
        pct::hull_bits_kernel<<<pct::grid_for(words * 32, 256), 256, 0, s>>>(words, ctx->cfg.NUM_VOXELS, p->hull, p->hull_bits);
        ctx->launches += 1;
        // grids lower than a fifth of their width: most lines leave through the top or the bottom.  500k histories,
        // timed / mixed / reference steps, us: 200x200 voxels of 1 slice 424 / 777 / 424, 2 353 / 608 / 415, 4 520 / 648 /
        // 637, 8 350 / 392 / 508; 128x128x16 188 / 182 / 278, 48x48x32 88 / 81 / 106, 200x200x32 41 / 37 / 29
        const auto kernel = !g.fast_walks     ? pct::endpoints_kernel<pct::kReferenceWalk>
                            : 10 * g.H <= 4 * g.R ? pct::endpoints_kernel<pct::kTimedWalk>
                                                  : pct::endpoints_kernel<pct::kMixedWalk>;
        kernel<<<pct::grid_for(n, 128), 128, 0, s>>>(g, n, order, p->hull_bits, geom_ptrs(p->vec_geom), p->vec_first_voxel,
                                                     p->flags);
    }
    PRE_TRY(cudaGetLastError(), "endpoints kernel");
    ctx->launches += 1;
    // keep histories whose entry and exit walks hit the hull, in order (B.cu:8286-8294); the first
    // MLP voxel is compacted by a second pass through the integer slot
    PRE_TRY(pct::exclusive_scan_i32_to_i64(p->flags, n, p->offsets, p->scan_tmp, s), "scan");
    long long total = 0;
    PRE_TRY(cudaMemcpyAsync(&total, p->offsets + n, sizeof(long long), cudaMemcpyDeviceToHost, s), "count");
    pct::CompactArrays c{};
    int nf = 0;
    for (int k = 0; k < pct::kNumGeom; k++) {
        c.in_f[nf] = p->vec_geom[k];
        c.out_f[nf++] = p->tmp_geom[k];
    }
    c.in_f[nf] = p->vec_wepl;
    c.out_f[nf++] = p->tmp_wepl;
    c.nf = nf;
    c.in_i[0] = reinterpret_cast<const int*>(p->vec_first_voxel);
    c.out_i[0] = p->tmp_bin_num;
    c.ni = 1;
    if (n > 0) pct::compact_kernel<<<pct::grid_for(n, 256), 256, 0, s>>>(n, p->flags, p->offsets, c);
    PRE_TRY(cudaGetLastError(), "compaction");
    PRE_TRY(cudaStreamSynchronize(s), "sync");
    ctx->launches += 4;
    for (int k = 0; k < pct::kNumGeom; k++) std::swap(p->vec_geom[k], p->tmp_geom[k]);
    std::swap(p->vec_wepl, p->tmp_wepl);
    PRE_TRY(cudaMemcpyAsync(p->vec_first_voxel, p->tmp_bin_num, sizeof(uint32_t) * total, cudaMemcpyDeviceToDevice, s), "copy");
    p->n_vec = total;
    // hand the reconstruction histories to the DROP stage (device to device)
    pct_histories h;
    h.x_entry = p->vec_geom[pct::kXE];
    h.y_entry = p->vec_geom[pct::kYE];
    h.z_entry = p->vec_geom[pct::kZE];
    h.x_exit = p->vec_geom[pct::kXO];
    h.y_exit = p->vec_geom[pct::kYO];
    h.z_exit = p->vec_geom[pct::kZO];
    h.xy_entry_angle = p->vec_geom[pct::kXYE];
    h.xz_entry_angle = p->vec_geom[pct::kXZE];
    h.xy_exit_angle = p->vec_geom[pct::kXYO];
    h.xz_exit_angle = p->vec_geom[pct::kXZO];
    h.WEPL = p->vec_wepl;
    h.first_MLP_voxel = p->vec_first_voxel;
    pct_status st = pct::load_histories(ctx, &h, total, PCT_DEVICE);
    // apply_history_sequence (B.cu:8691): the reconstruction order of the histories
    if (st == PCT_OK && ctx->cfg.RECON_HISTORY_ORDERING == PCT_PRIME_PERMUTATION)
        st = pct_apply_history_sequence(ctx, ctx->cfg.PRIME_OFFSET);
    return st;
}

extern "C" pct_status pct_set_history_vectors(pct_ctx* ctx, const pct_histories* h, int64_t n, pct_memory where)
{
    if (!ctx || !h || n < 0 || n > 0x7fffffffLL) return PCT_ERR_ARG;
    cudaSetDevice(ctx->device);
    Preproc* p = pre_of(ctx);
    pct_status st = ensure_fixed(ctx, p);
    if (st != PCT_OK) return st;
    if (n > p->cap_vec) {
        cudaError_t e = cudaSuccess;
        for (int k = 0; k < pct::kNumGeom && e == cudaSuccess; k++) e = alloc(p->vec_geom[k], n);
        if (e == cudaSuccess) e = alloc(p->vec_wepl, n);
        if (e == cudaSuccess) e = alloc(p->vec_bin_num, n);
        if (e == cudaSuccess) e = alloc(p->vec_first_voxel, n);
        if (e != cudaSuccess) {
            cudaGetLastError();
            p->cap_vec = 0;
            return fail(ctx, PCT_ERR_NOMEM, "history vectors", e);
        }
        p->cap_vec = n;
    }
    st = ensure_scratch(ctx, p, n);
    if (st != PCT_OK) return st;
    const float* src[pct::kNumGeom] = {h->x_entry, h->y_entry, h->z_entry, h->x_exit, h->y_exit, h->z_exit,
                                       h->xy_entry_angle, h->xz_entry_angle, h->xy_exit_angle, h->xz_exit_angle};
    const cudaMemcpyKind kind = where == PCT_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
    for (int k = 0; k < pct::kNumGeom && n > 0; k++) {
        if (!src[k]) return PCT_ERR_ARG;
        PRE_TRY(cudaMemcpyAsync(p->vec_geom[k], src[k], sizeof(float) * n, kind, ctx->stream), "vector copy");
    }
    if (n > 0) {
        if (!h->WEPL) return PCT_ERR_ARG;
        PRE_TRY(cudaMemcpyAsync(p->vec_wepl, h->WEPL, sizeof(float) * n, kind, ctx->stream), "vector copy");
        PRE_TRY(cudaMemsetAsync(p->vec_bin_num, 0, sizeof(int) * n, ctx->stream), "vector clear");
    }
    PRE_TRY(cudaStreamSynchronize(ctx->stream), "vector sync");
    p->n_vec = n;
    return PCT_OK;
}

namespace {

// The stages of preprocessing() + the first half of image_reconstruction() (B.cu:7394,
// 10650-10660) after the tracker data is loaded.
pct_status preprocessing_stages(pct_ctx* ctx)
{
    pct_status st = pct_recon_volume_intersections(ctx);
    if (st == PCT_OK) st = pct_binning(ctx);
    if (st == PCT_OK) st = pct_hull_detection(ctx);
    if (st == PCT_OK) st = pct_hull_detection_finish(ctx);
    if (st == PCT_OK) st = pct_calculate_means(ctx);
    if (st == PCT_OK) st = pct_sum_squared_deviations(ctx);
    if (st == PCT_OK) st = pct_calculate_standard_deviations(ctx);
    if (st == PCT_OK) st = pct_statistical_cuts(ctx);
    if (st == PCT_OK) st = pct_construct_sinogram(ctx);
    if (st == PCT_OK) st = pct_FBP(ctx);
    if (st == PCT_OK) st = pct_hull_selection(ctx);
    if (st == PCT_OK) st = pct_define_initial_iterate(ctx);
    if (st == PCT_OK) st = pct_reconstruction_cuts(ctx);
    return st;
}

}  // namespace

extern "C" pct_status pct_preprocessing(pct_ctx* ctx, const pct_tracker_data* t, int64_t n, pct_memory where,
                                        int integer_angles)
{
    pct_status st = pct_load_tracker_data(ctx, t, n, where, integer_angles);
    return st == PCT_OK ? preprocessing_stages(ctx) : st;
}

extern "C" pct_status pct_preprocessing_from_files(pct_ctx* ctx, const char* directory)
{
    int64_t n = 0;
    pct_status st = pct_load_projection_data(ctx, directory, &n);
    return st == PCT_OK ? preprocessing_stages(ctx) : st;
}

// ---- named arrays ----
namespace {

struct NamedArray {
    void* ptr;
    size_t elem;
    long long count;
};

bool lookup(pct_ctx* ctx, const char* name, NamedArray& out)
{
    Preproc* p = ctx->pre;
    const long long nb = ctx->cfg.NUM_BINS, nv = ctx->cfg.NUM_VOXELS;
    std::string s(name);
    if (s == "x") {
        out = {ctx->d_x, 4, nv};
        return true;
    }
    // the reconstruction histories, in reconstruction order (the *_vector_reconstruction
    // vectors of apply_history_sequence, B.cu:8691)
    {
        pct::HistorySoA& h = ctx->hist;
        const struct {
            const char* n;
            void* ptr;
        } rec[] = {{"x_entry_reconstruction", h.x_entry}, {"y_entry_reconstruction", h.y_entry},
                   {"z_entry_reconstruction", h.z_entry}, {"x_exit_reconstruction", h.x_exit},
                   {"y_exit_reconstruction", h.y_exit}, {"z_exit_reconstruction", h.z_exit},
                   {"xy_entry_angle_reconstruction", h.xy_entry_angle},
                   {"xz_entry_angle_reconstruction", h.xz_entry_angle},
                   {"xy_exit_angle_reconstruction", h.xy_exit_angle},
                   {"xz_exit_angle_reconstruction", h.xz_exit_angle}, {"WEPL_reconstruction", h.WEPL},
                   {"first_MLP_voxel_reconstruction", h.first_MLP_voxel}};
        for (const auto& e : rec)
            if (s == e.n) {
                out = {e.ptr, 4, ctx->n_hist};
                return e.ptr != nullptr && ctx->n_hist > 0;
            }
    }
    if (!p) return false;
    for (int k = 0; k < pct::kNumTracker; k++)
        if (s == pct::kTrackerNames[k]) {
            out = {p->tracker[k], 4, p->n_raw};
            return true;
        }
    for (int k = 0; k < pct::kNumGeom; k++) {
        if (s == pct::kGeomNames[k]) {
            out = {p->raw_geom[k], 4, p->n_raw};
            return true;
        }
        if (s == std::string(pct::kGeomNames[k]) + "_vector") {
            out = {p->vec_geom[k], 4, p->n_vec};
            return true;
        }
    }
    const struct {
        const char* n;
        void* ptr;
        size_t elem;
        long long count;
    } table[] = {
        {"gantry_angle", p->gantry_angle, 4, p->n_raw},
        {"WEPL", p->raw_wepl, 4, p->n_raw},
        {"missed_recon_volume", p->missed, 1, p->n_raw},
        {"bin_num", p->raw_bin_num, 4, p->n_raw},
        {"WEPL_vector", p->vec_wepl, 4, p->n_vec},
        {"bin_num_vector", p->vec_bin_num, 4, p->n_vec},
        {"first_MLP_voxel_vector", p->vec_first_voxel, 4, p->n_vec},
        {"bin_counts", p->bin_counts, 4, nb},
        {"mean_WEPL", p->mean_WEPL, 4, nb},
        {"mean_rel_ut_angle", p->mean_rel_ut_angle, 4, nb},
        {"mean_rel_uv_angle", p->mean_rel_uv_angle, 4, nb},
        {"stddev_WEPL", p->stddev_WEPL, 4, nb},
        {"stddev_rel_ut_angle", p->stddev_rel_ut_angle, 4, nb},
        {"stddev_rel_uv_angle", p->stddev_rel_uv_angle, 4, nb},
        {"sinogram", p->sinogram, 4, nb},
        {"sinogram_filtered", p->sinogram_filtered, 4, nb},
        {"FBP_image", p->FBP_image, 4, nv},
        {"FBP_median_filtered", p->FBP_median, 4, nv},
        {"FBP_hull", p->FBP_hull, 1, nv},
        {"SC_hull", p->SC_hull, 1, nv},
        {"MSC_counts", p->MSC_counts, 4, nv},
        {"SM_counts", p->SM_counts, 4, nv},
        {"hull", p->hull, 1, nv},
    };
    for (const auto& e : table)
        if (s == e.n) {
            out = {e.ptr, e.elem, e.count};
            return e.ptr != nullptr;
        }
    return false;
}

}  // namespace

extern "C" int64_t pct_array_length(pct_ctx* ctx, const char* name)
{
    NamedArray a;
    if (!ctx || !name || !lookup(ctx, name, a)) return -1;
    return a.count;
}

extern "C" pct_status pct_get_array(pct_ctx* ctx, const char* name, void* dst, int64_t capacity_bytes, pct_memory where)
{
    NamedArray a;
    if (!ctx || !name || !dst) return PCT_ERR_ARG;
    if (!lookup(ctx, name, a)) return fail(ctx, PCT_ERR_ARG, std::string("unknown or unset array ") + name);
    const size_t bytes = a.elem * (size_t)a.count;
    if ((int64_t)bytes > capacity_bytes) return fail(ctx, PCT_ERR_ARG, std::string("buffer too small for ") + name);
    cudaSetDevice(ctx->device);
    if (bytes)
        PRE_TRY(cudaMemcpyAsync(dst, a.ptr, bytes, where == PCT_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice,
                                ctx->stream), "pct_get_array copy");
    PRE_TRY(cudaStreamSynchronize(ctx->stream), "pct_get_array sync");
    return PCT_OK;
}

extern "C" pct_status pct_set_array(pct_ctx* ctx, const char* name, const void* src, int64_t bytes, pct_memory where)
{
    NamedArray a;
    if (!ctx || !name || !src) return PCT_ERR_ARG;
    cudaSetDevice(ctx->device);
    if (ctx->pre) {
        pct_status st = ensure_fixed(ctx, ctx->pre);
        if (st != PCT_OK) return st;
    } else {
        pre_of(ctx);
        pct_status st = ensure_fixed(ctx, ctx->pre);
        if (st != PCT_OK) return st;
    }
    if (!lookup(ctx, name, a)) return fail(ctx, PCT_ERR_ARG, std::string("unknown or unset array ") + name);
    const std::string sn(name);
    if (sn.size() > 15 && sn.compare(sn.size() - 15, 15, "_reconstruction") == 0)
        return fail(ctx, PCT_ERR_ARG, sn + " is read-only: load histories with pct_set_reconstruction_histories");
    if ((size_t)bytes != a.elem * (size_t)a.count) return fail(ctx, PCT_ERR_ARG, std::string("size mismatch for ") + name);
    if (bytes)
        PRE_TRY(cudaMemcpyAsync(a.ptr, src, (size_t)bytes, where == PCT_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice,
                                ctx->stream), "pct_set_array copy");
    PRE_TRY(cudaStreamSynchronize(ctx->stream), "pct_set_array sync");
    if (std::string(name) == "hull") ctx->pre->hull_ready = true;
    return PCT_OK;
}

extern "C" pct_status pct_selftest_quotient(int64_t n, uint64_t seed, int64_t* mismatches)
{
    if (n < 0 || !mismatches) return PCT_ERR_ARG;
    unsigned long long *d = nullptr, h = 0;
    if (cudaMalloc(&d, sizeof(*d)) != cudaSuccess) return PCT_ERR_NOMEM;
    cudaError_t e = cudaMemset(d, 0, sizeof(*d));
    pct::quotient_check_kernel<<<148 * 4, 256>>>(n, seed, d);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess) return PCT_ERR_CUDA;
    *mismatches = (int64_t)h;
    return PCT_OK;
}
