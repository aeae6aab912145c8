// pct_mlp.cuh -- the most-likely-path (MLP) walk, exact mode.
//
// mlp_walk_exact() restates find_MLP_path_GPU_tabulated (B.cu:9104-9262) operation for
// operation in IEEE double: same table indices, same operand order, same float round trips
// (and the same CUDA powf/sinf/cosf calls) where the reference drops to float.  The translation
// unit that includes this header is compiled with -fmad=false so no multiply-add pair is fused.
// The CPU oracle squares with the correctly rounded float product instead of CUDA's powf, so the
// two voxel lists can differ where an MLP point falls within ~1e-7 cm of a voxel boundary; the
// parity tests count those ties.
//
// Two restructurings that do not change a single rounding:
//  * the Sigma_1 terms of step k depend only on k (u_1 = k*MLP_U_STEP), so they are read from a
//    per-step table built once on the device with the same expressions (build_step_table_kernel);
//  * the running depth (depth_2_go -= MLP_U_STEP) and position (u_shifted += MLP_U_STEP) are
//    carried exactly as the reference carries them.
#pragma once

#include "pct_common.cuh"
#include "pct_tables.h"

namespace pct {

// Maximum MLP voxel-list length handled per history: MLP_U_STEP >= 0.03125 cm (half of the
// reference's smallest 0.0625 cm voxel) over the 40 cm polynomial-table range gives
// <= 1281 entries (the reference's MAX_INTERSECTIONS is 1280, B.h:342).
constexpr int kPathCap = PCT_MLP_PATH_CAP;
// Path storage is written in chunks of 8 entries (one 32-byte sector); kPathCap is a multiple.
constexpr int kPathChunk = 8;
static_assert(kPathCap % kPathChunk == 0, "path cap must be a multiple of the write chunk");
static_assert(kSCurveEntries >= kPathCap, "the S-curve table covers every path index");

// Flags reported per history (same bits as the oracle).
enum WalkFlag : unsigned { kFlagVoxelOOB = 1u, kFlagPathOverflow = 2u, kFlagTableRange = 4u };

// Adds one history's walk flags to the context counters read by pct_get_counters.
__device__ __forceinline__ void count_flags(unsigned flags, unsigned long long* counters)
{
    if (flags & kFlagVoxelOOB) atomicAdd(counters + kCntVoxelOOB, 1ull);
    if (flags & kFlagPathOverflow) atomicAdd(counters + kCntPathOverflow, 1ull);
    if (flags & kFlagTableRange) atomicAdd(counters + kCntTableRange, 1ull);
}

struct WalkResult {
    int n;          // number_of_intersections (capped at kPathCap)
    unsigned flags;
    double chord;   // effective_chord_length
    double axk;     // a_i_dot_x_k_partially: sum of x over the path
    double aia;     // a_i_dot_a_i_partially: powf(chord, 2)
};

// powf(v, 2) on a double argument, as the reference writes it: v is rounded to float and CUDA's
// powf is called.  CUDA's powf(f, 2.0f) is not always the correctly rounded product f*f (the
// device self-test pct_selftest_powf_square counts about 6% of inputs one float ulp away), so the
// call is kept to reproduce the reference's values.
__device__ __forceinline__ double powf_square(double v)
{
    return (double)powf((float)v, 2.0f);
}

// calculate_voxel_GPU (B.cu:11091): int(|position - zero| / size); -1 when it does not fit an int.
__device__ __forceinline__ int voxel_index_1d(double zero, double pos, double size)
{
    const double q = fabs(pos - zero) / size;
    return (q < 2147483647.0) ? (int)q : -1;
}

// The same index without the division in the common case.  p = |pos - zero| * RN(1/size) is
// within 3.4e-16 relative of the exact quotient, and the reference's RN(quotient) is within
// 1.2e-16 of it; when p is farther than 1e-14 (relative) from every integer, no integer can lie
// between p and RN(quotient), so floor(p) == (int)RN(quotient).  Otherwise (about 2e-14 of calls,
// and when p = 0) the exact division decides.
__device__ __forceinline__ int voxel_index_1d_fast(double zero, double pos, double size, double inv_size)
{
    const double a = fabs(pos - zero);
    const double p = a * inv_size;
    if (p < 2147483000.0) {
        const double f = floor(p);
        const double guard = p * 1.0e-14;
        if (p - f > guard && (f + 1.0) - p > guard) return (int)f;
    }
    return voxel_index_1d(zero, pos, size);
}

// EffectiveChordLength_GPU (B.cu:8873-8894).  sinf/cosf receive float arguments; the sum of two
// float results is a float addition, as in the reference.  The reference is compiled with
// multiply-add contraction, which fuses a product into the addition that consumes it; where both
// operands of an addition are products it fuses the one with fewer uses.  The fused forms are
// written out here (this translation unit does not contract): eff_angle_t = fma(-k, PI/2, angle),
// the numerators and denominators fma(a, b, -c), and the 3-D numerator fma(-6, h, sf^2 sin 2v),
// whose other product sf^2 sin 2v is also used by the last term.  Comparing the possible forms
// with the reference's chords on the head grid (2000 histories, tests/golden/ref_mlp_head.npz)
// singles out the 3-D numerator's; the others do not change a chord there and follow the same rule.
__device__ __forceinline__ double effective_chord_length(const Geometry& g, double abs_angle_t, double abs_angle_v)
{
    const double PI = ref_pi();
    const int quadrants = (int)(abs_angle_t / (PI / 2));
    const double eff_angle_t = __fma_rn(-(double)quadrants, PI / 2, abs_angle_t);
    const double eff_angle_v = fabs(abs_angle_v);
    double step_fraction = g.mlp_u_step / g.voxel_width;
    const float s2t = sinf((float)(2 * eff_angle_t));
    const float ct_plus_st = __fadd_rn(cosf((float)eff_angle_t), sinf((float)eff_angle_t));
    const double sf2_s2t = __dmul_rn(__dmul_rn(step_fraction, step_fraction), (double)s2t);
    const double chord_length_2D =
        (1 / 3.0) * (__fma_rn(__dmul_rn(step_fraction, step_fraction), (double)s2t, -6.0) /
                         __fma_rn(step_fraction, (double)s2t, -(double)(2 * ct_plus_st)) +
                     sf2_s2t / (double)(2 * ct_plus_st));
    const double mean_pixel_width = g.voxel_width / ct_plus_st;
    const double height_fraction = g.voxel_thickness / mean_pixel_width;
    step_fraction = g.mlp_u_step / mean_pixel_width;
    const float s2v = sinf((float)(2 * eff_angle_v));
    const float cv = cosf((float)eff_angle_v);
    const float sv = sinf((float)eff_angle_v);
    const double inner2 = 2 * __fma_rn(height_fraction, (double)cv, (double)sv);
    const double sf2_s2v = __dmul_rn(__dmul_rn(step_fraction, step_fraction), (double)s2v);
    const double chord_length_3D =
        (1 / 3.0) * (__fma_rn(-6.0, height_fraction, sf2_s2v) / __fma_rn(step_fraction, (double)s2v, -inner2) +
                     sf2_s2v / inner2);
    return g.voxel_width * chord_length_2D * chord_length_3D;
}

// u_2 = |u_out - u_in| of a history in its entry-angle frame, exactly as the walk computes it.
__device__ __forceinline__ double mlp_u_extent(const Geometry& g, const Tables& tab, double x_in, double y_in,
                                               double x_out, double y_out, double xy_entry_angle)
{
    unsigned trig_index = (unsigned)((xy_entry_angle - g.trig_min) / g.trig_step + 0.5);
    double sin_term = __ldg(tab.sin_table + trig_index);
    double cos_term = __ldg(tab.cos_table + trig_index);
    double u_in = cos_term * x_in + sin_term * y_in;
    double u_out = cos_term * x_out + sin_term * y_out;
    if (u_in > u_out) {
        trig_index = (unsigned)((xy_entry_angle + ref_pi() - g.trig_min) / g.trig_step + 0.5);
        sin_term = __ldg(tab.sin_table + trig_index);
        cos_term = __ldg(tab.cos_table + trig_index);
        u_in = cos_term * x_in + sin_term * y_in;
        u_out = cos_term * x_out + sin_term * y_out;
    }
    return fabs(u_out - u_in);
}

// Per-history constants of the MLP loop (B.cu:9104-9158).
struct MlpHistory {
    double sin_term, cos_term;
    double t_in, t_out, z_in, z_out, T_2_1, V_2_1;
    double u_2, u_2_sq, two_u_2;
    double u_2_poly_3_12, u_2_poly_2_6, u_2_poly_1_2;
    double mag_tv;  // max(|t_in| + |t_out| + |T_2_1|, |z_in| + |z_out| + |V_2_1|): the guarded fast point's bound
};

// The same in shared memory, field f of this thread at byte address at + f * kStride, each loaded where it is
// used: the loads are volatile, so that they stay inside the loop trip and the constants are not held in
// registers across trips.
constexpr int kHistoryFields = 15;
static_assert(sizeof(MlpHistory) == kHistoryFields * sizeof(double), "MlpHistory is 15 doubles");
template <int kStride>
struct ParkedHistory {
    template <int F>
    struct Field {
        uint32_t at;
        __device__ __forceinline__ operator double() const
        {
            double v;
            asm volatile("ld.shared.f64 %0, [%1 + %2];" : "=d"(v) : "r"(at), "n"(F * kStride));
            return v;
        }
    };
    Field<0> sin_term;
    Field<1> cos_term;
    Field<2> t_in;
    Field<3> t_out;
    Field<4> z_in;
    Field<5> z_out;
    Field<6> T_2_1;
    Field<7> V_2_1;
    Field<8> u_2;
    Field<9> u_2_sq;
    Field<10> two_u_2;
    Field<11> u_2_poly_3_12;
    Field<12> u_2_poly_2_6;
    Field<13> u_2_poly_1_2;
    Field<14> mag_tv;
    Field<15> chord;  // the walk's, while it loops
    __device__ __forceinline__ explicit ParkedHistory(uint32_t a)
        : sin_term{a}, cos_term{a}, t_in{a}, t_out{a}, z_in{a}, z_out{a}, T_2_1{a}, V_2_1{a}, u_2{a}, u_2_sq{a}, two_u_2{a},
          u_2_poly_3_12{a}, u_2_poly_2_6{a}, u_2_poly_1_2{a}, mag_tv{a}, chord{a}
    {
    }
    __device__ __forceinline__ void park(const MlpHistory& h, double chord_length) const
    {
        const double* f = reinterpret_cast<const double*>(&h);
#pragma unroll
        for (int i = 0; i <= kHistoryFields; i++)
            asm volatile("st.shared.f64 [%0], %1;" ::"r"(chord.at + i * kStride), "d"(i < kHistoryFields ? f[i] : chord_length) : "memory");
    }
    __device__ __forceinline__ MlpHistory all() const
    {
        return MlpHistory{sin_term, cos_term, t_in, t_out, z_in, z_out, T_2_1, V_2_1, u_2, u_2_sq, two_u_2, u_2_poly_3_12,
                          u_2_poly_2_6, u_2_poly_1_2, mag_tv};
    }
};

// MLP point (t_1, v_1) of one loop iteration (B.cu:9180-9226): Sigma_2 from the tables, its
// inverse, the 2x2 solve for t and v.  Same operations, same order as the reference.
struct Sigma2 {
    double sigma_t2, sigma_t2_theta2, sigma_theta2, determinant;
};

// The Sigma_2 moments of one point and their determinant (B.cu:9180-9186), in the reference's
// operations and order.
template <class History>
__device__ __forceinline__ Sigma2 sigma2_moments(const History& h, const StepConst& st,
                                                 const double* __restrict__ scattering, unsigned sigma_2_index)
{
    Sigma2 m;
    m.sigma_t2 = h.u_2_poly_3_12 - h.u_2_sq * st.p12 + h.two_u_2 * st.p23 - st.p34;
    m.sigma_t2_theta2 = h.u_2_poly_2_6 - h.u_2 * st.p12 + st.p23;
    m.sigma_theta2 = h.u_2_poly_1_2 - st.p12;
    m.determinant = __ldg(scattering + sigma_2_index) * (m.sigma_t2 * m.sigma_theta2 - powf_square(m.sigma_t2_theta2));
    return m;
}

__device__ __forceinline__ void mlp_point_rest(const MlpHistory& h, const StepConst& st, const Sigma2& m,
                                               double depth_2_go, double& t_1, double& v_1)
{
    const double sigma_t2 = m.sigma_t2, sigma_t2_theta2 = m.sigma_t2_theta2, sigma_theta2 = m.sigma_theta2;
    const double determinant_Sigma_2 = m.determinant;
    const double Sigma_2I_0 = sigma_theta2 / determinant_Sigma_2;
    const double Sigma_2I_1 = sigma_t2_theta2 / determinant_Sigma_2;
    const double Sigma_2I_2 = sigma_t2 / determinant_Sigma_2;

    const double first_term_common_24_1 = Sigma_2I_0 * depth_2_go - Sigma_2I_1;
    const double first_term_0 = st.s1i0 + Sigma_2I_0;
    const double first_term_1 = first_term_common_24_1 - st.s1i1;
    const double first_term_2 = depth_2_go * Sigma_2I_0 - st.s1i1 - Sigma_2I_1;
    const double first_term_3 = st.s1i2 + Sigma_2I_2 + depth_2_go * (first_term_common_24_1 - Sigma_2I_1);
    const double determinant_first_term = first_term_0 * first_term_3 - first_term_1 * first_term_2;

    double second_term_common_3 = Sigma_2I_0 * h.t_out - Sigma_2I_1 * h.T_2_1;
    double second_term_0 = st.s1i0 * h.t_in + second_term_common_3;
    double second_term_1 =
        depth_2_go * second_term_common_3 + Sigma_2I_2 * h.T_2_1 - Sigma_2I_1 * h.t_out - st.s1i1 * h.t_in;
    t_1 = (first_term_3 * second_term_0 - first_term_1 * second_term_1) / determinant_first_term;

    second_term_common_3 = Sigma_2I_0 * h.z_out - Sigma_2I_1 * h.V_2_1;
    second_term_0 = st.s1i0 * h.z_in + second_term_common_3;
    second_term_1 =
        depth_2_go * second_term_common_3 + Sigma_2I_2 * h.V_2_1 - Sigma_2I_1 * h.z_out - st.s1i1 * h.z_in;
    v_1 = (first_term_3 * second_term_0 - first_term_1 * second_term_1) / determinant_first_term;
}

__device__ __forceinline__ void mlp_point(const MlpHistory& h, const StepConst& st, const double* __restrict__ scattering,
                                          double depth_2_go, unsigned sigma_2_index, double& t_1, double& v_1)
{
    mlp_point_rest(h, st, sigma2_moments(h, st, scattering, sigma_2_index), depth_2_go, t_1, v_1);
}

// ---- Guarded fast points (exact mode, EXACT_FAST_POINTS = 1) ----------------------------------
// Only the voxel of an MLP point enters the voxel list, so a point needs the reference's rounding
// only when it lies near a voxel face.  mlp_point_fast keeps the part of the point where the
// reference's cancellation lives -- the Sigma_2 moments and their determinant, computed by the
// caller with the reference's operations in its order -- and evaluates the rest (Sigma_2's
// inverse, M = Sigma_1^-1 + R_1^T Sigma_2^-1 R_1, its determinant, the two solves and the
// rotation) with refined reciprocals and fused multiply-adds: about half the FP64 instructions
// of five IEEE divisions and a shorter dependency chain.  Alongside it bounds the difference
// between its result and the reference's by first-order forward error analysis: every quantity q
// carries a magnitude M(q), the sum of the absolute values of the terms it is built from, and
// both evaluations' rounding errors are at most a few units in the last place times M(q); kBoundK
// (2^-40, about 8000 units) covers both with a wide margin.  For t = num / det the bound is
// K (M(num) + |t| M(det)) / |det|, valid while K M(det) is well below |det| (checked).  A point
// whose bound does not keep every coordinate clear of a voxel face, or whose M is not
// well-conditioned, returns false and is recomputed in the reference's order, so the voxel list
// is the reference's either way.
constexpr double kBoundK = 9.094947017729282e-13;  // 2^-40

// rcp.approx.ftz.f64 (a coarse hardware reciprocal of the high word) refined by two Newton steps:
// within a few units in the last place of 1/b for the normal values it sees here.
__device__ __forceinline__ double rcp_refined(double b)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    double e = __fma_rn(-b, r, 1.0);
    r = __fma_rn(r, e, r);
    e = __fma_rn(-b, r, 1.0);
    return __fma_rn(r, e, r);
}

// The three indices int(|pos - zero| / size) of (x, y, z) when every coordinate is provably more than
// err (cm) away from a voxel face, with the subtraction and scaling roundings of either evaluation
// included; false otherwise.  One tolerance serves all three axes: (K max_a + err) max(1/size) is at
// least each axis's own (K a + err) / size.  The distance to the nearest face, |p - rint(p)|, is
// exact (p and rint(p) are multiples of p's last place, and the difference is at most 1/2), and the
// index is the truncation int(p), as the reference writes it.  The conditions are combined without
// branches: every point of a warp is almost always proven.
__device__ __forceinline__ bool guarded_indices(const Geometry& g, double x, double y, double z, double err,
                                                int& vx, int& vy, int& vz)
{
    const double ax = fabs(__dsub_rn(x, g.x_zero)), ay = fabs(__dsub_rn(y, g.y_zero)), az = fabs(__dsub_rn(z, g.z_zero));
    const double amax = fmax(fmax(ax, ay), az);
    const double tol = __dmul_rn(__fma_rn(kBoundK, amax, err), g.inv_voxel_max);
    const double px = __dmul_rn(ax, g.inv_voxel_width), py = __dmul_rn(ay, g.inv_voxel_height),
                 pz = __dmul_rn(az, g.inv_voxel_thickness);
    const bool ok = (__dmul_rn(amax, g.inv_voxel_max) < 2147483000.0) & (fabs(__dsub_rn(px, rint(px))) > tol) &
                    (fabs(__dsub_rn(py, rint(py))) > tol) & (fabs(__dsub_rn(pz, rint(pz))) > tol);
    if (!ok) return false;
    vx = (int)px;
    vy = (int)py;
    vz = (int)pz;
    return true;
}

// The fast point and its voxel (see above); false when the bound cannot prove the voxel.
// h.mag_tv is |t_in| + |t_out| + |T_2_1| and the same for v, the larger of the two.
template <class History>
__device__ __forceinline__ bool mlp_point_fast(const Geometry& g, const History& h, const StepConst& st, double sigma_t2,
                                               double sigma_t2_theta2, double sigma_theta2, double det2, double d,
                                               double u_shifted, uint32_t& voxel)
{
    const double r2 = rcp_refined(det2);
    const double S0 = __dmul_rn(sigma_theta2, r2), S1 = __dmul_rn(sigma_t2_theta2, r2), S2 = __dmul_rn(sigma_t2, r2);
    const double c = __fma_rn(S0, d, -S1);
    const double m0 = __dadd_rn(st.s1i0, S0);
    const double m1 = __dsub_rn(c, st.s1i1);
    const double m3 = __fma_rn(d, __dsub_rn(c, S1), __dadd_rn(st.s1i2, S2));
    const double det = __fma_rn(m0, m3, -__dmul_rn(m1, m1));
    // magnitudes
    const double aS0 = fabs(S0), aS1 = fabs(S1), aS2 = fabs(S2);
    const double Mc = __fma_rn(aS0, d, aS1);
    const double Mm0 = __dadd_rn(fabs(st.s1i0), aS0);
    const double Mm1 = __dadd_rn(Mc, fabs(st.s1i1));
    const double Mm3 = __fma_rn(d, __dadd_rn(Mc, aS1), __dadd_rn(fabs(st.s1i2), aS2));
    const double Mdet = __fma_rn(Mm0, Mm3, __dmul_rn(Mm1, Mm1));
    const double adet = fabs(det);
    if (!(__dmul_rn(4.0 * kBoundK, Mdet) < adet)) return false;
    const double rdet = rcp_refined(det);
    // the right-hand sides and the solves for t and v
    double c3 = __fma_rn(S0, h.t_out, -__dmul_rn(S1, h.T_2_1));
    double r0 = __fma_rn(st.s1i0, h.t_in, c3);
    double r1 = __fma_rn(d, c3, __fma_rn(S2, h.T_2_1, -__fma_rn(S1, h.t_out, __dmul_rn(st.s1i1, h.t_in))));
    const double t_1 = __dmul_rn(__fma_rn(m3, r0, -__dmul_rn(m1, r1)), rdet);
    c3 = __fma_rn(S0, h.z_out, -__dmul_rn(S1, h.V_2_1));
    r0 = __fma_rn(st.s1i0, h.z_in, c3);
    r1 = __fma_rn(d, c3, __fma_rn(S2, h.V_2_1, -__fma_rn(S1, h.z_out, __dmul_rn(st.s1i1, h.z_in))));
    const double v_1 = __dmul_rn(__fma_rn(m3, r0, -__dmul_rn(m1, r1)), rdet);
    // one bound for both solves: each right-hand-side input is at most mag_tv in magnitude
    // M(r0) = mag (|s1i0| + |S0| + |S1|) = mag (M(m0) + |S1|) and
    // M(r1) = mag (d (|S0| + |S1|) + |S2| + |S1| + |s1i1|) = mag (M(m1) + d |S1| + |S2|), so
    // M(num) = M(m3) M(r0) + M(m1) M(r1) = mag (M(m3) (M(m0) + |S1|) + M(m1) (M(m1) + d |S1| + |S2|))
    const double mag_tv = h.mag_tv;
    const double Mnum = __dmul_rn(mag_tv, __fma_rn(Mm3, __dadd_rn(Mm0, aS1), __dmul_rn(Mm1, __dadd_rn(Mm1, __fma_rn(d, aS1, aS2)))));
    const double err = __dmul_rn(kBoundK, __dmul_rn(__fma_rn(fmax(fabs(t_1), fabs(v_1)), Mdet, Mnum), fabs(rdet)));
    // rotation back to x/y (B.cu:9229-9232) and the voxel indices (calculate_voxel_GPU B.cu:11091)
    const double x_1 = __fma_rn(h.cos_term, u_shifted, -__dmul_rn(h.sin_term, t_1));
    const double y_1 = __fma_rn(h.sin_term, u_shifted, __dmul_rn(h.cos_term, t_1));
    const double Mrot = __fma_rn(fabs(h.cos_term) + fabs(h.sin_term), fabs(u_shifted) + fabs(t_1), 0.0);
    const double err_xy = __fma_rn(kBoundK, Mrot, err);
    int vx, vy, vz;
    if (!guarded_indices(g, x_1, y_1, v_1, err_xy, vx, vy, vz)) return false;  // err_xy >= err
    long long v64 = (long long)vx + (long long)vy * g.columns + (long long)vz * g.columns * g.rows;
    if (v64 > 0x7fffffffLL) v64 = 0x7fffffffLL;
    voxel = (uint32_t)v64;
    return true;
}

// Voxel of an MLP point after rotating back to x/y (B.cu:9229-9235); 0x7fffffff when an index
// does not fit.
__device__ __forceinline__ uint32_t mlp_voxel(const Geometry& g, const MlpHistory& h, double u_shifted, double t_1,
                                              double v_1)
{
    const double x_1 = h.cos_term * u_shifted - h.sin_term * t_1;
    const double y_1 = h.sin_term * u_shifted + h.cos_term * t_1;
    const int vx = voxel_index_1d_fast(g.x_zero, x_1, g.voxel_width, g.inv_voxel_width);
    const int vy = voxel_index_1d_fast(g.y_zero, y_1, g.voxel_height, g.inv_voxel_height);
    const int vz = voxel_index_1d_fast(g.z_zero, v_1, g.voxel_thickness, g.inv_voxel_thickness);
    long long v64 = (long long)vx + (long long)vy * g.columns + (long long)vz * g.columns * g.rows;
    if (vx < 0 || vy < 0 || vz < 0 || v64 > 0x7fffffffLL) v64 = 0x7fffffffLL;
    return (uint32_t)v64;
}

// State of one history's walk after the setup of B.cu:9104-9178: the per-history constants, the
// running depth and position, the Sigma_2 table index, and the first path entry.
struct MlpStart {
    MlpHistory h;
    double depth_2_go, u_shifted, u_in;
    unsigned sigma_2_index;
    bool tables_ok;
};

// Per-history setup of find_MLP_path_GPU_tabulated (B.cu:9104-9178), shared by both walks.
__device__ __forceinline__ MlpStart mlp_start(const Geometry& g, const Tables& tab, double x_in_object,
                                              double y_in_object, double z_in_object, double x_out_object,
                                              double y_out_object, double z_out_object, double& xy_entry_angle,
                                              double& xy_exit_angle, double xz_entry_angle, double xz_exit_angle,
                                              unsigned& flags)
{
    const double PI = ref_pi();
    const double s = g.mlp_u_step;
    MlpStart m;
    MlpHistory& h = m.h;
    unsigned trig_index = (unsigned)((xy_entry_angle - g.trig_min) / g.trig_step + 0.5);
    double sin_term = __ldg(tab.sin_table + trig_index);
    double cos_term = __ldg(tab.cos_table + trig_index);
    double u_in_object = cos_term * x_in_object + sin_term * y_in_object;
    double u_out_object = cos_term * x_out_object + sin_term * y_out_object;
    if (u_in_object > u_out_object) {
        xy_entry_angle += PI;
        xy_exit_angle += PI;
        trig_index = (unsigned)((xy_entry_angle - g.trig_min) / g.trig_step + 0.5);
        sin_term = __ldg(tab.sin_table + trig_index);
        cos_term = __ldg(tab.cos_table + trig_index);
        u_in_object = cos_term * x_in_object + sin_term * y_in_object;
        u_out_object = cos_term * x_out_object + sin_term * y_out_object;
    }
    h.sin_term = sin_term;
    h.cos_term = cos_term;
    h.t_in = cos_term * y_in_object - sin_term * x_in_object;
    h.t_out = cos_term * y_out_object - sin_term * x_out_object;
    h.z_in = z_in_object;
    h.z_out = z_out_object;
    h.T_2_1 = xy_exit_angle - xy_entry_angle;
    h.V_2_1 = xz_exit_angle - xz_entry_angle;
    h.u_2 = fabs(u_out_object - u_in_object);
    m.depth_2_go = h.u_2 - s;
    m.u_shifted = u_in_object;
    m.u_in = u_in_object;

    m.tables_ok = (h.u_2 / kPolyTableStep + 0.5) < (double)g.poly_elements && m.depth_2_go >= 0;
    unsigned u_2_poly_index = 0;
    m.sigma_2_index = 0;
    if (m.tables_ok) {
        m.sigma_2_index = (unsigned)(m.depth_2_go / kCoeffTableStep + 0.5);
        u_2_poly_index = (unsigned)(h.u_2 / kPolyTableStep + 0.5);
    } else {
        flags |= kFlagTableRange;
    }
    h.u_2_poly_3_12 = __ldg(tab.poly_3_12 + u_2_poly_index);
    h.u_2_poly_2_6 = __ldg(tab.poly_2_6 + u_2_poly_index);
    h.u_2_poly_1_2 = __ldg(tab.poly_1_2 + u_2_poly_index);
    h.u_2_sq = powf_square(h.u_2);
    h.two_u_2 = 2 * h.u_2;
    h.mag_tv = fmax(fabs(h.t_in) + fabs(h.t_out) + fabs(h.T_2_1), fabs(h.z_in) + fabs(h.z_out) + fabs(h.V_2_1));
    return m;
}

// Appends voxels to the path unless they repeat the previous entry (B.cu:9244-9251) and sums x
// over the path when kSumX.
template <bool kSumX, class Emit>
struct PathWriter {
    const Geometry& g;
    const float* __restrict__ x;
    Emit& emit;
    WalkResult& r;
    uint32_t last;
    int n;
    __device__ __forceinline__ void first(uint32_t voxel)
    {
        emit(0, voxel);
        n = 1;
        last = voxel;
        r.axk = 0.0;
        if (voxel < (uint32_t)g.padded_voxels) {
            if (kSumX) r.axk = (double)__ldg(x + voxel);
        } else {
            r.flags |= kFlagVoxelOOB;
        }
    }
    __device__ __forceinline__ void visit(uint32_t voxel)
    {
        if (voxel != last) {
            if (n < kPathCap) emit(n, voxel);
            else r.flags |= kFlagPathOverflow;
            if (voxel < (uint32_t)g.padded_voxels) {
                if (kSumX) r.axk += (double)__ldg(x + voxel);
            } else {
                r.flags |= kFlagVoxelOOB;
            }
            last = voxel;
            n++;
        }
    }
};

// One history's MLP.  emit(j, voxel) is called for every path entry j in order.  With kSumX the
// walk also sums the padded image x over the path (reads beyond it are reported and count as 0);
// without it x is not touched (the voxel list does not depend on the image).  kTryFast: with
// EXACT_FAST_POINTS, points whose voxel is certain skip the reference's order of operations.  kPark > 0 keeps the
// history's constants and the chord in shared memory at `parked`, kPark bytes apart.
template <bool kSumX, bool kTryFast = true, int kPark = 0, class Emit>
__device__ __forceinline__ WalkResult mlp_walk_exact(const Geometry& g, const Tables& tab,
                                                     const StepConst* __restrict__ steps, int kmax,
                                                     const float* __restrict__ x, uint32_t first_MLP_voxel,
                                                     double x_in_object, double y_in_object, double z_in_object,
                                                     double x_out_object, double y_out_object, double z_out_object,
                                                     double xy_entry_angle, double xz_entry_angle,
                                                     double xy_exit_angle, double xz_exit_angle, Emit emit,
                                                     uint32_t parked = 0)
{
    const double s = g.mlp_u_step;
    WalkResult r;
    r.flags = 0;
    MlpStart m = mlp_start(g, tab, x_in_object, y_in_object, z_in_object, x_out_object, y_out_object, z_out_object,
                           xy_entry_angle, xy_exit_angle, xz_entry_angle, xz_exit_angle, r.flags);
    double depth_2_go = m.depth_2_go, u_shifted = m.u_shifted;
    unsigned sigma_2_index = m.sigma_2_index;

    PathWriter<kSumX, Emit> w{g, x, emit, r, 0u, 0};
    w.first(first_MLP_voxel);
    r.chord = effective_chord_length(g, (xy_entry_angle + xy_exit_angle) / 2.0, (xz_entry_angle + xz_exit_angle) / 2.0);
    r.aia = powf_square(r.chord);
    const ParkedHistory<kPark> ph(parked);
    if (kPark > 0) ph.park(m.h, r.chord);

    int k = 1;
    while (m.tables_ok && depth_2_go > s) {
        if (k > kmax) {  // cannot happen while the u_2 index is inside the tables
            r.flags |= kFlagTableRange;
            break;
        }
        const StepConst& st = steps[k];
        u_shifted += s;
        uint32_t voxel;
        auto point = [&](const auto& h) {
            const Sigma2 m2 = sigma2_moments(h, st, tab.scattering_table, sigma_2_index);
            if (kTryFast && g.exact_fast_points &&
                mlp_point_fast(g, h, st, m2.sigma_t2, m2.sigma_t2_theta2, m2.sigma_theta2, m2.determinant, depth_2_go,
                               u_shifted, voxel))
                return;
            MlpHistory all;
            if constexpr (kPark > 0) all = h.all();
            else all = h;
            double t_1, v_1;
            mlp_point_rest(all, st, m2, depth_2_go, t_1, v_1);
            voxel = mlp_voxel(g, all, u_shifted, t_1, v_1);
        };
        if constexpr (kPark > 0) point(ph);
        else point(m.h);
        w.visit(voxel);
        depth_2_go -= s;
        sigma_2_index -= g.sigma_index_step;
        k++;
    }
    r.n = w.n < kPathCap ? w.n : kPathCap;
    if (kPark > 0) r.chord = ph.chord;
    return r;
}

// ---- Tabulated points (exact mode, EXACT_FAST_POINTS = 1) --------------------------------------
// Written out, the MLP point is linear in the history: with M = Sigma_1^-1 + R_1^T Sigma_2^-1 R_1,
//     t = t_in + B (t_out - t_in) + C T_2_1        v = z_in + B (z_out - z_in) + C V_2_1
// (the weights of t_in and t_out add up to 1), and the weights B and C depend only on the step k and
// on u_2.  What else enters them through the reference's arithmetic is small and per history: the
// distance delta of u_2 from its polynomial-table grid point, the error epsilon of its squared u_2
// (powf of a float), and the rounding of powf in the determinant of Sigma_2.  delta and epsilon act
// through Sigma_2's first moment, as -2 poly_2_6(u_2) delta and -poly_1_2(u_1) epsilon, and
// poly_1_2(u_1) is nearly proportional to k.  So B and C are tabulated once per context
// (build_mlp_table_kernel): for every bucket of u_2 (MLP_U_STEP wide, at most 0.05 cm) and every step
// k, a quadratic in u_2 plus a linear term in sigma = delta + k kappa epsilon, as 8 floats, and per
// bucket an estimate of how far the tabulated weights can be from the ones the reference's operations
// give.  It adds
//   * twice the largest difference between the float evaluation and the double-precision formula
//     over a 9 x 3 x 3 grid of (u_2, delta, epsilon),
//   * twice the largest change of B and C, over the bucket's ends and centre, when Sigma_2 is scaled by
//     the largest relative error of its determinant (powf's rounding and a scattering-table index one
//     entry off), and
//   * twice the forward rounding error bound of the guarded fast point (kBoundK, some 8000 units in the last
//     place where the evaluations differ by a few) at the bucket's centre, on the history's scale; its largest
//     value over the grid instead made a head iteration 2% longer.
// Sampled, not derived: the weights are smooth over a bucket (0.05 cm of u_2), and the factors of two stand
// for what lies between the samples.  A point's voxel is accepted when its position is farther than that
// (plus the fixed-point and float roundings below) from every voxel face, which leaves a few points in 10^5;
// those, and steps without a usable row, are computed by the guarded fast point or in the reference's order.
// In the tests' tens of millions of points every list is the reference's.
//
// The position is fixed point, in voxels from the grid's corner with frac_bits fraction bits: the
// straight line u -> (u cos - t_in sin, u sin + t_in cos) advances in a 64-bit accumulator per axis,
// and the lateral offset is added as a float whose mantissa holds it in units of 2^(4 - frac_bits)
// voxels (adding kMagic leaves it there), so the voxel index is a shift and the face test one
// unsigned comparison per axis.
constexpr float kMagic = 12582912.0f;          // 1.5 * 2^23: the unit of last place is 1
constexpr unsigned kMagicBits = 0x4B400000u;   // its bit pattern
constexpr int kOffsetShift = 4;                // offset units of 2^(4 - frac_bits) voxels
constexpr float kMaxOffset = 4.0e6f;           // < 2^22 units: the sum with kMagic keeps its exponent

// One tabulated weight: quadratic in zeta (u_2 in [-1, 1] over its bucket), linear in sigma.
__device__ __forceinline__ float table_weight(const float4& r, float zeta, float sigma)
{
    return __fmaf_rn(zeta, __fmaf_rn(zeta, r.z, r.y), __fmaf_rn(sigma, r.w, r.x));
}

// What a history's tabulated walk keeps in registers.
struct TableWalk {
    float zeta, sigma, dsigma;        // sigma of the next step and its increment
    float dt, T, dz, V;               // dz and V already in offset units of the z axis
    float sx, sy;                     // offset units of x and y per cm of t
    long long ax, ay, dx, dy;         // line accumulators (frac_bits + 32 fraction bits) and their steps
    unsigned pz, tol;                 // z of the line; face tolerance, left-aligned
    int klast;                        // last step with a row; 0: no table for this history
    bool whole;                       // klast is the walk's last step
    int early;                        // klast of a walk that leaves the table early
    const float4* row;                // row of step 1
};

// (one lane's) set-up; everything in double, the range checks included, so that nothing overflows.
__device__ __forceinline__ TableWalk table_walk_start(const Geometry& g, const MlpTable& tb, const MlpHistory& h,
                                                      double u_in, bool tables_ok)
{
    TableWalk t{};
    t.early = kPathCap;
    const double s = g.mlp_u_step;
    const double q = h.u_2 * tb.inv_width;
    if (!tables_ok || !(q >= 0.0 && q < (double)tb.buckets)) return t;
    const int b = (int)q;
    const MlpBucket bk = tb.bucket[b];
    if (bk.klast <= 0) return t;
    // the walk's loop runs while u_2 - k s > s: b / per_step - 1 steps, unless u_2 / s is so near a whole
    // number that the rounding of the depth recurrence decides; then the rows stop one step earlier
    const double turns = h.u_2 / s, whole = rint(turns);
    const bool regular = fabs(turns - whole) > 1.0e-6;
    t.whole = regular && bk.klast == bk.steps;
    const double unit = (double)(1u << tb.frac_bits);  // fraction units per voxel
    const double limit = 2147483648.0 / unit - 20.0;   // voxels a 32-bit position can hold, offsets included
    const double delta = h.u_2 - (double)(unsigned)(h.u_2 / kPolyTableStep + 0.5) * kPolyTableStep;
    const double epsilon = __fma_rn(-h.u_2, h.u_2, h.u_2_sq);
    t.zeta = (float)((q - b) * 2.0 - 1.0);
    t.dsigma = (float)(bk.kappa * epsilon * kInvSigmaUnit);
    t.sigma = (float)(delta * kInvSigmaUnit) + t.dsigma;
    const double dt = h.t_out - h.t_in, dz = h.z_out - h.z_in;
    const double px = (h.cos_term * u_in - h.sin_term * h.t_in - g.x_zero) * g.inv_voxel_width;
    const double py = (g.y_zero - (h.sin_term * u_in + h.cos_term * h.t_in)) * g.inv_voxel_height;
    const double pz = (g.z_zero - h.z_in) * g.inv_voxel_thickness;
    const double sx = h.cos_term * s * g.inv_voxel_width, sy = -h.sin_term * s * g.inv_voxel_height;
    const double reach = (double)bk.klast;
    const double offset_unit = (double)(1u << (tb.frac_bits - kOffsetShift));
    const double d_max = fmax(fabs(dt), fabs(dz)), a_max = fmax(fabs(h.T_2_1), fabs(h.V_2_1));
    // face tolerance in fraction units: the table's bound, the float evaluation (four roundings of the
    // offset's terms), and 24 units for the offset's rounding to 2^kOffsetShift units and the line's
    const double tol = ((double)bk.err_b * d_max + (double)bk.err_c * a_max + (double)bk.err_r * h.mag_tv +
                        2.4e-7 * (d_max * bk.max_b + (double)bk.max_c * a_max)) * g.inv_voxel_max * unit + 24.0;
    const bool ok = (fabs(px) < limit) & (fabs(px + reach * sx) < limit) & (fabs(py) < limit) &
                    (fabs(py + reach * sy) < limit) & (fabs(pz) < limit) & (tol < unit * 0.125);
    if (!ok) {
        t.whole = false;
        return t;
    }
    const unsigned corner = kMagicBits << kOffsetShift;  // the offset's bits carry kMagic's
    const double scale = unit * 4294967296.0;
    t.ax = __double2ll_rn(px * scale) - ((long long)corner << 32);
    t.ay = __double2ll_rn(py * scale) - ((long long)corner << 32);
    t.dx = __double2ll_rn(sx * scale);
    t.dy = __double2ll_rn(sy * scale);
    t.pz = (unsigned)__double2int_rn(pz * unit) - corner;
    t.tol = (unsigned)__double2int_ru(tol) << (32 - tb.frac_bits);
    t.dt = (float)dt;
    t.T = (float)h.T_2_1;
    t.dz = (float)(-dz * g.inv_voxel_thickness * offset_unit);
    t.V = (float)(-h.V_2_1 * g.inv_voxel_thickness * offset_unit);
    t.sx = (float)(-h.sin_term * g.inv_voxel_width * offset_unit);
    t.sy = (float)(-h.cos_term * g.inv_voxel_height * offset_unit);
    t.klast = regular || bk.klast < bk.steps ? bk.klast : bk.klast - 1;
    t.row = tb.rows + 2 * (long long)bk.row;
    // A point that is not proven costs a start from the history's inputs (general_point_of), which pays for a few
    // of them only.  Where many are to be expected the walk leaves the table early: at once for a line that ends
    // beyond the grid's zero corner, and for an oblique line over thin slices at the step where its offset
    // outgrows the fixed point.  300k histories of a 20 degree cone over the head grid with slices of 0.625 /
    // 0.3125 mm: path kernel 0.78 / 0.96 ms; with a general point for each such step 1.81 / 2.29, with certain points
    // from the start 0.93 / 0.93.  (Not for lines along a voxel face: of 4M head histories 25 to 40 have eight points
    // that are not proven, and walking on without the table from the eighth made an iteration 150 us longer, the
    // time that one such walk takes on its own.)
    if (fmin(fmin(px, px + reach * sx), fmin(py, py + reach * sy)) < -2.0) t.klast = t.early = 0;
    const float dt_max = tb.t_max, dz_max = kMaxOffset;
    if (fabsf(t.dt) * bk.max_b + fabsf(t.T) * bk.max_c >= dt_max || fabsf(t.dz) * bk.max_b + fabsf(t.V) * bk.max_c >= dz_max)
        while (t.klast > 0) {
            const float4* r = t.row + 2 * (t.klast - 1);
            const float sigma = t.sigma + (t.klast - 1) * t.dsigma;
            const float B = table_weight(__ldg(r), t.zeta, sigma), C = table_weight(__ldg(r + 1), t.zeta, sigma);
            if (fabsf(B * t.dt + C * t.T) < dt_max && fabsf(B * t.dz + C * t.V) < dz_max) break;
            t.klast = t.early = t.klast * 7 / 8;
        }
    t.whole = t.whole && t.klast == bk.klast;
    return t;
}

// The tabulated point of the step whose row is r0, r1: its voxel, and whether the estimated error clears the faces.
__device__ __forceinline__ bool table_point(const Geometry& g, const MlpTable& tb, const TableWalk& t, const float4& r0,
                                            const float4& r1, uint32_t& voxel)
{
    const float B = table_weight(r0, t.zeta, t.sigma), C = table_weight(r1, t.zeta, t.sigma);
    const float lateral = __fmaf_rn(B, t.dt, __fmul_rn(C, t.T));
    const float vertical = __fmaf_rn(B, t.dz, __fmul_rn(C, t.V));
    const unsigned px = (unsigned)(t.ax >> 32) + (__float_as_uint(__fmaf_rn(lateral, t.sx, kMagic)) << kOffsetShift);
    const unsigned py = (unsigned)(t.ay >> 32) + (__float_as_uint(__fmaf_rn(lateral, t.sy, kMagic)) << kOffsetShift);
    const unsigned pz = t.pz + (__float_as_uint(__fadd_rn(vertical, kMagic)) << kOffsetShift);
    const int frac_bits = tb.frac_bits, left = 32 - frac_bits;
    const unsigned band = t.tol << 1;
    const bool proven = ((px << left) + t.tol >= band) & ((py << left) + t.tol >= band) & ((pz << left) + t.tol >= band) &
                        ((int)(px | py) >= 0) & (fabsf(lateral) < tb.t_max) & (fabsf(vertical) < kMaxOffset);
    // above the grid's top the index is mirrored (calculate_voxel_GPU takes |z - zero|); faces mirror with it
    voxel = (px >> frac_bits) + (py >> frac_bits) * (unsigned)g.columns +
            ((unsigned)abs((int)pz) >> frac_bits) * (unsigned)(g.columns * g.rows);
    return proven;
}

// A history's voxel list on its way to path storage: entries wait in a 16-slot ring in shared memory
// and leave it 8 at a time, as one 32-byte sector.  flush() is called by all lanes of a warp at the
// same steps, at most 8 put() apart, so it runs for most lanes at once: flushing each lane when its 8
// entries are full ran that code for one or two lanes in most loop trips.
constexpr int kStageSlots = 16;
constexpr int kStageStride = kStageSlots + 4;  // words per thread: 16-byte aligned, spread over the banks
struct ListStage {
    uint32_t slots;  // shared-memory address of this thread's ring
    uint32_t* out;   // 32-byte aligned; the history's path bound covers every entry, rounded up to 8
    int n, sent;
    uint32_t last;
    __device__ __forceinline__ void store(int slot, uint32_t voxel)
    {
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(slots + 4 * slot), "r"(voxel) : "memory");
    }
    __device__ __forceinline__ void first(uint32_t voxel)
    {
        last = voxel;
        store(0, voxel);
        n = 1;
        sent = 0;
    }
    // Appends voxel unless it repeats the last entry (B.cu:9244-9251), without a branch: the slot of
    // the last entry is written again.
    __device__ __forceinline__ void put(uint32_t voxel)
    {
        n += voxel != last ? 1 : 0;
        last = voxel;
        store((n - 1) & (kStageSlots - 1), voxel);
    }
    __device__ __forceinline__ void send()
    {
        const uint32_t from = slots + 4 * (sent & (kStageSlots - 1));
        uint4 a, b;
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w) : "r"(from) : "memory");
        asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w) : "r"(from + 16) : "memory");
        uint4* to = reinterpret_cast<uint4*>(out + sent);
        to[0] = a;
        to[1] = b;
        sent += 8;
    }
    __device__ __forceinline__ void flush()
    {
        if (n - sent >= 8) send();
    }
    __device__ __forceinline__ void finish()
    {
        while (sent < n) send();  // the last sector padded with stale slots
    }
};

// The set-up of history i (position in h), from its inputs.
__device__ __forceinline__ MlpStart mlp_start_of(const Geometry& g, const Tables& tab, const HistorySoA& h, long long i,
                                                 unsigned& flags, double* chord)
{
    double xy_entry_angle = __ldg(h.xy_entry_angle + i), xy_exit_angle = __ldg(h.xy_exit_angle + i);
    const double xz_entry_angle = __ldg(h.xz_entry_angle + i), xz_exit_angle = __ldg(h.xz_exit_angle + i);
    const MlpStart m = mlp_start(g, tab, __ldg(h.x_entry + i), __ldg(h.y_entry + i), __ldg(h.z_entry + i),
                                 __ldg(h.x_exit + i), __ldg(h.y_exit + i), __ldg(h.z_exit + i), xy_entry_angle,
                                 xy_exit_angle, xz_entry_angle, xz_exit_angle, flags);
    if (chord)
        *chord = effective_chord_length(g, (xy_entry_angle + xy_exit_angle) / 2.0, (xz_entry_angle + xz_exit_angle) / 2.0);
    return m;
}

// The voxel of one point (step k, u and depth as the walk carries them) by the guarded fast point or
// in the reference's order.
__device__ __forceinline__ uint32_t general_point(const Geometry& g, const Tables& tab,
                                                  const StepConst* __restrict__ steps, const MlpStart& m, int k,
                                                  double depth_2_go, double u_shifted)
{
    const StepConst& st = steps[k];
    const Sigma2 m2 = sigma2_moments(m.h, st, tab.scattering_table,
                                     m.sigma_2_index - (unsigned)(k - 1) * g.sigma_index_step);
    uint32_t voxel;
    if (g.exact_fast_points && mlp_point_fast(g, m.h, st, m2.sigma_t2, m2.sigma_t2_theta2, m2.sigma_theta2,
                                              m2.determinant, depth_2_go, u_shifted, voxel))
        return voxel;
    double t_1, v_1;
    mlp_point_rest(m.h, st, m2, depth_2_go, t_1, v_1);
    return mlp_voxel(g, m.h, u_shifted, t_1, v_1);
}

// The depth and position of step k as the walk's recurrences carry them (step 1: u_2 - s and u_in + s).
__device__ __forceinline__ void recurrences(const MlpStart& m, double s, int k, double& depth_2_go, double& u_shifted)
{
    depth_2_go = m.depth_2_go;
    u_shifted = m.u_shifted + s;
    for (int j = 1; j < k; j++) {
        depth_2_go -= s;
        u_shifted += s;
    }
}

// What the table loop leaves to the general points starts again from the history's inputs, so that the
// loop keeps nothing for it.  The voxel of step k of history i of h:
__device__ __forceinline__ uint32_t general_point_of(const Geometry& g, const Tables& tab,
                                                         const StepConst* __restrict__ steps, const HistorySoA& h,
                                                         int i, int k)
{
    unsigned flags = 0;
    const MlpStart m = mlp_start_of(g, tab, h, i, flags, nullptr);
    double depth_2_go, u_shifted;
    recurrences(m, g.mlp_u_step, k, depth_2_go, u_shifted);
    return general_point(g, tab, steps, m, k, depth_2_go, u_shifted);
}

// The walk of history i from step k to its end (not inlined: few histories need it), its list of at most cap entries finished; returns the
// list's length, and adds the walk's flags.
static __device__ __noinline__ int general_walk_of(const Geometry& g, const Tables& tab,
                                                   const StepConst* __restrict__ steps, int kmax, const HistorySoA& h,
                                                   int i, int k, int cap, ListStage list, unsigned* flags)
{
    const double s = g.mlp_u_step;
    unsigned f = 0;
    const MlpStart m = mlp_start_of(g, tab, h, i, f, nullptr);
    double depth_2_go, u_shifted;
    recurrences(m, s, k, depth_2_go, u_shifted);
    int trips = 0;
    while (m.tables_ok && depth_2_go > s) {
        if (k > kmax) {  // cannot happen while the u_2 index is inside the tables
            f |= kFlagTableRange;
            break;
        }
        const uint32_t voxel = general_point(g, tab, steps, m, k, depth_2_go, u_shifted);
        if (voxel >= (uint32_t)g.padded_voxels) f |= kFlagVoxelOOB;
        if (list.n < cap) list.put(voxel);
        else f |= kFlagPathOverflow;  // cannot happen: cap bounds the loop count
        depth_2_go -= s;
        u_shifted += s;
        k++;
        if ((++trips & 7) == 0) list.flush();
    }
    list.finish();
    *flags |= f;
    return list.n;
}

// The exact walk of the path kernel: the same voxel list as mlp_walk_exact, without the sum over x, for
// history i of h; all lanes of a warp call it, those without a history (cap = 0) write nothing.  The
// warp runs its lanes' table rows in lockstep in an inner loop, and leaves that loop together when a
// point is not proven.  With the general point inside the hot loop, called or inlined, its registers
// were spilled in every step (7.7 ms per 4M head histories against 3.3 this way and 3.1 without any
// general point).
__device__ __forceinline__ int mlp_walk_table(const Geometry& g, const Tables& tab, const MlpTable& tb,
                                              const StepConst* __restrict__ steps, int kmax, const HistorySoA& h,
                                              int i, int cap, uint32_t slots, uint32_t* out, double* chord,
                                              unsigned* flags)
{
    TableWalk t{};
    t.whole = true;
    t.early = kPathCap;
    uint32_t first = 0;
    if (cap > 0) {
        double c;
        const MlpStart m = mlp_start_of(g, tab, h, i, *flags, &c);
        *chord = c;
        t = table_walk_start(g, tb, m.h, m.u_in, m.tables_ok);
        if (t.klast >= cap) {  // cannot happen: the bound is at least the steps + 2
            t.klast = cap - 1;
            t.whole = false;
        }
        first = __ldg(h.first_MLP_voxel + i);
    }
    // once one lane of the warp walks on without the table, the others' points cost nothing there
    const int early = __reduce_min_sync(0xffffffffu, t.early);
    if (t.klast > early) {
        t.klast = early;
        t.whole = false;
    }
    ListStage list{slots, out, 0, 0, 0u};
    list.first(first);
    bool outside = first >= (uint32_t)g.padded_voxels;
    const int warp_last = __reduce_max_sync(0xffffffffu, t.klast);
    for (int k = 1; k <= warp_last;) {
        uint32_t voxel = 0;
        bool proven = true;
        for (;;) {
            const bool on = k <= t.klast;
            voxel = list.last;
            if (on) {
                const float4 r0 = __ldg(t.row), r1 = __ldg(t.row + 1);
                t.row += 2;
                t.ax += t.dx;
                t.ay += t.dy;
                proven = table_point(g, tb, t, r0, r1, voxel);
                t.sigma += t.dsigma;
            }
            if (__any_sync(0xffffffffu, !proven)) break;
            outside |= voxel >= (uint32_t)g.padded_voxels;
            list.put(voxel);
            if ((k & 7) == 0) list.flush();
            if (++k > warp_last) break;
        }
        if (k > warp_last) break;
        if (!proven) voxel = general_point_of(g, tab, steps, h, i, k);
        __syncwarp();
        outside |= voxel >= (uint32_t)g.padded_voxels;
        list.put(voxel);
        if ((k & 7) == 0) list.flush();
        k++;
    }
    if (cap <= 0) return 0;
    if (outside) *flags |= kFlagVoxelOOB;
    if (t.whole) {
        list.finish();
        return list.n;
    }
    list.flush();
    return general_walk_of(g, tab, steps, kmax, h, i, t.klast + 1, cap, list, flags);
}

// ------------------------------------------------------------------------------------------
// Mixed precision (PCT_PRECISION_MIXED).  FP64 is kept where cancellation needs it: the Sigma_2
// moments (differences of tabulated integrals, which cancel towards the exit) at every point, and
// within Geometry::mixed_fp64_margin of the entry or the exit also the inverse of Sigma_2, the
// matrix M = Sigma_1^-1 + R_1^T Sigma_2^-1 R_1 and its determinant (ill-conditioned there; FP32
// in between).  The right-hand sides, the solve t_1 = [M^-1]_0 . rhs, the rotation back to x/y
// and the voxel indices run in FP32.  Every operation is an explicit
// intrinsic, so the result does not depend on the translation unit's contraction flags.
// ------------------------------------------------------------------------------------------

struct MlpHistoryF {
    float sin_term, cos_term, t_in, t_out, z_in, z_out, T_2_1, V_2_1;
};

__device__ __forceinline__ MlpHistoryF mlp_history_f(const MlpHistory& h)
{
    return MlpHistoryF{(float)h.sin_term, (float)h.cos_term, (float)h.t_in, (float)h.t_out,
                       (float)h.z_in,     (float)h.z_out,    (float)h.T_2_1, (float)h.V_2_1};
}

// Whether the mixed walk inverts Sigma_2 and M in FP64 at loop trip k: within
// g.mixed_fp64_margin of the entry (u_1 = k * MLP_U_STEP, where Sigma_1 is small) or of the exit
// (depth_2_go, where Sigma_2 is small) both are ill-conditioned; in between FP32 suffices.
__device__ __forceinline__ bool mixed_fp64_inverse(const Geometry& g, int k, double depth_2_go)
{
    return depth_2_go < g.mixed_fp64_margin || (double)k * g.mlp_u_step < g.mixed_fp64_margin;
}

__device__ __forceinline__ void mlp_point_mixed(const MlpHistory& h, const MlpHistoryF& hf, const StepConst& st,
                                                const double* __restrict__ scattering, double depth_2_go,
                                                unsigned sigma_2_index, bool fp64_inverse, float& t_1, float& v_1)
{
    // FP64: the Sigma_2 moments (differences of tabulated integrals)
    const double sigma_t2 =
        __dsub_rn(__fma_rn(h.two_u_2, st.p23, __fma_rn(-h.u_2_sq, st.p12, h.u_2_poly_3_12)), st.p34);
    const double sigma_t2_theta2 = __dadd_rn(__fma_rn(-h.u_2, st.p12, h.u_2_poly_2_6), st.p23);
    const double sigma_theta2 = __dsub_rn(h.u_2_poly_1_2, st.p12);
    const double scat = __ldg(scattering + sigma_2_index);
    const float d = (float)depth_2_go;
    float i00, i01, a0, a1, a2;
    if (fp64_inverse) {
        // FP64: Sigma_2^-1, M and the first row of M^-1
        const double det2 =
            __dmul_rn(scat, __fma_rn(sigma_t2, sigma_theta2, -__dmul_rn(sigma_t2_theta2, sigma_t2_theta2)));
        const double r2 = __drcp_rn(det2);
        const double S0 = __dmul_rn(sigma_theta2, r2), S1 = __dmul_rn(sigma_t2_theta2, r2), S2 = __dmul_rn(sigma_t2, r2);
        const double c = __fma_rn(S0, depth_2_go, -S1);
        const double m0 = __dadd_rn(st.s1i0, S0);
        const double m1 = __dsub_rn(c, st.s1i1);
        const double m3 = __fma_rn(depth_2_go, __dsub_rn(c, S1), __dadd_rn(st.s1i2, S2));
        const double rM = __drcp_rn(__fma_rn(m0, m3, -__dmul_rn(m1, m1)));
        i00 = (float)__dmul_rn(m3, rM);
        i01 = (float)(-__dmul_rn(m1, rM));
        a0 = (float)S0;
        a1 = (float)S1;
        a2 = (float)S2;
    } else {
        // FP32: the same inversions away from the entry and the exit
        const float st2 = (float)sigma_t2, stt = (float)sigma_t2_theta2, sth = (float)sigma_theta2;
        const float det2 = __fmul_rn((float)scat, __fmaf_rn(st2, sth, -__fmul_rn(stt, stt)));
        const float r2 = __frcp_rn(det2);
        a0 = __fmul_rn(sth, r2);
        a1 = __fmul_rn(stt, r2);
        a2 = __fmul_rn(st2, r2);
        const float c = __fmaf_rn(a0, d, -a1);
        const float m0 = __fadd_rn(st.s1i0f, a0);
        const float m1 = __fsub_rn(c, st.s1i1f);
        const float m3 = __fmaf_rn(d, __fsub_rn(c, a1), __fadd_rn(st.s1i2f, a2));
        const float rM = __frcp_rn(__fmaf_rn(m0, m3, -__fmul_rn(m1, m1)));
        i00 = __fmul_rn(m3, rM);
        i01 = -__fmul_rn(m1, rM);
    }
    // FP32: right-hand sides and the solve
    float c3 = __fmaf_rn(a0, hf.t_out, -__fmul_rn(a1, hf.T_2_1));
    float r0 = __fmaf_rn(st.s1i0f, hf.t_in, c3);
    float r1 = __fmaf_rn(d, c3, __fmaf_rn(a2, hf.T_2_1, -__fmaf_rn(a1, hf.t_out, __fmul_rn(st.s1i1f, hf.t_in))));
    t_1 = __fmaf_rn(i00, r0, __fmul_rn(i01, r1));
    c3 = __fmaf_rn(a0, hf.z_out, -__fmul_rn(a1, hf.V_2_1));
    r0 = __fmaf_rn(st.s1i0f, hf.z_in, c3);
    r1 = __fmaf_rn(d, c3, __fmaf_rn(a2, hf.V_2_1, -__fmaf_rn(a1, hf.z_out, __fmul_rn(st.s1i1f, hf.z_in))));
    v_1 = __fmaf_rn(i00, r0, __fmul_rn(i01, r1));
}

__device__ __forceinline__ int voxel_index_1d_f(float zero, float pos, float inv_size)
{
    const float q = __fmul_rn(fabsf(__fsub_rn(pos, zero)), inv_size);
    return q < 2147483000.0f ? (int)q : -1;
}

__device__ __forceinline__ uint32_t mlp_voxel_mixed(const Geometry& g, const MlpHistoryF& hf, float u_shifted,
                                                    float t_1, float v_1)
{
    const float x_1 = __fmaf_rn(hf.cos_term, u_shifted, -__fmul_rn(hf.sin_term, t_1));
    const float y_1 = __fmaf_rn(hf.sin_term, u_shifted, __fmul_rn(hf.cos_term, t_1));
    const int vx = voxel_index_1d_f(g.x_zero_f, x_1, g.inv_voxel_width_f);
    const int vy = voxel_index_1d_f(g.y_zero_f, y_1, g.inv_voxel_height_f);
    const int vz = voxel_index_1d_f(g.z_zero_f, v_1, g.inv_voxel_thickness_f);
    long long v64 = (long long)vx + (long long)vy * g.columns + (long long)vz * g.columns * g.rows;
    if (vx < 0 || vy < 0 || vz < 0 || v64 > 0x7fffffffLL) v64 = 0x7fffffffLL;
    return (uint32_t)v64;
}

// The mixed-precision walk: same control flow, depth/position recurrences and de-duplication as
// the exact walk; the points and voxels as above.
template <bool kSumX, class Emit>
__device__ __forceinline__ WalkResult mlp_walk_mixed(const Geometry& g, const Tables& tab,
                                                     const StepConst* __restrict__ steps, int kmax,
                                                     const float* __restrict__ x, uint32_t first_MLP_voxel,
                                                     double x_in_object, double y_in_object, double z_in_object,
                                                     double x_out_object, double y_out_object, double z_out_object,
                                                     double xy_entry_angle, double xz_entry_angle,
                                                     double xy_exit_angle, double xz_exit_angle, Emit emit)
{
    const double s = g.mlp_u_step;
    WalkResult r;
    r.flags = 0;
    MlpStart m = mlp_start(g, tab, x_in_object, y_in_object, z_in_object, x_out_object, y_out_object, z_out_object,
                           xy_entry_angle, xy_exit_angle, xz_entry_angle, xz_exit_angle, r.flags);
    const MlpHistoryF hf = mlp_history_f(m.h);
    double depth_2_go = m.depth_2_go, u_shifted = m.u_shifted;
    unsigned sigma_2_index = m.sigma_2_index;
    PathWriter<kSumX, Emit> w{g, x, emit, r, 0u, 0};
    w.first(first_MLP_voxel);
    r.chord = effective_chord_length(g, (xy_entry_angle + xy_exit_angle) / 2.0, (xz_entry_angle + xz_exit_angle) / 2.0);
    r.aia = r.chord * r.chord;
    int k = 1;
    while (m.tables_ok && depth_2_go > s) {
        if (k > kmax) {
            r.flags |= kFlagTableRange;
            break;
        }
        float t_1, v_1;
        mlp_point_mixed(m.h, hf, steps[k], tab.scattering_table, depth_2_go, sigma_2_index,
                        mixed_fp64_inverse(g, k, depth_2_go), t_1, v_1);
        u_shifted = __dadd_rn(u_shifted, s);
        w.visit(mlp_voxel_mixed(g, hf, (float)u_shifted, t_1, v_1));
        depth_2_go = __dsub_rn(depth_2_go, s);
        sigma_2_index -= g.sigma_index_step;
        k++;
    }
    r.n = w.n < kPathCap ? w.n : kPathCap;
    return r;
}

}  // namespace pct
