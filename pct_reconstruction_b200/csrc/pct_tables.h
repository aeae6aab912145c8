// pct_tables.h -- host construction of the MLP lookup tables and the per-step table.
#pragma once

#include <vector>

#include "pct_common.cuh"

namespace pct {

struct HostTables {
    std::vector<double> sin_table, cos_table, scattering_table;
    std::vector<double> poly_1_2, poly_2_3, poly_3_4, poly_2_6, poly_3_12;
};

// History-independent terms of MLP step k (u_1 = k*MLP_U_STEP): the u_1 polynomials used by
// Sigma_2 and the inverse of Sigma_1 (entries Sigma_1I[0..2] of B.cu:9193-9195).
struct StepConst {
    double p12, p23, p34;
    double s1i0, s1i1, s1i2;
    float s1i0f, s1i1f, s1i2f;  // float copies for the mixed-precision right-hand sides and inversions
};

// Tabulated MLP points (pct_mlp.cuh, "Tabulated points"): per bucket of u_2 its first row (2 float4
// per row, step 1 first), last step with a row (0: none) and the bounds on its rows.
struct MlpBucket {
    int row, klast, steps;  // steps: those of a walk whose u_2 lies inside the bucket
    float err_b, err_c;  // largest deviation of the weights B and C from the reference's
    float err_r;         // rounding error of the reference's point per cm of the history's scale (mag_tv)
    float max_b, max_c;  // largest |B| and |C|
    double kappa;        // sigma = delta + k kappa epsilon
};
struct MlpTable {
    const float4* rows;
    const MlpBucket* bucket;
    int buckets;     // 0: no table (every point by the guarded fast point or in the reference's order)
    int frac_bits;   // fraction bits of the fixed-point positions
    float t_max;       // largest lateral offset (cm) a position's offset holds
    double inv_width;  // 1 / bucket width
};
constexpr double kSigmaUnit = 2.5e-5;  // half the polynomial-table step: delta in units of its range
constexpr double kInvSigmaUnit = 40000.0;

double trig_table_min();
double trig_table_step();
int trig_table_elements();
int coeff_table_elements();
int poly_table_elements();

void build_host_tables(HostTables& t);
// Last MLP loop iteration k whose u_1 indices (k*pstep, k*sstep) stay inside the tables.
int step_table_kmax(const HostTables& t, double mlp_u_step);

}  // namespace pct
