// emu_fp64.cuh -- building blocks of the FP64 step kernels that work on the
// combined self-interaction layout (Comb<NF>: k_steps_1d).
#pragma once
#include "emu_device.cuh"

namespace emu {

// a combined FP64 mesh: per cell the NG combined values, then the diagonal
// number densities N_ii, Nbar_ii (kDiagSlots) that compute_dt reads
template <int NF>
constexpr int kCombSlots = Comb<NF>::NG + kDiagSlots;

// D += A B on the FP64 tensor cores, 8 x 4 by 4 x 8: lane l holds A[l / 4][l % 4],
// B[l % 4][l / 4] and D[l / 4][2 (l % 4) + {0, 1}].  IEEE FMAs, at the rate of
// the FP64 pipe (measured 64 FMA per clock and SM), for one issue slot per
// 256 FMAs.
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

// H of species sp from the self-interaction part hs (nu): vacuum and matter
// added, nubar with the reference's sign rule (generate_code.py:317-355).
// h may be hs.
template <int NF>
__device__ __forceinline__ void species_hamiltonian(const DevParams& P, const double* hs, double vscale, int sp,
                                                    double* h)
{
    using H = Herm<NF>;
    const double mat = P.sqrt2GF_inv_vol * P.matter;
#pragma unroll
    for (int e = 0; e < NF * NF; e++) {
        const double m2 = sp == 0 ? P.M2[0][e] : P.M2[1][e];
        double si = hs[e];
        if (e == 0) si += mat;
        h[e] = fma(m2, vscale, (sp == 0 || H::is_im(e)) ? si : -si);
    }
}

// compute_dt without the adaptive branch (the operations of cell_potentials
// and dt_finish): the factor from a number per cell to V_stupid, and dt from
// the largest number vmax (vacuum bound included); st_dt: no limiter
template <int NF>
__device__ __forceinline__ double stupid_factor(const DevParams& P)
{
    return 2.0 * NF * M_SQRT2 * P.GF / P.cell_volume;
}
__device__ __forceinline__ double next_dt_stupid(const DevParams& P, double vmax, double factor, int& st_dt)
{
    const double vs = vmax * factor + P.vvac_max;
    const double dtf = P.flavor_cfl_factor > 0.0 ? kHbar / vs * P.flavor_cfl_factor : 0.0;
    const double dtt = P.dt_translation;
    if (dtt != 0.0 && dtf != 0.0) return fmin(dtt, dtf);
    if (dtt != 0.0) return dtt;
    if (dtf == 0.0) st_dt = 1;
    return dtf;
}

}  // namespace emu
