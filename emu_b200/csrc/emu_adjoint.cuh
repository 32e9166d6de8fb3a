// emu_adjoint.cuh -- per-particle pieces of the discrete adjoint, shared by the
// tile kernels (emu_adjoint.cu) and the 1D sweep (emu_k_steps1d.cu).
#pragma once
#include "emu_device.cuh"

namespace emu {
namespace {

// VJP of K = C(H, F) = -i/hbar [H, F].  With the Hermitian matrix L whose
// trace product is the contraction with lam, Tr(L K) = sum_c lam_c K_c (L_ii =
// lam_ii, L_ij = (lam_re + i lam_im) / 2), cyclic permutation of the trace
// gives Tr(L C(H, F)) = Tr(C(L, H) F) = Tr(C(F, L) H): two commutators (the
// sums over unit vectors they replace were 18 of them for three flavors, half
// of the adjoint stage's arithmetic).
template <int NF>
__device__ __forceinline__ void commutator_vjp(const double* h, const double* f, const double* lam, double* lamH,
                                               double* lamF, double inv_hbar)
{
    using H = Herm<NF>;
    constexpr int NH = NF * NF;
    double l[NH];
#pragma unroll
    for (int e = 0; e < NH; e++) l[e] = H::is_diag(e) ? lam[e] : 0.5 * lam[e];
    commutator<NF, double>(l, h, lamF, inv_hbar);
    commutator<NF, double>(f, l, lamH, inv_hbar);
#pragma unroll
    for (int e = 0; e < NH; e++)
        if (!H::is_diag(e)) {
            lamF[e] *= 2.0;
            lamH[e] *= 2.0;
        }
}

// VJP of renormalize<NF>() at input fin (one species): replays the forward
// branch decisions with the same arithmetic.
template <int NF>
__device__ __forceinline__ void renormalize_vjp(const double* fin, double L, double maxError, const double* lam_out,
                                                double* lam_in)
{
    using H = Herm<NF>;
    constexpr int NH = NF * NF;
    double f[NH];
#pragma unroll
    for (int e = 0; e < NH; e++) f[e] = fin[e];
    double sumP = 0.0;
#pragma unroll
    for (int i = 0; i < NF; i++) sumP = __dadd_rn(sumP, f[H::re(i, i)]);
    const double err = sumP - 1.0;
    const bool trace_fix = fabs(err) > maxError;
    if (trace_fix) {
#pragma unroll
        for (int i = 0; i < NF; i++) f[H::re(i, i)] = __dsub_rn(f[H::re(i, i)], __ddiv_rn(err, (double)NF));
    }
    bool clamped[NF];
#pragma unroll
    for (int i = 0; i < NF; i++) {
        clamped[i] = f[H::re(i, i)] < -maxError;
        if (clamped[i]) f[H::re(i, i)] = 0;
    }
    const double length = su_length<NF>(f);
    const bool rescale = fabs(length - L) > maxError;
    double lam[NH];
#pragma unroll
    for (int e = 0; e < NH; e++) lam[e] = lam_out[e];
    if (rescale) {
        // f' = f L / length(f):  lam_f = (L/len) lam - (L/len^2) (lam . f) grad len
        double g[NH];
#pragma unroll
        for (int e = 0; e < NH; e++) g[e] = H::is_diag(e) ? 0.0 : f[e] / length;
#pragma unroll
        for (int l = 1; l < NF; l++) {
            const double cl = (l == 1) ? 0.5 : 0.28867513459481287;
            double t = 0.0;
#pragma unroll
            for (int i = 0; i < l; i++) t += cl * f[H::re(i, i)];
            t -= cl * l * f[H::re(l, l)];
#pragma unroll
            for (int i = 0; i < l; i++) g[H::re(i, i)] += t * cl / length;
            g[H::re(l, l)] -= t * cl * l / length;
        }
        double dot = 0.0;
#pragma unroll
        for (int e = 0; e < NH; e++) dot += lam[e] * f[e];
        const double a = L / length, b = L / (length * length) * dot;
#pragma unroll
        for (int e = 0; e < NH; e++) lam[e] = a * lam[e] - b * g[e];
    }
#pragma unroll
    for (int i = 0; i < NF; i++)
        if (clamped[i]) lam[H::re(i, i)] = 0.0;
    if (trace_fix) {
        double m = 0.0;
#pragma unroll
        for (int i = 0; i < NF; i++) m += lam[H::re(i, i)];
        m /= NF;
#pragma unroll
        for (int i = 0; i < NF; i++) lam[H::re(i, i)] -= m;
    }
#pragma unroll
    for (int e = 0; e < NH; e++) lam_in[e] = lam[e];
}

}  // namespace
}  // namespace emu
