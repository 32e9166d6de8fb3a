// emu_fp64_impl.cuh -- the FP64 RK4 stage kernels on combined meshes
// (k_stage64) and their deposits, instantiated per flavor count in
// emu_k_comb64_<nf>.cu.  Interpolation and deposit: emu_tile64.cuh.
#pragma once
#include "emu_kernels_impl.cuh"

namespace emu {
namespace {

template <int NF, class T>
constexpr int stage64_smem()
{
    return 8 * (kBlock * T::template row<Comb<NF>::NV>() + (3 + 2 * NF) * T::VS) + 4 * (2 * kBlock + 8);
}

// the stage-4 push of the FP64 path (x += sum_i dt b_i c p/p^t, t likewise,
// then the wrap; one definition for stage 4 and the re-sort keys before it)
__device__ __forceinline__ void rk4_push64(const DevParams& P, double dt, const double* v, double* xn, double& tn)
{
    const double kxv[3] = {v[0] * kC, v[1] * kC, v[2] * kC};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const double w = dt * kRK4B[i];
#pragma unroll
        for (int d = 0; d < 3; d++) xn[d] = __dadd_rn(__dmul_rn(w, kxv[d]), xn[d]);
        tn = __dadd_rn(w, tn);
    }
#pragma unroll
    for (int d = 0; d < 3; d++) xn[d] = wrap_coord(xn[d], P.L[d]);
}

// compute_dt over a combined mesh's diagonal slots, in a kernel of which
// every block calls it once (the scheme of dt_reduce_and_finish)
template <int NF>
__device__ __forceinline__ void dt_reduce_comb64(const DevParams& P, const double* __restrict__ mesh, StepCtl* ctl,
                                                 unsigned ncb)
{
    double vm = 0.0, unused = 0.0;
    if (P.flavor_cfl_factor > 0.0 && blockIdx.x < ncb) {
        const long long stride = (long long)ncb * blockDim.x;
        for (long long c = blockIdx.x + (long long)ncb * threadIdx.x; c < P.ncells; c += stride) {
            const double2* d = reinterpret_cast<const double2*>(mesh + c * kCombSlots<NF> + Comb<NF>::NG);
#pragma unroll
            for (int i = 0; i < NF; i++) {
                const double2 t = __ldcg(d + i);
                vm = fmax(vm, fmax(t.x, t.y));
            }
        }
        vm = fmax(vm, P.cell_volume * P.Ye * P.rho / kMp) * stupid_factor<NF>(P);
    }
    // (the barrier: every thread of the block has read this step's dt)
    if (blockIdx.x < ncb) block_max2(vm, unused);
    else __syncthreads();
    if (threadIdx.x == 0) {
        if (blockIdx.x < ncb) {
            atomicMax(&ctl->vmax_bits[1], (unsigned long long)__double_as_longlong(vm));
            __threadfence();
        }
        if (atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1) {
            __threadfence();
            dt_finish(P, ctl, DT_ADVANCE);
        }
    }
}

// the state of a step that a re-sort scatters: fields that no stage changes
// (not rslot: both particle buffers share it, and other CTAs of stage 4 still
// read it; the deposit that follows sets it)
__device__ __forceinline__ void sc_static64(const DevState& S, const DevState& D, long long p, long long q)
{
    D.id[q] = S.id[p];
#pragma unroll
    for (int sp = 0; sp < 2; sp++) {
        D.Nn[sp][q] = S.Nn[sp][p];
        D.Ll[sp][q] = S.Ll[sp][p];
    }
#pragma unroll
    for (int d = 0; d < 4; d++) D.pup[d][q] = S.pup[d][p];
    D.vscale[q] = S.vscale[p];
#pragma unroll
    for (int d = 0; d < 3; d++) D.vhat[d][q] = S.vhat[d][p];
}

// Stage SG of an FP64 RK4 step on combined meshes.  A stage stores its K in
// fs, from which the next one forms Y = y0 + a dt K, and stage 2 alone the
// running sum acc = y0 + dt b_1 K_1 + dt b_2 K_2 (the terms of K_1 and K_3 are
// added by the stages that read those anyway): 234 words of state per
// particle and step where Y and the sum stored by every stage took 288, with
// the same operations in the reference's order.
// What bounds it: the phases of a tile add up (stage 1 at 32^3 cells x 96
// directions, 650 us: base 254, interpolation 160, deposit 235; the matrix
// instruction's floor is 185 us for each of the two products, 27 cells padded
// to 28).  Stages 1-4 and the re-sort there: 637/690/865/772 + 471 us, where a
// thread per particle on the full meshes took 3710/4057/4065/2321 + 2352; 90
// x 77 cells x 60 directions: 2149 -> 445 us a step.  Four CTAs per SM: five
// (677 us) spill, three (741) leave latency open.
// SC (stage 4 before a re-sort): the new state and every unchanged field of
// particle p go to slot inv[p] of D, the other particle buffer (keys by stage
// 3 into kout, iout, the sort before this kernel, D's deposit after it).
template <int NF, int WX, int WY, int WZ, int KS, int SG, bool SC>
__global__ void __launch_bounds__(kBlock, 4)
    k_stage64(DevParams P, DevState S, const double* __restrict__ mesh_in, double* __restrict__ mesh_out,
              double* mesh_zero, double* full_zero, StepCtl* ctl, int dt_mode, DevState D,
              const unsigned* __restrict__ inv, unsigned* __restrict__ kout, unsigned* __restrict__ iout)
{
    using T = Tile64<NF, WX, WY, WZ, KS>;
    using H = Herm<NF>;
    using C = Comb<NF>;
    constexpr int NH = NF * NF, NV = C::NV, WP = T::WP, VS = T::VS, RW = T::template row<NV>();
    constexpr int s = SG;
    static_assert(!SC || SG == 4, "the re-sort scatter is stage 4's");
    extern __shared__ __align__(16) unsigned char tile_smem[];
    Smem64<NF, T, RW> sm(tile_smem);
    if (s == 1) grid_dep_wait();   // (the control block is the previous step's last kernel's)
    const int done = __ldcg(&ctl->done);
    const double dt = __ldcg(&ctl->dt);
    const int t = threadIdx.x;
    const long long p = (long long)blockIdx.x * kBlock + t;
    const bool active = p < S.n;
    const long long cap = S.cap;
    if (done) {
        if constexpr (SG == 3)
            if (kout && active) {   // (keys of the unchanged positions)
                Stencil<double> st;
                make_stencil<double>(P, S.pos[0][p], S.pos[1][p], S.pos[2][p], st);
                kout[p] = (unsigned)stencil_key(P, st.b);
                iout[p] = (unsigned)p;
            }
        if constexpr (SC) {
            grid_dep_wait();
            if (active) {
                const long long q = inv[p];
                sc_static64(S, D, p, q);
                for (int d = 0; d < 3; d++) D.pos[d][q] = S.pos[d][p];
                D.time[q] = S.time[p];
                for (int c = 0; c < 2 * NH; c++) D.f0[c * cap + q] = S.f0[c * cap + p];
            }
        }
        return;
    }
    if (s == 1) record_dt(ctl, dt);

    // prologue: fields that no kernel of this step writes, and the tile's
    // weights
    Stencil<double> st{};
    double x = 0, y = 0, z = 0, v[3] = {0, 0, 0}, vsc = 0;
    int slot = t, key = -1;
    if (active) {
        x = __ldcg(S.pos[0] + p);
        y = __ldcg(S.pos[1] + p);
        z = __ldcg(S.pos[2] + p);
#pragma unroll
        for (int d = 0; d < 3; d++) v[d] = __ldcg(S.vhat[d] + p);
        vsc = __ldcg(S.vscale + p);
        // the slot in key order that the last stage 4 stored for these
        // positions (identity after a load or re-sort)
        if (P.rank_stages) slot = __ldcg(S.rslot + p);
        make_stencil<double>(P, x, y, z, st);
        key = stencil_key(P, st.b);
        if constexpr (SG == 3)
            if (kout) {   // (a re-sort follows the step: its keys)
                double xn[3] = {x, y, z}, tn = 0.0;
                rk4_push64(P, dt, v, xn, tn);
                Stencil<double> sn;
                make_stencil<double>(P, xn[0], xn[1], xn[2], sn);
                kout[p] = (unsigned)stencil_key(P, sn.b);
                iout[p] = (unsigned)p;
            }
    }
    double* const rec = sm.rec + slot * RW;
    write_weights<T, WX, WY, WZ>(P, rec, active, st);
    sm.key[slot] = key;
#pragma unroll
    for (int d = 0; d < 3; d++) sm.v[d * VS + slot] = v[d];
    __syncthreads();
    if (s < 4) run_starts(sm.key, sm.starts);
    prefetch_slices<2 * NH>(S.f0, cap, t);
    grid_dep_wait();
    grid_dep_launch();
    if (SG > 1) prefetch_slices<2 * NH>(S.fs, cap, t);
    if (SG == 4) prefetch_slices<2 * NH>(S.acc, cap, t - 32);
    if (s == 4 && dt_mode == DT_ADVANCE) dt_reduce_comb64<NF>(P, mesh_in, ctl, reduce_blocks(P));
    zero_slice(mesh_zero, P.ncells * T::NCS);
    if constexpr (SG == 2)
        if (m4_full_step(ctl)) zero_slice(full_zero, P.ncells * (8 * NH));
    interp64<NF, T, WX, WY, RW>(P, mesh_in, sm.rec, sm.key, sm.v);
    if (P.rank_stages) __syncthreads();   // (slots of other warps)
    else __syncwarp();
    double hs[NH];
    {
        double u[NV];
#pragma unroll
        for (int j = 0; j < NV; j += 2) {
            const double2 t2 = *reinterpret_cast<const double2*>(rec + WP + j);
            u[j] = t2.x * P.sqrt2GF_inv_vol;
            u[j + 1] = t2.y * P.sqrt2GF_inv_vol;
        }
        C::hermitian(u, hs);
    }
    double xn[3] = {x, y, z};
    if (active) {
        double cc[NH];
        int stt = 0;
        long long qsc = 0;
        if constexpr (SC) qsc = (long long)inv[p];
        const double* __restrict__ f0p = S.f0;
        const double* __restrict__ kp = S.fs;
        const double* __restrict__ accp = S.acc;
        // Y_s = y0 + a_s dt K_{s-1}, Y_{s+1} = y0 + a_{s+1} dt K_s
        const double ain = dt * (SG == 4 ? 1.0 : 0.5), aout = dt * (SG == 3 ? 1.0 : 0.5);
        const double b1 = dt * kRK4B[0], b2 = dt * kRK4B[1];   // (b_4 = b_1, b_3 = b_2)
#pragma unroll
        for (int sp = 0; sp < 2; sp++) {
            double y0[NH], f[NH], K[NH], h[NH], ac[NH], fn[NH];
#pragma unroll
            for (int e = 0; e < NH; e++) {
                const long long o = (sp * NH + e) * cap + p;
                y0[e] = f0p[o];
                f[e] = y0[e];
                if constexpr (SG > 1) {
                    const double k = kp[o];
                    f[e] = __dadd_rn(__dmul_rn(ain, k), y0[e]);
                    if constexpr (SG == 2) ac[e] = __dadd_rn(__dmul_rn(b1, k), y0[e]);
                    if constexpr (SG == 4) ac[e] = __dadd_rn(__dmul_rn(b2, k), accp[o]);
                }
            }
            species_hamiltonian<NF>(P, hs, vsc, sp, h);
            commutator<NF, double>(h, f, K, P.inv_hbar);
            if constexpr (SG < 4) {
#pragma unroll
                for (int e = 0; e < NH; e++) {
                    const long long o = (sp * NH + e) * cap + p;
                    S.fs[o] = K[e];
                    if constexpr (SG == 2) S.acc[o] = __dadd_rn(__dmul_rn(b2, K[e]), ac[e]);
                    fn[e] = __dadd_rn(__dmul_rn(aout, K[e]), y0[e]);
                }
            } else {
#pragma unroll
                for (int e = 0; e < NH; e++) fn[e] = __dadd_rn(__dmul_rn(b1, K[e]), ac[e]);
                stt |= renormalize<NF>(fn, S.Ll[sp][p], P.maxError);
            }
            if constexpr (SG == 4) {
#pragma unroll
                for (int e = 0; e < NH; e++) {
                    if constexpr (SC) D.f0[(sp * NH + e) * cap + qsc] = fn[e];
                    else S.f0[(sp * NH + e) * cap + p] = fn[e];
                }
            }
            if constexpr (!SC) {
                const double Ns = S.Nn[sp][p];
#pragma unroll
                for (int e = 0; e < NH; e++) {
                    const double a = fn[e] * Ns;
                    cc[e] = sp == 0 ? a : (H::is_im(e) ? cc[e] + a : cc[e] - a);
                    if ((SG == 3 || SG == 4) && H::is_diag(e))
                        sm.d[(sp * NF + (e == 0 ? 0 : e == NH - 1 ? NF - 1 : 1)) * VS + slot] = a;
                }
            }
        }
        if constexpr (SG == 4) {
            double tn = S.time[p];
            rk4_push64(P, dt, v, xn, tn);
            if constexpr (SC) {
#pragma unroll
                for (int d = 0; d < 3; d++) D.pos[d][qsc] = xn[d];
                D.time[qsc] = tn;
                sc_static64(S, D, p, qsc);
            } else {
#pragma unroll
                for (int d = 0; d < 3; d++) S.pos[d][p] = xn[d];
                S.time[p] = tn;
            }
            if (stt) report_bad(ctl, stt, S.id[p]);
        }
        if constexpr (!SC && SG < 4) {
            double c[NV];
            C::values(cc, c);
#pragma unroll
            for (int j = 0; j < NV; j += 2) *reinterpret_cast<double2*>(rec + WP + j) = make_double2(c[j], c[j + 1]);
        }
        if constexpr (!SC && SG == 4) {
            // (kept in the diagonal slots' place until the new slots are known)
            C::values(cc, hs);
        }
    }
    if constexpr (SC) return;
    if constexpr (SG == 4) {
        // the deposit at the moved positions: their rank, weights and records
        double dnum[2 * NF];
#pragma unroll
        for (int i = 0; i < 2 * NF; i++) dnum[i] = active ? sm.d[i * VS + slot] : 0.0;
        __syncthreads();
        key = -1;
        if (active) {
            make_stencil<double>(P, xn[0], xn[1], xn[2], st);
            key = stencil_key(P, st.b);
        }
        slot = rank_slots(P, key, sm.rec, sm.rank);
        double* const r4 = sm.rec + slot * RW;
        write_weights<T, WX, WY, WZ>(P, r4, active, st);
        sm.key[slot] = key;
#pragma unroll
        for (int d = 0; d < 3; d++) sm.v[d * VS + slot] = v[d];
#pragma unroll
        for (int i = 0; i < 2 * NF; i++) sm.d[i * VS + slot] = dnum[i];
#pragma unroll
        for (int j = 0; j < NV; j += 2)
            *reinterpret_cast<double2*>(r4 + WP + j) = make_double2(active ? hs[j] : 0.0, active ? hs[j + 1] : 0.0);
        if (active) S.rslot[p] = slot;
        __syncthreads();
        run_starts(sm.key, sm.starts);
    }
    __syncthreads();
    // (the diagonal slots: compute_dt reads M_4's, and M_1's at a run's start)
    if (SG == 3 || (SG == 4 && __ldcg(&ctl->m4_full)))
        deposit_comb64<NF, T, WX, WY, RW, true>(P, mesh_out, sm.rec, sm.key, sm.starts, sm.v, sm.d);
    else
        deposit_comb64<NF, T, WX, WY, RW, false>(P, mesh_out, sm.rec, sm.key, sm.starts, sm.v, sm.d);
}

// the combined deposit of a state that stage 4 has re-sorted (M_1)
template <int NF, int WX, int WY, int WZ, int KS>
__global__ void __launch_bounds__(kBlock, 4)
    k_deposit_comb64(DevParams P, DevState S, double* __restrict__ mesh, const StepCtl* ctl)
{
    using T = Tile64<NF, WX, WY, WZ, KS>;
    using H = Herm<NF>;
    using C = Comb<NF>;
    constexpr int NH = NF * NF, NV = C::NV, WP = T::WP, VS = T::VS, RW = T::template row<NV>();
    extern __shared__ __align__(16) unsigned char tile_smem[];
    Smem64<NF, T, RW> sm(tile_smem);
    const int mode = ctl ? ctl->m4_full : 0;
    const int t = threadIdx.x;
    const long long p = (long long)blockIdx.x * kBlock + t;
    const bool active = p < S.n;
    if (active && ctl) S.rslot[p] = t;   // in cell order: the identity rank
    if (mode == 2) return;        // (the run had ended before this step: the mesh stands)
    Stencil<double> st{};
    int key = -1;
    double* const rec = sm.rec + t * RW;
    if (active) {
        make_stencil<double>(P, S.pos[0][p], S.pos[1][p], S.pos[2][p], st);
        key = stencil_key(P, st.b);
        double cc[NH], c[NV];
#pragma unroll
        for (int sp = 0; sp < 2; sp++) {
            const double Ns = S.Nn[sp][p];
#pragma unroll
            for (int e = 0; e < NH; e++) {
                const double a = S.f0[(sp * NH + e) * S.cap + p] * Ns;
                cc[e] = sp == 0 ? a : (H::is_im(e) ? cc[e] + a : cc[e] - a);
                if (H::is_diag(e)) sm.d[(sp * NF + (e == 0 ? 0 : e == NH - 1 ? NF - 1 : 1)) * VS + t] = a;
            }
        }
        C::values(cc, c);
#pragma unroll
        for (int j = 0; j < NV; j += 2) *reinterpret_cast<double2*>(rec + WP + j) = make_double2(c[j], c[j + 1]);
#pragma unroll
        for (int d = 0; d < 3; d++) sm.v[d * VS + t] = S.vhat[d][p];
    }
    write_weights<T, WX, WY, WZ>(P, rec, active, st);
    sm.key[t] = key;
    __syncthreads();
    run_starts(sm.key, sm.starts);
    __syncthreads();
    if (mode) deposit_comb64<NF, T, WX, WY, RW, true>(P, mesh, sm.rec, sm.key, sm.starts, sm.v, sm.d);
    else deposit_comb64<NF, T, WX, WY, RW, false>(P, mesh, sm.rec, sm.key, sm.starts, sm.v, sm.d);
}

// The full deposit (8 NF^2 values per cell) of state f.  ctl != nullptr: the
// stage-4 mesh between stages 3 and 4 of a step (f = y0, the state Y_4 = y0 +
// dt K_3, K_3 in S.fs), made only on the steps after
// which it can be read (m4_full_step), and the note of which kind of step
// this is (StepCtl::m4_full).  A CTA takes tiles of 128 particles in turn, so
// that a step without it costs one small grid.  (32^3 cells x 96 directions:
// the last step of a call takes 1.2 ms longer than the others' 3.8.)
template <int NF, int WX, int WY, int WZ, int KS>
__global__ void __launch_bounds__(kBlock, 3)
    k_deposit_full64(DevParams P, DevState S, const double* __restrict__ f, double* __restrict__ mesh, StepCtl* ctl)
{
    using T = Tile64<NF, WX, WY, WZ, KS>;
    constexpr int NH = NF * NF, NS = 2 * NH, ND = 8 * NH, WP = T::WP, VS = T::VS, RW = T::template row<NS>();
    extern __shared__ __align__(16) unsigned char tile_smem[];
    Smem64<NF, T, RW> sm(tile_smem);
    double dt = 0.0;
    if (ctl) {
        grid_dep_wait();
        grid_dep_launch();
        dt = ctl->dt;
        const bool done = ctl->done, full = !done && m4_full_step(ctl);
        if (blockIdx.x == 0 && threadIdx.x == 0) ctl->m4_full = done ? 2 : full ? 1 : 0;
        if (!full) return;
    }
    const int t = threadIdx.x, w = t >> 5;
    const long long ntile = (S.n + kBlock - 1) / kBlock;
    for (long long tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
        const long long p = tile * kBlock + t;
        const bool active = p < S.n;
        Stencil<double> st{};
        int key = -1;
        if (active) {
            make_stencil<double>(P, S.pos[0][p], S.pos[1][p], S.pos[2][p], st);
            key = stencil_key(P, st.b);
        }
        const int slot = rank_slots(P, key, sm.rec, sm.rank);
        double* const rec = sm.rec + slot * RW;
        write_weights<T, WX, WY, WZ>(P, rec, active, st);
        sm.key[slot] = key;
#pragma unroll
        for (int d = 0; d < 3; d++) sm.v[d * VS + slot] = active ? S.vhat[d][p] : 0.0;
#pragma unroll
        for (int c = 0; c < NS; c++) {
            double y = 0.0;
            if (active) {
                y = f[c * S.cap + p];
                if (ctl) y = __dadd_rn(__dmul_rn(dt, S.fs[c * S.cap + p]), y);
                y *= S.Nn[c / NH][p];
            }
            rec[WP + c] = y;
        }
        __syncthreads();
        run_starts(sm.key, sm.starts);
        __syncthreads();
        for (int nt = w; nt < NH; nt += 4) {
            auto value = [&](int s, int n) {
                const int q = 8 * nt + (n >> 1) + 4 * (n & 1), d = q / NS;
                const double c = sm.rec[s * RW + WP + q % NS];
                return d == 0 ? c : c * sm.v[(d - 1) * VS + s];
            };
            auto add = [&](int cell, int q, double xx) {
                if (xx != 0.0) atomic_add_mesh(mesh + (long long)cell * ND + 8 * nt + q, xx);
            };
            deposit_runs64<T, WX, WY, RW, false>(P, sm.rec, sm.key, sm.starts, 0, kBlock, value, add, 0, 1, NoVal(),
                                                 NoAdd());
        }
        __syncthreads();
    }
}

template <int NF, class T>
constexpr int full64_smem()
{
    return 8 * (kBlock * T::template row<2 * NF * NF>() + (3 + 2 * NF) * T::VS) + 4 * (2 * kBlock + 8);
}

}  // namespace

// The stencil classes: TSC in three dimensions, in the y-z plane and along z
// with fixed widths (unrolled weights), any other stencil of at most 4 or 12
// cells (all that orders 0 to 2 can give) with widths at run time.
#define EMU_W64_DISPATCH(P, ...)                                                                  \
    do {                                                                                          \
        const int cells_ = (P).w[0] * (P).w[1] * (P).w[2];                                        \
        if ((P).w[0] == 3 && (P).w[1] == 3 && (P).w[2] == 3) {                                    \
            constexpr int WXv = 3, WYv = 3, WZv = 3, KSv = 7;                                     \
            __VA_ARGS__;                                                                          \
        } else if ((P).w[0] == 1 && (P).w[1] == 3 && (P).w[2] == 3) {                             \
            constexpr int WXv = 1, WYv = 3, WZv = 3, KSv = 3;                                     \
            __VA_ARGS__;                                                                          \
        } else if ((P).w[0] == 1 && (P).w[1] == 1 && (P).w[2] == 3) {                             \
            constexpr int WXv = 1, WYv = 1, WZv = 3, KSv = 1;                                     \
            __VA_ARGS__;                                                                          \
        } else if (cells_ <= 4) {                                                                 \
            constexpr int WXv = 0, WYv = 0, WZv = 0, KSv = 1;                                     \
            __VA_ARGS__;                                                                          \
        } else {                                                                                  \
            constexpr int WXv = 0, WYv = 0, WZv = 0, KSv = 3;                                     \
            __VA_ARGS__;                                                                          \
        }                                                                                         \
    } while (0)

template <int NF>
void launch_stage64_t(const DevParams& P, const DevState& S, int s, const double* mesh_in, double* mesh_out,
                      double* mesh_zero, double* full_zero, StepCtl* ctl, int dt_mode, cudaStream_t st,
                      const DevState* D, const unsigned* inv, unsigned* kout, unsigned* iout)
{
    EMU_W64_DISPATCH(P, {
        using T = Tile64<NF, WXv, WYv, WZv, KSv>;
        constexpr int bytes = stage64_smem<NF, T>();
        const DevState& Dv = D ? *D : S;
        auto go = [&](auto kern) {
            smem_optin(kern, bytes);
            launch_pdl(kern, grid_for(S.n), kBlock, bytes, st, P, S, mesh_in, mesh_out, mesh_zero, full_zero, ctl,
                       dt_mode, Dv, inv, kout, iout);
        };
        if (s == 1) go(k_stage64<NF, WXv, WYv, WZv, KSv, 1, false>);
        else if (s == 2) go(k_stage64<NF, WXv, WYv, WZv, KSv, 2, false>);
        else if (s == 3) go(k_stage64<NF, WXv, WYv, WZv, KSv, 3, false>);
        else if (D) go(k_stage64<NF, WXv, WYv, WZv, KSv, 4, true>);
        else go(k_stage64<NF, WXv, WYv, WZv, KSv, 4, false>);
    });
}

template <int NF>
void launch_deposit_comb64_t(const DevParams& P, const DevState& S, double* mesh, const StepCtl* ctl, cudaStream_t st)
{
    EMU_W64_DISPATCH(P, {
        using T = Tile64<NF, WXv, WYv, WZv, KSv>;
        constexpr int bytes = stage64_smem<NF, T>();
        smem_optin(k_deposit_comb64<NF, WXv, WYv, WZv, KSv>, bytes);
        k_deposit_comb64<NF, WXv, WYv, WZv, KSv><<<grid_for(S.n), kBlock, bytes, st>>>(P, S, mesh, ctl);
    });
}

template <int NF>
void launch_deposit_full64_t(const DevParams& P, const DevState& S, const double* f, double* mesh, StepCtl* ctl,
                             cudaStream_t st)
{
    EMU_W64_DISPATCH(P, {
        using T = Tile64<NF, WXv, WYv, WZv, KSv>;
        constexpr int bytes = full64_smem<NF, T>();
        auto kern = k_deposit_full64<NF, WXv, WYv, WZv, KSv>;
        smem_optin(kern, bytes);
        const unsigned grid = (unsigned)std::min<long long>(grid_for(S.n), 148 * 12);
        if (ctl) launch_pdl(kern, grid, kBlock, bytes, st, P, S, f, mesh, ctl);
        else kern<<<grid_for(S.n), kBlock, bytes, st>>>(P, S, f, mesh, (StepCtl*)nullptr);
    });
}

}  // namespace emu
