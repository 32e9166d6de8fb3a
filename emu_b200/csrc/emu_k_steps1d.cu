// emu_k_steps1d.cu -- whole runs of FP64 RK4 steps of small one-dimensional
// problems in one cooperative launch (k_steps_1d).
#include "emu_kernels_impl.cuh"
#include "emu_fp64.cuh"

namespace emu {
namespace {

// ---------------------------------------------------------------------------
// A 1D problem of at most one wave of CTAs (128 particles each) is bound by
// latency: the stage kernels of a graph step took 10-13 us each (2 flavors,
// 128 cells x 80 directions: 40 us per step; 50 cells x 2 beams: 54 us), of
// which the memory traffic accounts for well under 1 us.  Here one launch
// takes all steps up to the next re-sort:
//   - a thread pair per particle (one species each) keeps the RK state, the
//     position and the stencil in registers; nothing but the mesh goes
//     through memory between stages;
//   - the stage mesh holds the combined self-interaction layout (Comb<NF>:
//     all that a stage reads, half the values of the full mesh).  Each CTA
//     copies its window, the cells that its particles touch, to shared
//     memory and interpolates from there;
//   - a warp deposits its 16 particles as a small matrix product on the FP64
//     tensor cores (m8n8k4): window cells x particles times particles x
//     values.  No ranking and no runs of equal stencils are needed, and a
//     particle's weights are the sparse columns of the first factor;
//   - stages are separated by a grid barrier (measured 2350 clocks with the
//     mesh reductions it waits for; a kernel boundary cost about the same,
//     plus the reload of the state);
//   - every CTA reduces compute_dt over the stage-4 mesh by itself, so the
//     step control needs no further exchange.
// ONE: a problem of one CTA (at most kOneCells cells) keeps the meshes in
// shared memory and needs no grid barrier; a warp then owns 8 x 8 tiles of
// the mesh, whose sums are complete without reductions.
// ---------------------------------------------------------------------------
constexpr int kWin = 160;        // cells of a window staged in shared memory
constexpr int kOneCells = 128;

template <int NF>
struct Rec1D {
    // w[3], cells (3 x int16 + pad), v4[4] = (1, vx, vy, vz), c[NV], diag[2 NF]
    static constexpr int NV = Comb<NF>::NV;
    static constexpr int W = 0, CELLS = 3, V = 4, CV = 8, DG = 8 + NV;
    // (row lengths that put four particles' words into different banks)
    static constexpr int RW = NF == 2 ? 18 : 22;
    static constexpr int FW = 2 * NF * NF + 1;   // f N of both species (full deposit)
    static_assert(DG + 2 * NF <= RW, "record");
};

template <int NF, bool ONE>
constexpr int steps1d_smem()
{
    using R = Rec1D<NF>;
    constexpr int mesh = ONE ? kOneCells * (2 * Comb<NF>::NG + kDiagSlots) : kWin * Comb<NF>::NG;
    return 8 * (mesh + kBlock * (R::RW + R::FW));
}

// values of a deposit: the combined layout, the diagonal slots, the full one
enum Dep : int { DEP_COMB = 0, DEP_DIAG = 1, DEP_FULL = 2 };
template <int NF, int D>
struct DepN {
    static constexpr int NT = D == DEP_COMB ? Comb<NF>::NG / 8 : D == DEP_DIAG ? 1 : NF * NF;
    static constexpr int STRIDE = D == DEP_FULL ? 8 * NF * NF : kCombSlots<NF>;
    static constexpr int OFF = D == DEP_DIAG ? Comb<NF>::NG : 0;
};
// the value of column n of tile nt for one particle; column n of the product
// is mesh value 8 nt + (n >> 1) + 4 (n & 1), so that the four lanes that hold
// a row's columns 2 i + h write 32 contiguous bytes
template <int NF, int D>
__device__ __forceinline__ double dep_value(const double* rec, const double* fn, int nt, int n)
{
    using R = Rec1D<NF>;
    const int q = 8 * nt + (n >> 1) + 4 * (n & 1);
    if constexpr (D == DEP_COMB) return rec[R::CV + q % R::NV] * rec[R::V + q / R::NV];
    else if constexpr (D == DEP_DIAG) return q < 2 * NF ? rec[R::DG + (q < 2 * NF ? q : 0)] : 0.0;
    else return fn[q % (2 * NF * NF)] * rec[R::V + q / (2 * NF * NF)];
}
__device__ __forceinline__ double dep_weight(const double* rec, int cell)
{
    const int2 c = *reinterpret_cast<const int2*>(rec + 3);
    const int c0 = (short)(c.x & 0xffff), c1 = (short)(c.x >> 16), c2 = (short)(c.y & 0xffff);
    return (c0 == cell ? rec[0] : 0.0) + (c1 == cell ? rec[1] : 0.0) + (c2 == cell ? rec[2] : 0.0);
}

// the warp's own 16 particles (records r0..r0+15) into the global mesh
template <int NF, int D>
__device__ __forceinline__ void deposit_warp(const DevParams& P, double* mesh, const double* srec, const double* sfn,
                                             int r0, int klo, int khi, int c0)
{
    using R = Rec1D<NF>;
    constexpr int NT = DepN<NF, D>::NT;
    const int lane = threadIdx.x & 31, row = lane >> 2, col = lane & 3;
    const int lo = __reduce_min_sync(kFull, klo), hi = __reduce_max_sync(kFull, khi);
    if (hi < 0) return;   // no particle in this warp
    const double* rec[4];
    const double* fn[4];
    int kl[4], kh[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        rec[k] = srec + (r0 + 4 * k + col) * R::RW;
        fn[k] = sfn + (r0 + 4 * k + col) * R::FW;
        kl[k] = __shfl_sync(kFull, klo, 8 * k);
        kh[k] = __shfl_sync(kFull, khi, 8 * k);
    }
    for (int mt = lo >> 3; mt <= hi >> 3; mt++) {
        const int wl = 8 * mt + row;
        // (six tiles at a time: the full layout of three flavors has nine)
        constexpr int G = NT > 5 ? 3 : NT;
#pragma unroll 1
        for (int g = 0; g < NT; g += G) {
            double acc[G][2];
#pragma unroll
            for (int i = 0; i < G; i++) acc[i][0] = acc[i][1] = 0.0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (kh[k] < 8 * mt || kl[k] > 8 * mt + 7) continue;   // (uniform)
                const double a = dep_weight(rec[k], wl);
#pragma unroll
                for (int i = 0; i < G; i++) dmma(acc[i][0], acc[i][1], a, dep_value<NF, D>(rec[k], fn[k], g + i, row));
            }
            int cell = c0 + wl;
            cell = cell % P.n[2];
            if (cell < 0) cell += P.n[2];
            double* m = mesh + (long long)cell * DepN<NF, D>::STRIDE + DepN<NF, D>::OFF;
#pragma unroll
            for (int i = 0; i < G; i++)
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int q = 8 * (g + i) + col + 4 * h;
                    if (acc[i][h] != 0.0) atomic_add_mesh(m + q, acc[i][h]);
                }
        }
    }
}

// ONE: mesh tiles (8 cells x 8 values) summed over all particles by one warp
// each and stored: mesh[cell * stride + q]
template <int NF, int D>
__device__ __forceinline__ void deposit_tiles(int ncells, double* mesh, int stride, const double* srec,
                                              const double* sfn, const int2* krange)
{
    using R = Rec1D<NF>;
    constexpr int NT = DepN<NF, D>::NT;
    const int lane = threadIdx.x & 31, row = lane >> 2, col = lane & 3, w = threadIdx.x >> 5;
    const int nmt = (ncells + 7) >> 3;
    const int2 kr = krange[lane];
    for (int tile = w; tile < nmt * NT; tile += 2 * kBlock / 32) {
        const int mt = tile / NT, nt = tile - mt * NT;
        unsigned todo = __ballot_sync(kFull, kr.y >= 8 * mt && kr.x <= 8 * mt + 7);
        double a0 = 0.0, a1 = 0.0, b0 = 0.0, b1 = 0.0;
        while (todo) {
            const int k = __ffs(todo) - 1;
            todo &= todo - 1;
            const double* r = srec + (4 * k + col) * R::RW;
            dmma(a0, a1, dep_weight(r, 8 * mt + row), dep_value<NF, D>(r, sfn + (4 * k + col) * R::FW, nt, row));
            if (todo) {   // (two chains)
                const int k2 = __ffs(todo) - 1;
                todo &= todo - 1;
                const double* r2 = srec + (4 * k2 + col) * R::RW;
                dmma(b0, b1, dep_weight(r2, 8 * mt + row), dep_value<NF, D>(r2, sfn + (4 * k2 + col) * R::FW, nt, row));
            }
        }
        const int cell = 8 * mt + row;
        if (cell < ncells) {
            double* m = mesh + cell * stride + 8 * nt + col;
            m[0] = a0 + b0;
            m[4] = a1 + b1;
        }
    }
}

// grid barrier: arrivals counted up from 0 over the launch (the last CTA to
// leave the kernel sets the count back).  The wait is bounded; false: it gave
// up (ST_TIMEOUT is set, the CTA leaves the kernel).
__device__ __forceinline__ bool steps_barrier(StepCtl* ctl, unsigned target)
{
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        int good = 1;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&ctl->bar_count) : "memory");
        unsigned v;
        long long it = 0;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&ctl->bar_count) : "memory");
            if (v >= target) break;
            if (++it > kBarrierSpins) {
                atomicOr(&ctl->status, ST_TIMEOUT);
                good = 0;
                break;
            }
        }
        ok = good;
    }
    __syncthreads();
    return ok != 0;
}

struct Meshes4 {
    double* m[4];   // combined meshes, kCombSlots per cell: M_1, M_2, M_3, M_4
};

template <int NF, bool ONE>
__global__ void __launch_bounds__(2 * kBlock, ONE ? 1 : 2)
    k_steps_1d(DevParams P, DevState S, Meshes4 M, double* __restrict__ full, StepCtl* ctl, int nsteps, int dt_mode)
{
    using H = Herm<NF>;
    using C = Comb<NF>;
    using R = Rec1D<NF>;
    constexpr int NH = NF * NF, NV = C::NV, NG = C::NG, NCS = kCombSlots<NF>, ND = 8 * NH, HV = NV / 2;
    extern __shared__ __align__(16) double smem[];
    double* const smesh = smem;                                              // ONE: [2][cells][NG], [cells][8]
    double* const srec = smem + (ONE ? kOneCells * (2 * NG + kDiagSlots) : kWin * NG);
    double* const sfn = srec + kBlock * R::RW;
    double* const sdiag = smesh + 2 * kOneCells * NG;                        // (ONE)
    __shared__ int2 krange[32];
    __shared__ int swin[2][8];
    __shared__ double sred[8];
    __shared__ int sref;

    if (ctl->done) return;
    double t_run = ctl->t, dt = ctl->dt;
    const double end_time = ctl->end_time;
    int step = ctl->step, last = ctl->last, done = 0, st_dt = 0;
    const int max_step = ctl->max_step, full_from = ctl->m4_full_from;
    double* const hist = ctl->dt_hist;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int pl = tid >> 1, sp = tid & 1;
    const long long p = (long long)blockIdx.x * kBlock + pl;
    const bool active = p < S.n;
    const long long cap = S.cap;
    const int nz = P.n[2], ncells = (int)P.ncells;
    const int nthreads = gridDim.x * blockDim.x, gtid = blockIdx.x * blockDim.x + tid;

    // the particle (both threads of its pair), this thread's species
    double x = 0, y = 0, z = 0, tp = 0, v[3] = {0, 0, 0}, vs = 0, Ns = 0, Ls = 1;
    double y0[NH] = {}, acc[NH] = {}, f[NH] = {};
    if (active) {
        x = S.pos[0][p];
        y = S.pos[1][p];
        z = S.pos[2][p];
        tp = S.time[p];
#pragma unroll
        for (int d = 0; d < 3; d++) v[d] = S.vhat[d][p];
        vs = S.vscale[p];
        Ns = S.Nn[sp][p];
        Ls = S.Ll[sp][p];
#pragma unroll
        for (int e = 0; e < NH; e++) f[e] = y0[e] = S.f0[(sp * NH + e) * cap + p];
    }
    double* const rec = srec + pl * R::RW;
    if (sp == 0) {
        rec[R::V] = active ? 1.0 : 0.0;
#pragma unroll
        for (int d = 0; d < 3; d++) rec[R::V + 1 + d] = v[d];
    }
    if constexpr (ONE) {
        for (int i = tid; i < ncells * NG; i += blockDim.x)
            smesh[i] = M.m[0][(long long)(i / NG) * NCS + i % NG];
    }
    int c0 = 0, win = 0;        // window: cells c0 .. c0 + win - 1 (wrapped)
    bool wide = false;          // the window exceeds the staging area
    int ci[3] = {0, 0, 0};      // stencil cells (window index; wide, ONE: cell)
    double wz[3] = {0, 0, 0};
    int klo = 0, khi = -1;      // cells that this lane group's four particles touch
    unsigned nbar = 0;
    int cur = 0;                // ONE: which half of smesh holds the stage mesh

    // stencil, window and the weight part of the record, at the position z
    auto locate = [&]() {
        int first = 0;
        if (active) {
            shape<double>(z * P.dxi[2], P.ord[2], first, wz);
            first = wrapi(first, nz);
        }
        if constexpr (!ONE) {
            if (tid == 0) sref = first;   // (thread 0's particle exists)
            __syncthreads();
            // cells relative to the first particle's, in [-nz/2, nz/2)
            const int half = nz >> 1;
            int r = first - sref + half;
            if (r < 0) r += nz;
            if (r >= nz) r -= nz;
            r -= half;
            const int mn = __reduce_min_sync(kFull, active ? r : INT_MAX);
            const int mx = __reduce_max_sync(kFull, active ? r : INT_MIN);
            if (lane == 0) { swin[0][warp] = mn; swin[1][warp] = mx; }
            __syncthreads();
            int lo = swin[0][0], hi = swin[1][0];
#pragma unroll
            for (int w = 1; w < 8; w++) {
                lo = min(lo, swin[0][w]);
                hi = max(hi, swin[1][w]);
            }
            c0 = sref + lo;
            if (c0 < 0) c0 += nz;
            if (c0 >= nz) c0 -= nz;
            win = hi - lo + P.w[2];
            wide = win > kWin;
            ci[0] = wide ? first : r - lo;
        } else {
            ci[0] = first;
        }
#pragma unroll
        for (int i = 1; i < 3; i++) {
            int c = ci[0] + i;
            if (ONE || wide) c = c >= nz ? c % nz : c;
            ci[i] = i < P.w[2] ? c : ci[0];
        }
        // the range of each group of four particles (eight lanes)
        int a = min(ci[0], min(ci[1], ci[2])), b = max(ci[0], max(ci[1], ci[2]));
        if (!active) { a = INT_MAX; b = -1; }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            a = min(a, __shfl_xor_sync(kFull, a, o));
            b = max(b, __shfl_xor_sync(kFull, b, o));
        }
        klo = a;
        khi = b;
        if constexpr (ONE) {
            if ((lane & 7) == 0) krange[tid >> 3] = make_int2(a, b);
        }
        if (sp == 0) {
#pragma unroll
            for (int i = 0; i < 3; i++) rec[R::W + i] = wz[i];
            *reinterpret_cast<int2*>(rec + R::CELLS) =
                make_int2((ci[0] & 0xffff) | (ci[1] << 16), ci[2] & 0xffff);
        }
    };
    locate();
    bool alive = true;

    for (int it = 0; it < nsteps && alive; it++) {
        if (hist && gtid == 0) hist[step] = dt;
        const bool want_full = step >= full_from || last || step + 1 >= max_step;
        const bool final_step = it + 1 == nsteps;   // (or the run ends: see below)
        double dt_next = dt, t_next = t_run;
        int last_next = last, step_next = step;
#pragma unroll 1
        for (int s = 1; s <= 4; s++) {
            double* const min_ = M.m[s - 1];
            double* const mout = M.m[s & 3];
            const double* mrow = smesh;
            if constexpr (!ONE) {
                // the mesh deposited two stages on, and the full mesh
                double* mz = M.m[(s + 1) & 3];
                for (int i = gtid; i < ncells * NCS; i += nthreads) mz[i] = 0.0;
                if (s == 1 && want_full)
                    for (int i = gtid; i < ncells * ND; i += nthreads) full[i] = 0.0;
                if (!wide) {
                    for (int i = tid; i < win * (NG / 2); i += blockDim.x) {
                        int c = c0 + i / (NG / 2);
                        c = c >= nz ? c % nz : c;
                        reinterpret_cast<double2*>(smesh)[i] =
                            __ldcg(reinterpret_cast<const double2*>(min_ + (long long)c * NCS) + i % (NG / 2));
                    }
                }
            } else {
                mrow = smesh + cur * kOneCells * NG;
            }
            if (s == 4 && dt_mode == DT_ADVANCE) {
                // compute_dt on the stage-4 mesh (Evolve.cpp:22-89 with
                // max_adaptive_speedup <= 1: V_stupid of the diagonal)
                double vm = 0.0;
                if (P.flavor_cfl_factor > 0.0)
                    for (int c = tid; c < ncells; c += blockDim.x) {
                        const double* dg = ONE ? sdiag + c * kDiagSlots : min_ + (long long)c * NCS + NG;
#pragma unroll
                        for (int i = 0; i < 2 * NF; i++) vm = fmax(vm, ONE ? dg[i] : __ldcg(dg + i));
                    }
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1) vm = fmax(vm, __shfl_xor_sync(kFull, vm, o));
                if (lane == 0) sred[warp] = vm;
            }
            __syncthreads();
            if (s == 4 && dt_mode == DT_ADVANCE) {
                double vm = sred[0];
#pragma unroll
                for (int w = 1; w < 8; w++) vm = fmax(vm, sred[w]);
                dt_next = next_dt_stupid<NF>(P, vm, st_dt);
                t_next = t_run + dt;
                step_next = step + 1;
                if (last || step_next >= max_step) done = 1;
                if (end_time - t_next < dt_next) {
                    dt_next = end_time - t_next;
                    last_next = 1;
                }
                if (st_dt) done = 1;
            }
            // interpolation: this thread's half of the NV values
            double u[HV];
#pragma unroll
            for (int j = 0; j < HV; j++) u[j] = 0.0;
            if (active) {
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    double g[4][HV];
                    if (!ONE && wide) {
#pragma unroll
                        for (int d = 0; d < 4; d++)
#pragma unroll
                            for (int j = 0; j < HV; j++)
                                g[d][j] = __ldcg(min_ + (long long)ci[i] * NCS + d * NV + sp * HV + j);
                    } else {
#pragma unroll
                        for (int d = 0; d < 4; d++)
#pragma unroll
                            for (int j = 0; j < HV; j += 2) {
                                const double2 t2 = *reinterpret_cast<const double2*>(mrow + ci[i] * NG + d * NV +
                                                                                     sp * HV + j);
                                g[d][j] = t2.x;
                                g[d][j + 1] = t2.y;
                            }
                    }
#pragma unroll
                    for (int j = 0; j < HV; j++) {
                        const double a = ((g[0][j] - g[1][j] * v[0]) - g[2][j] * v[1]) - g[3][j] * v[2];
                        u[j] += wz[i] * a;
                    }
                }
            }
            double hv[NV];
#pragma unroll
            for (int j = 0; j < HV; j++) {
                const double own = u[j] * P.sqrt2GF_inv_vol, other = __shfl_xor_sync(kFull, own, 1);
                hv[j] = sp == 0 ? own : other;
                hv[HV + j] = sp == 0 ? other : own;
            }
            double h[NH], K[NH];
            C::hermitian(hv, h);
            species_hamiltonian<NF>(P, h, vs, sp, h);
            commutator_lean<NF, double>(h, f, K, P.inv_hbar);
            const double bw = dt * (s == 1 || s == 4 ? 1. / 6. : 1. / 3.);
            if (s < 4) {
                const double aw = dt * (s == 3 ? 1.0 : 0.5);
#pragma unroll
                for (int e = 0; e < NH; e++) {
                    acc[e] = __dadd_rn(__dmul_rn(bw, K[e]), s == 1 ? y0[e] : acc[e]);
                    f[e] = __dadd_rn(__dmul_rn(aw, K[e]), y0[e]);
                }
            } else {
#pragma unroll
                for (int e = 0; e < NH; e++) f[e] = __dadd_rn(__dmul_rn(bw, K[e]), acc[e]);
                if (active) {
                    const int stt = renormalize<NF>(f, Ls, P.maxError);
                    if (stt) report_bad(ctl, stt, S.id[p]);
                    // (the reference's order: four contributions per step)
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const double w = dt * kRK4B[i];
                        x = __dadd_rn(__dmul_rn(w, v[0] * kC), x);
                        y = __dadd_rn(__dmul_rn(w, v[1] * kC), y);
                        z = __dadd_rn(__dmul_rn(w, v[2] * kC), z);
                        tp = __dadd_rn(w, tp);
                    }
                    x = wrap_coord(x, P.L[0]);
                    y = wrap_coord(y, P.L[1]);
                    z = wrap_coord(z, P.L[2]);
                }
#pragma unroll
                for (int e = 0; e < NH; e++) y0[e] = f[e];
                __syncthreads();   // (every thread has read this stage's window)
                locate();
            }
            // the record: the NV combined values (each thread of the pair
            // half of them), and the species' diagonal and f N where wanted
            double fN[NH], fo[NH], cc[NH], cv[NV];
#pragma unroll
            for (int e = 0; e < NH; e++) {
                fN[e] = f[e] * Ns;
                fo[e] = __shfl_xor_sync(kFull, fN[e], 1);
            }
#pragma unroll
            for (int e = 0; e < NH; e++) {
                const double a = sp == 0 ? fN[e] : fo[e], b = sp == 0 ? fo[e] : fN[e];
                cc[e] = H::is_im(e) ? a + b : a - b;
            }
            C::values(cc, cv);
#pragma unroll
            for (int j = 0; j < HV; j++) rec[R::CV + sp * HV + j] = sp == 0 ? cv[j] : cv[HV + j];
            const bool diag = s == 3 || s == 4;
            const bool fdep = s == 3 && want_full;
            if (diag) {
#pragma unroll
                for (int i = 0; i < NF; i++) rec[R::DG + sp * NF + i] = fN[H::re(i, i)];
            }
            if (fdep) {
#pragma unroll
                for (int e = 0; e < NH; e++) sfn[pl * R::FW + sp * NH + e] = fN[e];
            }
            if constexpr (ONE) {
                __syncthreads();
                double* const out = smesh + (1 - cur) * kOneCells * NG;
                deposit_tiles<NF, DEP_COMB>(ncells, out, NG, srec, sfn, krange);
                if (diag) deposit_tiles<NF, DEP_DIAG>(ncells, sdiag, kDiagSlots, srec, sfn, krange);
                if (fdep) deposit_tiles<NF, DEP_FULL>(ncells, full, ND, srec, sfn, krange);
                cur = 1 - cur;
                // (the barrier at the head of the next stage follows)
            } else if (!wide) {
                __syncwarp();   // (a warp reads only its own records)
                const int r0 = warp * 16;
                deposit_warp<NF, DEP_COMB>(P, mout, srec, sfn, r0, klo, khi, c0);
                if (diag) deposit_warp<NF, DEP_DIAG>(P, mout, srec, sfn, r0, klo, khi, c0);
                if (fdep) deposit_warp<NF, DEP_FULL>(P, full, srec, sfn, r0, klo, khi, c0);
            } else if (active) {
#pragma unroll 1
                for (int i = 0; i < P.w[2]; i++) {
                    double* m = mout + (long long)ci[i] * NCS;
#pragma unroll
                    for (int d = 0; d < 4; d++) {
                        const double wd = d == 0 ? wz[i] : wz[i] * v[d - 1];
#pragma unroll
                        for (int j = 0; j < HV; j++)
                            atomic_add_mesh(m + d * NV + sp * HV + j, wd * (sp == 0 ? cv[j] : cv[HV + j]));
                        if (fdep) {
#pragma unroll
                            for (int e = 0; e < NH; e++)
                                atomic_add_mesh(full + (long long)ci[i] * ND + (2 * d + sp) * NH + e, wd * fN[e]);
                        }
                    }
                    if (diag) {
#pragma unroll
                        for (int k = 0; k < NF; k++)
                            atomic_add_mesh(m + NG + sp * NF + k, wz[i] * fN[H::re(k, k)]);
                    }
                }
            }
            if constexpr (ONE) __syncthreads();
            else if (!(s == 4 && (final_step || done))) {
                nbar++;
                if (!steps_barrier(ctl, nbar * gridDim.x)) {
                    alive = false;
                    break;
                }
            }
        }
        t_run = t_next;
        step = step_next;
        dt = dt_next;
        last = last_next;
        if (done) break;
    }
    if (!alive) return;

    if (active) {
#pragma unroll
        for (int e = 0; e < NH; e++) S.f0[(sp * NH + e) * cap + p] = y0[e];
        if (sp == 0) {
            S.pos[0][p] = x;
            S.pos[1][p] = y;
            S.pos[2][p] = z;
            S.time[p] = tp;
        }
    }
    if constexpr (ONE) {
        // the new state's mesh and a clean next one, as a step leaves them
        for (int i = tid; i < ncells * NCS; i += blockDim.x) {
            const int c = i / NCS, q = i - c * NCS;
            M.m[0][i] = q < NG ? smesh[cur * kOneCells * NG + c * NG + q] : sdiag[c * kDiagSlots + q - NG];
            M.m[1][i] = 0.0;
        }
    }
    // the last CTA to leave writes the step control (all hold the same)
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1) {
            __threadfence();
            ctl->blocks_done = 0u;
            ctl->bar_count = 0u;
            if (dt_mode == DT_ADVANCE) {
                ctl->t = t_run;
                ctl->dt = dt;
                ctl->step = step;
                ctl->last = last;
                ctl->done = done;
                if (st_dt) atomicOr(&ctl->status, ST_DT);
            }
        }
    }
}

template <int NF, bool ONE>
bool fits(long long n)
{
    auto kern = k_steps_1d<NF, ONE>;
    constexpr int bytes = steps1d_smem<NF, ONE>();
    smem_optin(kern, bytes);
    int per_sm = 0, dev = 0, nsm = 0;
    const bool ok = cudaGetDevice(&dev) == cudaSuccess &&
                    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 2 * kBlock, bytes) == cudaSuccess &&
                    (long long)per_sm * nsm >= (long long)grid_for(n);
    cudaGetLastError();
    return ok;
}

template <int NF, bool ONE>
cudaError_t launch(const DevParams& P, const DevState& S, double* const cmesh[4], double* full, StepCtl* ctl,
                   int nsteps, int dt_mode, cudaStream_t st)
{
    constexpr int bytes = steps1d_smem<NF, ONE>();
    smem_optin(k_steps_1d<NF, ONE>, bytes);
    DevParams Pc = P;
    DevState Sc = S;
    Meshes4 M{{cmesh[0], cmesh[1], cmesh[2], cmesh[3]}};
    void* args[] = {&Pc, &Sc, &M, &full, &ctl, &nsteps, &dt_mode};
    return cudaLaunchCooperativeKernel((const void*)k_steps_1d<NF, ONE>, dim3(grid_for(S.n)), dim3(2 * kBlock), args,
                                       bytes, st);
}

bool one_cta(const DevParams& P, long long n) { return n <= kBlock && P.ncells <= kOneCells; }

}  // namespace

bool steps_1d_fit(int nf, const DevParams& P, long long n)
{
    if (P.n[0] != 1 || P.n[1] != 1 || P.max_adaptive_speedup > 1.0) return false;
    if (P.ncells > (1 << 20)) return false;   // (mesh indices are ints)
    if (one_cta(P, n)) return nf == 2 ? fits<2, true>(n) : fits<3, true>(n);
    return nf == 2 ? fits<2, false>(n) : fits<3, false>(n);
}

cudaError_t launch_steps_1d(int nf, const DevParams& P, const DevState& S, double* const cmesh[4], double* full,
                            StepCtl* ctl, int nsteps, int dt_mode, cudaStream_t st)
{
    if (one_cta(P, S.n))
        return nf == 2 ? launch<2, true>(P, S, cmesh, full, ctl, nsteps, dt_mode, st)
                       : launch<3, true>(P, S, cmesh, full, ctl, nsteps, dt_mode, st);
    return nf == 2 ? launch<2, false>(P, S, cmesh, full, ctl, nsteps, dt_mode, st)
                   : launch<3, false>(P, S, cmesh, full, ctl, nsteps, dt_mode, st);
}

}  // namespace emu
