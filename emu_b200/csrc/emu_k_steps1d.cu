// emu_k_steps1d.cu -- whole runs of FP64 RK4 steps of small one-dimensional
// problems in one cooperative launch (k_steps_1d).
#include "emu_adjoint.cuh"
#include "emu_fp64.cuh"
#include "emu_kernels_impl.cuh"
#include "emu_window.h"

namespace emu {
namespace {

// ---------------------------------------------------------------------------
// A 1D problem of at most one CTA per SM is bound by latency: the stage
// kernels of a graph step took 10-13 us each (2 flavors, 128 cells x 80
// directions: 40 us per step; 50 cells x 2 beams: 54 us), of which the memory
// traffic accounts for well under 1 us.  Here one launch takes all steps up
// to the next re-sort:
//   - a thread pair per particle (one species each) keeps the RK state, the
//     position and the stencil in registers; nothing but the mesh goes
//     through memory between stages.  The particles are spread evenly over
//     the SMs (a multiple of 16 per CTA);
//   - the stage mesh holds the combined self-interaction layout (Comb<NF>:
//     all that a stage reads, half the values of the full mesh).  Each CTA
//     copies its window, the cells that its particles touch, to shared
//     memory;
//   - a warp interpolates and deposits its 16 particles as small matrix
//     products on the FP64 tensor cores (m8n8k4): particles x cells times
//     cells x values, and the transpose.  No ranking and no runs of equal
//     stencils are needed, the weights are the sparse first factors, kept in
//     registers for the four stages of a step.  (With scalar interpolation
//     and the weights looked up per stage: 20.5 against 14.4 us per step for
//     the two-flavor run above, 38 against 24 us for 256 cells x 92
//     directions of three flavors.)
//   - stages are separated by a grid barrier (measured 2350 clocks with the
//     mesh reductions it waits for; a kernel boundary cost about the same,
//     plus the reload of the state).  What the next stage does not wait for
//     (zeroing) runs between arrival and wait;
//   - compute_dt over the stage-4 mesh: each CTA reduces its share of the
//     cells before it arrives at the step's last barrier (before it leaves, in
//     the last step of a launch).  (Every CTA all of
//     them behind its arrival, as it was: 30,000 particles in 30,000 cells
//     67 against 48 us a step, in 400,000 cells 557 against 136; the same to
//     300 cells.)
// ONE: a problem of one CTA (at most kOneCells cells) keeps the meshes in
// shared memory and needs no grid barrier: each warp leaves the rows of its
// cells in shared memory, and a thread per mesh value adds the rows of its
// cell (50 cells x 2 beams: 15.0 us per step when a warp owned 8 x 8 tiles of
// the mesh and looked for their particles, 11.0 now).
// What is left per stage (two flavors, 128 x 80, of 7200 clocks): the barrier
// about 2500, the window's load after it 900, products and their reductions
// 1200, the FP64 chains of the commutator, the update and Renormalize 1500.
// ---------------------------------------------------------------------------
constexpr int kWin = 160;        // cells of a window staged in shared memory
constexpr int kOneCells = 128;
constexpr int kOnePart = 128;    // particles of a one-CTA problem
constexpr int kNarrow = 16;      // cells of a warp's particles on the matrix path

template <int NF>
struct Rec1D {
    // w[3], 0, v4[4] = (1, vx, vy, vz), c[NV], diag[2 NF], first stencil cell
    // (an int: window index, or a one-CTA problem's cell)
    static constexpr int NV = Comb<NF>::NV, NG = Comb<NF>::NG;
    static constexpr int W = 0, V = 4, CV = 8, DG = 8 + NV, FIRST = DG + 2 * NF;
    // (row lengths that put four particles' words into different banks)
    static constexpr int RW = NF == 2 ? 18 : 26;
    static constexpr int FW = 2 * NF * NF + 1;   // f N of both species (full deposit)
    static constexpr int MR = NG + 4;            // row of a staged mesh
    static_assert(FIRST < RW, "record");
};

template <int NF, bool ONE>
int steps1d_smem(int npart)
{
    using R = Rec1D<NF>;
    const int mesh = ONE ? 2 * kOneCells * R::MR + kOneCells * kDiagSlots + (kOnePart + 1) * kCombSlots<NF>
                         : (kWin + 4) * R::MR;
    return 8 * (mesh + npart * (R::RW + R::FW));
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
// the weight of a particle on window cell `cell` (its stencil starts at its
// first cell; weights past the stencil's width are zero)
template <int NF>
__device__ __forceinline__ double dep_weight(const double* rec, int cell)
{
    const unsigned i = (unsigned)(cell - *reinterpret_cast<const int*>(rec + Rec1D<NF>::FIRST));
    return rec[i < 3u ? i : 3u];
}
// on cell `cell` of nz periodic cells
template <int NF>
__device__ __forceinline__ double dep_weight_periodic(const double* rec, int cell, int nz)
{
    int i = cell - *reinterpret_cast<const int*>(rec + Rec1D<NF>::FIRST);
    if (i < 0) i += nz;
    double w = 0.0;
    for (; i < 3; i += nz) w += rec[i];
    return w;
}

// the warp's own 16 particles (records r0..r0+15) into the global mesh:
// particles spread over any range [lo, hi] of window cells
template <int NF, int D, bool MINUS>
__device__ __noinline__ void deposit_spread(int nz, double* mesh, const double* srec, const double* sfn, int r0,
                                            int lo, int hi, int c0)
{
    using R = Rec1D<NF>;
    constexpr int NT = DepN<NF, D>::NT;
    const int lane = threadIdx.x & 31, row = lane >> 2, col = lane & 3;
    const int ntiles = cell_tiles(lo, hi);
    for (int tile = 0; tile < ntiles; tile++) {
        const int base = lo + 8 * tile;
        double a[4];
        bool any = false;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            a[k] = dep_weight<NF>(srec + (r0 + 4 * k + col) * R::RW, base + row);
            any = any || a[k] != 0.0;
        }
        if (!__any_sync(kFull, any)) continue;
        const int cell = (c0 + base + row) % nz;
        double* m = mesh + (long long)cell * DepN<NF, D>::STRIDE + DepN<NF, D>::OFF;
        for (int nt = 0; nt < NT; nt++) {
            double x = 0.0, y = 0.0;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int i = r0 + 4 * k + col;
                double b = dep_value<NF, D>(srec + i * R::RW, sfn + i * R::FW, nt, row);
                if (MINUS && (8 * nt + (row >> 1) + 4 * (row & 1)) / R::NV > 0) b = -b;
                dmma(x, y, a[k], b);
            }
            if (x != 0.0) atomic_add_mesh(m + 8 * nt + col, x);
            if (y != 0.0) atomic_add_mesh(m + 8 * nt + col + 4, y);
        }
    }
}

// ONE: mesh tiles (8 cells x 8 values) summed over all particles by one warp
// each and stored: mesh[cell * stride + q] (particles in any order; the full
// layout of a run's last step, and warps that are not narrow)
template <int NF, int D>
__device__ __noinline__ void deposit_tiles(int ncells, double* mesh, int stride, const double* srec,
                                           const double* sfn)
{
    using R = Rec1D<NF>;
    constexpr int NT = DepN<NF, D>::NT;
    const int lane = threadIdx.x & 31, row = lane >> 2, col = lane & 3, w = threadIdx.x >> 5;
    const int nmt = (ncells + 7) >> 3, nwarps = blockDim.x >> 5;
    for (int tile = w; tile < nmt * NT; tile += nwarps) {
        const int mt = tile / NT, nt = tile - mt * NT;
        double x = 0.0, y = 0.0;
        for (int k = 0; k < kOnePart / 4; k++) {
            const double* r = srec + (4 * k + col) * R::RW;
            const double a = dep_weight_periodic<NF>(r, 8 * mt + row, ncells);
            if (__any_sync(kFull, a != 0.0))
                dmma(x, y, a, dep_value<NF, D>(r, sfn + (4 * k + col) * R::FW, nt, row));
        }
        const int cell = 8 * mt + row;
        if (cell < ncells) {
            double* m = mesh + cell * stride + 8 * nt + col;
            m[0] = x;
            m[4] = y;
        }
    }
}

// ONE: the same value by value, a thread per mesh value, over the particles
// that touch the cell (CELLS, see k_steps_1d)
template <int NF, int D>
__device__ __noinline__ void deposit_cells(int ncells, double* mesh, int stride, const double* srec, const double* sfn)
{
    using R = Rec1D<NF>;
    constexpr int NQ = 8 * DepN<NF, D>::NT, NS = 2 * NF * NF;
    for (int i = threadIdx.x; i < ncells * NQ; i += blockDim.x) {
        const int c = i / NQ, q = i - c * NQ;
        double sum = 0.0;
        for (int k = 0; k < kOnePart; k++) {
            const double* r = srec + k * R::RW;
            const double w = dep_weight_periodic<NF>(r, c, ncells);
            if (w == 0.0) continue;
            if constexpr (D == DEP_COMB) sum += w * (r[R::CV + q % R::NV] * r[R::V + q / R::NV]);
            else if constexpr (D == DEP_DIAG) sum += w * (q < 2 * NF ? r[R::DG + (q < 2 * NF ? q : 0)] : 0.0);
            else sum += w * (sfn[k * R::FW + q % NS] * r[R::V + q / NS]);
        }
        mesh[c * stride + q] = sum;
    }
}

// Grid barrier in two halves: arrivals counted up from 0 over the launch (the
// last CTA to leave the kernel sets the count back).  The wait is bounded;
// false: it gave up (ST_TIMEOUT is set; steps_gave_up).
__device__ __forceinline__ bool steps_timed_out(const StepCtl* ctl)
{
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(&ctl->status) : "memory");
    return (v & ST_TIMEOUT) != 0;
}
// A CTA leaves after a wait that gave up (thread 0): the last one of all sets
// the counts back for the next launch and ends the run (the launches queued
// behind this one return at once)
__device__ __noinline__ void steps_gave_up(StepCtl* ctl)
{
    __threadfence();
    if (atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1) {
        __threadfence();
        ctl->blocks_done = 0u;
        ctl->bar_count = 0u;
        ctl->vmax_bits[0] = ctl->vmax_bits[1] = 0ull;
        ctl->done = 1;
    }
}
__device__ __forceinline__ void steps_arrive(StepCtl* ctl)
{
    __syncthreads();
    if (threadIdx.x == 0)
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&ctl->bar_count) : "memory");
}
// (A limit that is not a constant in the poll's loop cost 0.05 us a barrier:
// the first polls go without, a limit below them takes the slow loop at once.)
constexpr int kFirstPolls = 1 << 16;
__device__ __noinline__ int steps_wait_slow(StepCtl* ctl, unsigned target, long long polls)
{
    for (long long it = 0;;) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&ctl->bar_count) : "memory");
        if (v >= target) return 1;
        if (++it > polls) {
            atomicOr(&ctl->status, ST_TIMEOUT);
            return 0;
        }
    }
}
__device__ __forceinline__ bool steps_wait(StepCtl* ctl, unsigned target, bool patient, long long polls)
{
    __shared__ int ok;
    if (threadIdx.x == 0) {
        int it = patient ? 0 : kFirstPolls;
        for (; it < kFirstPolls; it++) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&ctl->bar_count) : "memory");
            if (v >= target) break;
        }
        ok = it < kFirstPolls ? 1 : steps_wait_slow(ctl, target, patient ? polls - kFirstPolls : polls);
    }
    __syncthreads();
    return ok != 0;
}

// Where a warp's 16 particles of a 1D problem sit, and the products' weights.
struct Place1D {
    int c0 = 0, win = 0;        // the CTA's window: cells c0 .. c0 + win - 1 (periodic)
    bool wide = false;          // the window exceeds the staging area
    int ci0 = 0;                // first stencil cell (window index; wide, one-CTA problems: the cell)
    double wz[3] = {0, 0, 0};
    int wlo = 0, whi = -1;      // window cells that the warp's particles touch
    bool narrow = false;        // at most kNarrow of them: the matrix path (one CTA: in every warp)
    double ai[2][kNarrow / 4], ad[2][4];   // its weights: interpolation, deposit
    int gcell[2] = {0, 0};      // deposit rows: mesh offset of cell wlo + 8 i + row
};

// r in [-nz/2, nz/2) of cell c relative to cell ref
__device__ __forceinline__ int relative_cell(int c, int ref, int nz)
{
    const int half = nz >> 1;
    int r = c - ref + half;
    if (r < 0) r += nz;
    if (r >= nz) r -= nz;
    return r - half;
}

// the record's weight part and the products' weights; r: the first stencil
// cell in the numbering of wlo, whi
template <int NF>
__device__ __forceinline__ void place_weights(Place1D& L, double* rec, const double* wrec, int sp, int r)
{
    using R = Rec1D<NF>;
    const int lane = threadIdx.x & 31, row = lane >> 2, col = lane & 3;
    if (sp == 0) {
#pragma unroll
        for (int i = 0; i < 3; i++) rec[R::W + i] = L.wz[i];
        *reinterpret_cast<int*>(rec + R::FIRST) = L.narrow ? r : L.ci0;
    }
    __syncwarp();
    if (L.narrow) {
#pragma unroll
        for (int m = 0; m < 2; m++) {
#pragma unroll
            for (int k = 0; k < kNarrow / 4; k++)
                L.ai[m][k] = dep_weight<NF>(wrec + (8 * m + row) * R::RW, L.wlo + 4 * k + col);
#pragma unroll
            for (int k = 0; k < 4; k++)
                L.ad[m][k] = dep_weight<NF>(wrec + (4 * k + col) * R::RW, L.wlo + 8 * m + row);
        }
    }
}

// stencil, window and weights at the position z (barrier inside).  sref: a
// cell near the CTA's particles
template <int NF, bool CELLS>
__device__ __forceinline__ void place_particles(const DevParams& P, Place1D& L, double z, bool active, int sp, int sref,
                                                int (*swin)[16], double* rec, const double* wrec)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5, nz = P.n[2];
    int first = 0;
    if (active) {
        shape<double>(z * P.dxi[2], P.ord[2], first, L.wz);
        first = wrapi(first, nz);
    }
    int r = relative_cell(first, sref, nz);
    const int mn = __reduce_min_sync(kFull, active ? r : INT_MAX);
    const int mx = __reduce_max_sync(kFull, active ? r : INT_MIN);
    if (lane == 0) { swin[0][warp] = mn; swin[1][warp] = mx; }
    __syncthreads();
    const int lo = __reduce_min_sync(kFull, swin[0][lane < nwarps ? lane : 0]);
    const int hi = __reduce_max_sync(kFull, swin[1][lane < nwarps ? lane : 0]);
    L.c0 = sref + lo;
    if (L.c0 < 0) L.c0 += nz;
    if (L.c0 >= nz) L.c0 -= nz;
    L.win = hi - lo + P.w[2];
    L.wide = L.win > kWin;
    r -= lo;
    L.ci0 = L.wide ? first : r;
    const CellRange own = warp_cells(mn, mx, lo, P.w[2]);
    L.wlo = own.lo;
    L.whi = own.hi;
    L.narrow = !CELLS && !L.wide && mx >= mn && L.whi - L.wlo < kNarrow;
    place_weights<NF>(L, rec, wrec, sp, r);
    if (L.narrow) {
#pragma unroll
        for (int m = 0; m < 2; m++) {
            int c = L.c0 + L.wlo + 8 * m + (lane >> 2);
            c = c >= nz ? c % nz : c;
            L.gcell[m] = c * kCombSlots<NF>;
        }
    }
}

// the window of a combined mesh into shared memory (four further rows of
// zeros: the last product's depth)
template <int NF>
__device__ __forceinline__ void stage_window(const Place1D& L, double* smesh, const double* mesh, int nz)
{
    using R = Rec1D<NF>;
    constexpr int NG = R::NG, NCS = kCombSlots<NF>;
    if (L.wide) return;
    for (int i = threadIdx.x; i < (L.win + 4) * (NG / 2); i += blockDim.x) {
        const int wl = i / (NG / 2), q = i - wl * (NG / 2);
        int c = L.c0 + wl;
        c = c >= nz ? c % nz : c;
        double2 t2 = make_double2(0.0, 0.0);
        if (wl < L.win) t2 = __ldcg(reinterpret_cast<const double2*>(mesh + c * NCS) + q);
        *reinterpret_cast<double2*>(smesh + wl * R::MR + 2 * q) = t2;
    }
}

// The interpolated sums u_j = G_0j - v . G_dj (PLUS: + v . G_dj) of the pair's
// particle, both threads.  ONE: mrow holds the whole mesh, mrow_of the rows of
// this lane's cells.
template <int NF, bool ONE, bool PLUS>
__device__ __forceinline__ void interp_1d(const DevParams& P, const Place1D& L, const double* mrow, const int* mrow_of,
                                          const double* mesh, double* rec, double* wrec, int sp, bool active, double* hv)
{
    using R = Rec1D<NF>;
    constexpr int NV = R::NV, NT = R::NG / 8, HV = NV / 2, NCS = kCombSlots<NF>;
    const int lane = threadIdx.x & 31, row = lane >> 2, col = lane & 3, nz = P.n[2];
    const double sg = PLUS ? -1.0 : 1.0;
    if (L.narrow) {
        double g[2][NT][2];
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int nt = 0; nt < NT; nt++) g[m][nt][0] = g[m][nt][1] = 0.0;
#pragma unroll
        for (int k = 0; k < kNarrow / 4; k++) {
            if (L.wlo + 4 * k > L.whi) break;   // (uniform)
            const double* b = mrow + (ONE ? mrow_of[k] : (L.wlo + 4 * k + col) * R::MR);
#pragma unroll
            for (int nt = 0; nt < NT; nt++) {
                // two flavors: column 2 e + i holds d = 2 nt + i of value e, so
                // that a lane's two columns are one value
                const double bv = b[NF == 2 ? (2 * nt + (row & 1)) * NV + (row >> 1) : nt * NV + row];
#pragma unroll
                for (int m = 0; m < 2; m++) dmma(g[m][nt][0], g[m][nt][1], L.ai[m][k], bv);
            }
        }
#pragma unroll
        for (int m = 0; m < 2; m++) {
            double* r = wrec + (8 * m + row) * R::RW;
            const double vx = sg * r[R::V + 1], vy = sg * r[R::V + 2], vz = sg * r[R::V + 3];
            if constexpr (NF == 2) {
                r[R::CV + col] = ((g[m][0][0] - vx * g[m][0][1]) - vy * g[m][1][0]) - vz * g[m][1][1];
            } else {
                double2 t2;
                t2.x = ((g[m][0][0] - vx * g[m][1][0]) - vy * g[m][2][0]) - vz * g[m][3][0];
                t2.y = ((g[m][0][1] - vx * g[m][1][1]) - vy * g[m][2][1]) - vz * g[m][3][1];
                *reinterpret_cast<double2*>(r + R::CV + 2 * col) = t2;
            }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < NV; j += 2) {
            const double2 t2 = *reinterpret_cast<const double2*>(rec + R::CV + j);
            hv[j] = t2.x;
            hv[j + 1] = t2.y;
        }
    } else {
        double u[HV];
#pragma unroll
        for (int j = 0; j < HV; j++) u[j] = 0.0;
        if (active) {
            const double vx = sg * rec[R::V + 1], vy = sg * rec[R::V + 2], vz = sg * rec[R::V + 3];
#pragma unroll 1
            for (int i = 0; i < P.w[2]; i++) {
                int cc = L.ci0 + i;
                if (ONE || L.wide) cc = cc % nz;
                const double wi = i == 0 ? L.wz[0] : i == 1 ? L.wz[1] : L.wz[2];
#pragma unroll
                for (int j = 0; j < HV; j++) {
                    double g[4];
#pragma unroll
                    for (int d = 0; d < 4; d++)
                        g[d] = !ONE && L.wide ? __ldcg(mesh + cc * NCS + d * NV + sp * HV + j)
                                              : mrow[cc * R::MR + d * NV + sp * HV + j];
                    u[j] += wi * (((g[0] - g[1] * vx) - g[2] * vy) - g[3] * vz);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < HV; j++) {
            const double other = __shfl_xor_sync(kFull, u[j], 1);
            hv[j] = sp == 0 ? u[j] : other;
            hv[HV + j] = sp == 0 ? other : u[j];
        }
    }
}

// the products of a narrow warp's deposit, window cells wlo + 8 m + row: g the
// combined values, gd the diagonal ones (diag).  MINUS: fluxes with -v
template <int NF, bool MINUS>
__device__ __forceinline__ void products_1d(const Place1D& L, const double* wrec, int m, bool diag,
                                            double (*g)[2], double* gd)
{
    using R = Rec1D<NF>;
    constexpr int NT = R::NG / 8, NV = R::NV;
    const int lane = threadIdx.x & 31, row = lane >> 2, col = lane & 3, q0 = (row >> 1) + 4 * (row & 1);
#pragma unroll
    for (int nt = 0; nt < NT; nt++) g[nt][0] = g[nt][1] = 0.0;
    gd[0] = gd[1] = 0.0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const double* r = wrec + (4 * k + col) * R::RW;
        const double c = r[R::CV + q0 % NV];
#pragma unroll
        for (int nt = 0; nt < NT; nt++) {
            const int d = (8 * nt + q0) / NV;
            double b = c * r[R::V + d];
            if (MINUS && d > 0) b = -b;
            dmma(g[nt][0], g[nt][1], L.ad[m][k], b);
        }
        if (diag) dmma(gd[0], gd[1], L.ad[m][k], q0 < 2 * NF ? r[R::DG + (q0 < 2 * NF ? q0 : 0)] : 0.0);
    }
}

// the warp's particles into a global combined mesh (not wide)
template <int NF, bool MINUS>
__device__ __forceinline__ void deposit_1d(const Place1D& L, const double* srec, const double* sfn, const double* wrec,
                                           double* mesh, int nz, bool diag)
{
    using R = Rec1D<NF>;
    constexpr int NG = R::NG, NT = NG / 8;
    const int lane = threadIdx.x & 31, row = lane >> 2, col = lane & 3, r0 = (threadIdx.x >> 5) * 16;
    if (L.narrow) {
#pragma unroll
        for (int m = 0; m < 2; m++) {
            if (L.wlo + 8 * m > L.whi) break;   // (uniform)
            double g[NT][2], gd[2];
            products_1d<NF, MINUS>(L, wrec, m, diag, g, gd);
            if (L.wlo + 8 * m + row <= L.whi) {
                double* o = mesh + L.gcell[m] + col;
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
                    atomic_add_mesh(o + 8 * nt, g[nt][0]);
                    atomic_add_mesh(o + 8 * nt + 4, g[nt][1]);
                }
                if (diag) {
                    atomic_add_mesh(o + NG, gd[0]);
                    if (NF == 3 && col < 2) atomic_add_mesh(o + NG + 4, gd[1]);
                }
            }
        }
    } else if (L.whi >= L.wlo) {
        deposit_spread<NF, DEP_COMB, MINUS>(nz, mesh, srec, sfn, r0, L.wlo, L.whi, L.c0);
        if (diag) deposit_spread<NF, DEP_DIAG, false>(nz, mesh, srec, sfn, r0, L.wlo, L.whi, L.c0);
    }
}
// value by value, cells first, first + 1, ..: this thread's half of the pair's
template <int NF, bool MINUS>
__device__ __forceinline__ void deposit_1d_cells(const DevParams& P, const Place1D& L, const double* rec, int sp,
                                                 int first, double* mesh, bool diag)
{
    using R = Rec1D<NF>;
    constexpr int NV = R::NV, HV = NV / 2, NG = R::NG, NCS = kCombSlots<NF>;
#pragma unroll 1
    for (int i = 0; i < P.w[2]; i++) {
        double* m = mesh + (first + i) % P.n[2] * NCS;
        const double wi = i == 0 ? L.wz[0] : i == 1 ? L.wz[1] : L.wz[2];
        for (int d = 0; d < 4; d++) {
            const double wd = MINUS && d > 0 ? -(wi * rec[R::V + d]) : wi * rec[R::V + d];
            for (int j = 0; j < HV; j++) atomic_add_mesh(m + d * NV + sp * HV + j, wd * rec[R::CV + sp * HV + j]);
        }
        if (diag)
            for (int k = 0; k < NF; k++) atomic_add_mesh(m + NG + sp * NF + k, wi * rec[R::DG + sp * NF + k]);
    }
}

// cmesh: four combined meshes (kCombSlots per cell) one after the other, M_1
// to M_4.  npart particles per CTA (a multiple of 16), 2 npart threads.
// REC (not ONE): a recorded run (Rec1DStore): every step's state, stage states
// and meshes are kept, the meshes where they are stored (zeroed; M_1 of the
// first step deposited) instead of in cmesh; the last step's M_1 is not made.
// CELLS: a state with values that are not finite.  The products meet a warp's
// other particles and cells with weight zero, which a finite value passes and
// this would not; these states go cell by cell (scalar interpolation and
// deposits), which takes such a value to the cells of its stencil only.
// (A second body behind one look at ctl->odd: looks at every stage's values,
// with the cell-by-cell code in their shadow, cost 1 to 4 % of a step.)
template <int NF, bool ONE, bool REC, bool CELLS>
__device__ __forceinline__ void steps_1d_body(const DevParams& P, const DevState& S, double* __restrict__ cmesh,
                                              double* __restrict__ full, StepCtl* ctl, int npart, int nsteps,
                                              int dt_mode, const Rec1DStore& store)
{
    using H = Herm<NF>;
    using C = Comb<NF>;
    using R = Rec1D<NF>;
    constexpr int NH = NF * NF, NV = C::NV, NG = C::NG, NCS = kCombSlots<NF>, ND = 8 * NH, HV = NV / 2;
    constexpr int NT = NG / 8, MR = R::MR, KI = kNarrow / 4;
    static_assert(!(ONE && REC), "recorded runs keep global meshes");
    extern __shared__ __align__(16) double smem[];
    double* const smesh = smem;                                  // ONE: two meshes, then the diagonal slots
    constexpr int kHalf = kOneCells * MR;
    double* const sdiag = smesh + 2 * kHalf;                     // (ONE)
    double* const spart = sdiag + kOneCells * kDiagSlots;        // (ONE) 16 rows of a mesh per warp
    double* const srec = ONE ? spart + (kOnePart + 1) * NCS : smesh + (kWin + 4) * MR;
    double* const sfn = srec + npart * R::RW;
    __shared__ int2 srange[2 * kOnePart / 32];                   // (ONE) first cell and cells of each warp
    // (ONE) the rows of spart that hold parts of a cell's sums: their count,
    // the first four (row kOnePart: zeros)
    __shared__ int scount[ONE ? kOneCells : 1];
    __shared__ __align__(4) unsigned char srows[ONE ? kOneCells : 1][4];
    __shared__ int swin[2][16];
    __shared__ double sred[16];
    __shared__ int sref;

    double t_run = ctl->t, dt = ctl->dt;
    const double end_time = ctl->end_time;
    int step = ctl->step, last = ctl->last, done = 0, st_dt = 0;
    const int max_step = ctl->max_step, full_from = ctl->m4_full_from;
    double* const hist = ctl->dt_hist;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int row = lane >> 2, col = lane & 3;
    const int pl = tid >> 1, sp = tid & 1;
    const long long p = (long long)blockIdx.x * npart + pl;
    const bool active = p < S.n;
    const long long cap = S.cap;
    const int nz = P.n[2], ncells = (int)P.ncells;
    const int nthreads = gridDim.x * blockDim.x, gtid = blockIdx.x * blockDim.x + tid;
    const int msize = ncells * NCS;

    // the particle (both threads of its pair), this thread's species
    double x = 0, yy = 0, z = 0, tp = 0, v[3] = {0, 0, 0}, vs = 0, Ns = 0, Ls = 1;
    double y0[NH] = {}, acc[NH] = {}, f[NH] = {};
    if (active) {
        x = S.pos[0][p];
        yy = S.pos[1][p];
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
    double* const wrec = srec + warp * 16 * R::RW;   // the warp's 16 records
    if (sp == 0) {
        rec[3] = 0.0;
        rec[R::V] = 1.0;
#pragma unroll
        for (int d = 0; d < 3; d++) rec[R::V + 1 + d] = v[d];
    }
    if constexpr (ONE) {
        for (int i = tid; i < kHalf; i += blockDim.x) {
            const int c = i / MR, q = i - c * MR;
            if (c < ncells && q < NG) smesh[i] = cmesh[c * NCS + q];
        }
        if (tid < NCS) spart[kOnePart * NCS + tid] = 0.0;
    } else if constexpr (!REC) {
        // (M_2's mesh is clean at a step boundary)
        for (int i = gtid; i < msize; i += nthreads) cmesh[2 * msize + i] = 0.0;
    }
    Place1D L;
    int mrow_of[KI] = {};       // (ONE) mesh rows of the interpolation's cells
    // stencil, window, weights and the weight part of the record, at the
    // position z
    auto locate = [&]() {
        if constexpr (!ONE) {
            // (cells relative to the first particle's at the launch)
            place_particles<NF, CELLS>(P, L, z, active, sp, sref, swin, rec, wrec);
        } else {
            int first = 0;
            if (active) {
                shape<double>(z * P.dxi[2], P.ord[2], first, L.wz);
                first = wrapi(first, nz);
            }
            // relative to the warp's first cell
            const int ref = __shfl_sync(kFull, first, 0);
            int r = relative_cell(first, ref, nz);
            const int mn = __reduce_min_sync(kFull, active ? r : INT_MAX);
            const int mx = __reduce_max_sync(kFull, active ? r : INT_MIN);
            const bool any = __any_sync(kFull, active);
            if (tid < kOneCells) {
                scount[tid] = 0;
                *reinterpret_cast<unsigned*>(srows[tid]) = 0x01010101u * kOnePart;
            }
            L.narrow = __syncthreads_and(!CELLS && (!any || mx - mn + P.w[2] <= kNarrow));
            L.c0 = any ? wrapi(ref + mn, nz) : 0;
            L.wlo = 0;
            L.whi = any ? mx - mn + P.w[2] - 1 : -1;
            L.ci0 = first;
            if (lane == 0) srange[warp] = make_int2(L.c0, L.whi + 1);
            if (L.narrow && lane <= L.whi) {
                const int c = (L.c0 + lane) % nz, k = atomicAdd(&scount[c], 1);
                if (k < 4) srows[c][k] = (unsigned char)(warp * 16 + lane);
            }
#pragma unroll
            for (int k = 0; k < KI; k++) mrow_of[k] = (L.c0 + 4 * k + col) % nz * MR;
            place_weights<NF>(L, rec, wrec, sp, any ? r - mn : 0);
        }
    };
    if constexpr (!ONE) {
        if (tid == 0) {   // (the CTA's first particle exists)
            int first;
            shape<double>(z * P.dxi[2], P.ord[2], first, L.wz);
            sref = wrapi(first, nz);
        }
    }
    __syncthreads();
    locate();
    const double dt_fac = stupid_factor<NF>(P), dt_vmin = P.cell_volume * P.Ye * P.rho / kMp;
    const bool patient = P.wait_polls >= kFirstPolls;
    unsigned nbar = 0;
    int slot = 0;  // of the control's vmax_bits: the step's largest number
    int cur = 0;   // ONE: which half of smesh holds the stage mesh

    for (int it = 0; it < nsteps; it++) {
        if (hist && gtid == 0) hist[step] = dt;
        const bool want_full = step >= full_from || last || step + 1 >= max_step;
        const bool final_step = it + 1 == nsteps;
        double dt_next = dt, t_next = t_run;
        int last_next = last, step_next = step;
#pragma unroll 1
        for (int s = 1; s <= 4; s++) {
            const double* mesh_in = cmesh + (s - 1) * msize;
            double* mesh_out = cmesh + (s & 3) * msize;
            if constexpr (REC) {
                mesh_in = store.mst + it * store.mst_stride + (s - 1) * msize;
                mesh_out = s < 4 ? store.mst + it * store.mst_stride + s * msize : store.mst + (it + 1) * store.mst_stride;
                if (s == 1 && active) {
                    double* y = store.seg + it * store.seg_stride;
#pragma unroll
                    for (int e = 0; e < NH; e++) y[(sp * NH + e) * cap + p] = y0[e];
                    if (sp == 0) {
                        y[(2 * NH) * cap + p] = x;
                        y[(2 * NH + 1) * cap + p] = yy;
                        y[(2 * NH + 2) * cap + p] = z;
                    }
                }
            }
            const double* mrow = smesh;
            if constexpr (!ONE) {
                // M_4's mesh: here, since a CTA may still read the last
                // step's for its timestep until it arrives at barrier 1
                if (!REC && s == 2)
                    for (int i = gtid; i < msize; i += nthreads) cmesh[3 * msize + i] = 0.0;
                stage_window<NF>(L, smesh, mesh_in, nz);
                __syncthreads();
            } else {
                mrow = smesh + cur * kHalf;
            }
            double hv[NV];
            interp_1d<NF, ONE, false>(P, L, mrow, mrow_of, mesh_in, rec, wrec, sp, active, hv);
#pragma unroll
            for (int j = 0; j < NV; j++) hv[j] *= P.sqrt2GF_inv_vol;
            double h[NH], K[NH];
            C::hermitian(hv, h);
            species_hamiltonian<NF>(P, h, vs, sp, h);
            commutator<NF, double>(h, f, K, P.inv_hbar);
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
            }
            if constexpr (REC) {   // Y_2, Y_3, Y_4, Y_n
                if (active) {
                    double* y = store.sst + it * store.sst_stride + (s - 1) * (2 * NH) * cap;
#pragma unroll
                    for (int e = 0; e < NH; e++) y[(sp * NH + e) * cap + p] = f[e];
                }
            }
            if (s == 4) {
                if (active) {
                    const int stt = renormalize<NF>(f, Ls, P.maxError);
                    if (stt) report_bad(ctl, stt, S.id[p]);
                    // (the reference's order: four contributions per step)
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const double w = dt * (i == 0 || i == 3 ? 1. / 6. : 1. / 3.);
                        x = __dadd_rn(__dmul_rn(w, v[0] * kC), x);
                        yy = __dadd_rn(__dmul_rn(w, v[1] * kC), yy);
                        z = __dadd_rn(__dmul_rn(w, v[2] * kC), z);
                        tp = __dadd_rn(w, tp);
                    }
                    x = wrap_coord(x, P.L[0]);
                    yy = wrap_coord(yy, P.L[1]);
                    z = wrap_coord(z, P.L[2]);
                }
#pragma unroll
                for (int e = 0; e < NH; e++) y0[e] = f[e];
                __syncwarp();
                locate();
            }
            // the record: the NV combined values (each thread of the pair
            // half of them), and the species' diagonal and f N where wanted
            const bool diag = s >= 3;
            const bool fdep = s == 3 && want_full;
            {
                double fN[NH], cc[NH], cv[NV];
#pragma unroll
                for (int e = 0; e < NH; e++) fN[e] = f[e] * Ns;
#pragma unroll
                for (int e = 0; e < NH; e++) {
                    const double o = __shfl_xor_sync(kFull, fN[e], 1);
                    cc[e] = H::is_im(e) ? fN[e] + o : (sp == 0 ? fN[e] - o : o - fN[e]);
                }
                C::values(cc, cv);
                __syncwarp();   // (the pair's reads of the interpolated values)
#pragma unroll
                for (int j = 0; j < HV; j++) rec[R::CV + sp * HV + j] = sp == 0 ? cv[j] : cv[HV + j];
                if (diag) {
#pragma unroll
                    for (int i = 0; i < NF; i++) rec[R::DG + sp * NF + i] = fN[H::re(i, i)];
                }
                if (fdep) {
#pragma unroll
                    for (int e = 0; e < NH; e++) sfn[pl * R::FW + sp * NH + e] = fN[e];
                }
            }
            if constexpr (ONE) {
                if (L.narrow) {
                    __syncwarp();   // (a warp reads only its own records)
#pragma unroll
                    for (int m = 0; m < 2; m++) {
                        if (8 * m > L.whi) break;   // (uniform)
                        double g[NT][2], gd[2];
                        products_1d<NF, false>(L, wrec, m, diag, g, gd);
                        // the warp's rows, summed over the warps below
                        double* o = spart + (warp * 16 + 8 * m + row) * NCS + col;
#pragma unroll
                        for (int nt = 0; nt < NT; nt++) {
                            o[8 * nt] = g[nt][0];
                            o[8 * nt + 4] = g[nt][1];
                        }
                        if (diag) {
                            o[NG] = gd[0];
                            o[NG + 4] = gd[1];
                        }
                    }
                }
            }
            if constexpr (ONE) {
                double* const out = smesh + (1 - cur) * kHalf;
                __syncthreads();
                if (L.narrow) {
                    const int nq = diag ? NCS : NG;
                    for (int i = tid; i < ncells * nq; i += blockDim.x) {
                        const int c = diag ? i / NCS : i / NG, q = i - c * nq;
                        const uchar4 r4 = *reinterpret_cast<const uchar4*>(srows[c]);
                        double t2 = (spart[r4.x * NCS + q] + spart[r4.y * NCS + q]) +
                                    (spart[r4.z * NCS + q] + spart[r4.w * NCS + q]);
                        if (scount[c] > 4) {
                            t2 = 0.0;
                            for (int w = 0; w < 2 * kOnePart / 32; w++) {
                                const int2 rg = srange[w];
                                int k = c - rg.x;
                                if (k < 0) k += nz;
                                for (; k < rg.y; k += nz) t2 += spart[(w * 16 + k) * NCS + q];
                            }
                        }
                        if (q < NG) out[c * MR + q] = t2;
                        else sdiag[c * kDiagSlots + q - NG] = t2;
                    }
                } else if constexpr (CELLS) {
                    deposit_cells<NF, DEP_COMB>(ncells, out, MR, srec, sfn);
                    if (diag) deposit_cells<NF, DEP_DIAG>(ncells, sdiag, kDiagSlots, srec, sfn);
                    if (fdep) deposit_cells<NF, DEP_FULL>(ncells, full, ND, srec, sfn);
                } else {
                    deposit_tiles<NF, DEP_COMB>(ncells, out, MR, srec, sfn);
                    if (diag) deposit_tiles<NF, DEP_DIAG>(ncells, sdiag, kDiagSlots, srec, sfn);
                }
                if (!CELLS && fdep) {
                    // (cells in place of rows relative to the warp's first)
                    if (L.narrow) {
                        __syncthreads();
                        if (sp == 0) *reinterpret_cast<int*>(rec + R::FIRST) = L.ci0;
                        __syncthreads();
                    }
                    deposit_tiles<NF, DEP_FULL>(ncells, full, ND, srec, sfn);
                }
                cur = 1 - cur;
                if (s == 3 && dt_mode == DT_ADVANCE) {
                    // the largest diagonal number, for the next step's dt
                    __syncthreads();
                    double vm = 0.0;
                    for (int i = tid; i < ncells * 2 * NF; i += blockDim.x)
                        vm = fmax(vm, sdiag[i / (2 * NF) * kDiagSlots + i % (2 * NF)]);
#pragma unroll
                    for (int o = 16; o >= 1; o >>= 1) vm = fmax(vm, __shfl_xor_sync(kFull, vm, o));
                    if (lane == 0) sred[warp] = vm;
                }
                __syncthreads();
            } else {
                if (!(REC && s == 4 && final_step)) {
                    __syncwarp();   // (a warp reads only its own records)
                    if (!CELLS && !L.wide) {
                        deposit_1d<NF, false>(L, srec, sfn, wrec, mesh_out, nz, diag);
                        if (fdep && L.whi >= L.wlo)
                            deposit_spread<NF, DEP_FULL, false>(nz, full, srec, sfn, warp * 16, L.wlo, L.whi, L.c0);
                    } else if (active) {
                        const int first = CELLS && !L.wide ? L.c0 + L.ci0 : L.ci0;
                        deposit_1d_cells<NF, false>(P, L, rec, sp, first, mesh_out, diag);
                        if (fdep) {
#pragma unroll 1
                            for (int i = 0; i < P.w[2]; i++) {
                                double* m = full + (long long)((first + i) % nz) * ND;
                                const double wi = i == 0 ? L.wz[0] : i == 1 ? L.wz[1] : L.wz[2];
                                for (int d = 0; d < 4; d++)
                                    for (int e = 0; e < NH; e++)
                                        atomic_add_mesh(m + (2 * d + sp) * NH + e,
                                                        wi * rec[R::V + d] * sfn[pl * R::FW + sp * NH + e]);
                            }
                        }
                    }
                }
                // compute_dt on the stage-4 mesh (Evolve.cpp:22-89 with
                // max_adaptive_speedup <= 1: V_stupid of the diagonal): the
                // CTA's share of the cells, the largest over all behind the
                // barrier
                if (s == 4 && dt_mode == DT_ADVANCE) {
                    double vm = 0.0;
                    for (int i = gtid; i < ncells * NF; i += nthreads) {
                        const double2 t2 = __ldcg(reinterpret_cast<const double2*>(mesh_in + i / NF * NCS + NG) + i % NF);
                        vm = fmax(vm, fmax(t2.x, t2.y));
                    }
#pragma unroll
                    for (int o = 16; o >= 1; o >>= 1) vm = fmax(vm, __shfl_xor_sync(kFull, vm, o));
                    if (lane == 0) sred[warp] = vm;
                    __syncthreads();
                    if (tid == 0) {
                        for (int w = 1; w < nwarps; w++) vm = fmax(vm, sred[w]);
                        atomicMax(&ctl->vmax_bits[it & 1], (unsigned long long)__double_as_longlong(vm));
                    }
                }
                // (the launch's last step ends without a barrier: the last CTA to
                // leave finds the next timestep)
                const bool wait = s < 4 || !(final_step || (dt_mode == DT_ADVANCE && (last || step + 1 >= max_step)));
                if (wait) steps_arrive(ctl);
                // the mesh deposited two stages on (its last readers are past
                // the previous barrier)
                {
                    double* mz = cmesh + ((s + 2) & 3) * msize;
                    if (!REC && (s == 2 || s == 3 || (s == 4 && wait)))
                        for (int i = gtid; i < msize; i += nthreads) mz[i] = 0.0;
                    if (s == 1 && want_full)
                        for (int i = gtid; i < ncells * ND; i += nthreads) full[i] = 0.0;
                }
                if (wait) {
                    nbar++;
                    if (!steps_wait(ctl, nbar * gridDim.x, patient, P.wait_polls)) {
                        if (tid == 0) steps_gave_up(ctl);
                        return;
                    }
                }
                if (s == 4 && dt_mode == DT_ADVANCE) {
                    slot = it & 1;
                    dt_next = -INFINITY;
                    if (wait) {
                        const double vm = __longlong_as_double((long long)__ldcg(&ctl->vmax_bits[slot]));
                        dt_next = next_dt_stupid(P, fmax(P.flavor_cfl_factor > 0.0 ? vm : 0.0, dt_vmin), dt_fac, st_dt);
                    }
                } else if (s == 2 && gtid == 0) {
                    ctl->vmax_bits[(it + 1) & 1] = 0ull;   // (every CTA has read the last step's)
                }
            }
            if (s == 4 && dt_mode == DT_ADVANCE) {
                if constexpr (ONE) {
                    double vm = sred[0];
                    for (int w = 1; w < nwarps; w++) vm = fmax(vm, sred[w]);
                    dt_next = next_dt_stupid(P, fmax(P.flavor_cfl_factor > 0.0 ? vm : 0.0, dt_vmin), dt_fac, st_dt);
                }
                t_next = t_run + dt;
                step_next = step + 1;
                if (last || step_next >= max_step) done = 1;
                if (end_time - t_next < dt_next) {
                    dt_next = end_time - t_next;
                    last_next = 1;
                }
                if (st_dt) done = 1;
            }
        }
        t_run = t_next;
        step = step_next;
        dt = dt_next;
        last = last_next;
        if (done) break;
    }

    if (active) {
#pragma unroll
        for (int e = 0; e < NH; e++) S.f0[(sp * NH + e) * cap + p] = y0[e];
        if (not_finite<NH>(y0)) ctl->odd = 1;
        if (sp == 0) {
            S.pos[0][p] = x;
            S.pos[1][p] = yy;
            S.pos[2][p] = z;
            S.time[p] = tp;
        }
    }
    if constexpr (ONE) {
        // the new state's mesh and a clean next one, as a step leaves them
        for (int i = tid; i < msize; i += blockDim.x) {
            const int c = i / NCS, q = i - c * NCS;
            cmesh[i] = q < NG ? smesh[cur * kHalf + c * MR + q] : sdiag[c * kDiagSlots + q - NG];
            cmesh[msize + i] = 0.0;
        }
    }
    // the last CTA to leave writes the step control (all hold the same), unless
    // another gave up a wait: then the run ends with the steps before this launch
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1) {
            __threadfence();
            ctl->blocks_done = 0u;
            ctl->bar_count = 0u;
            if (!ONE && dt_mode == DT_ADVANCE) {
                const double vm = __longlong_as_double((long long)__ldcg(&ctl->vmax_bits[slot]));
                dt = next_dt_stupid(P, fmax(P.flavor_cfl_factor > 0.0 ? vm : 0.0, dt_vmin), dt_fac, st_dt);
                if (end_time - t_run < dt) {
                    dt = end_time - t_run;
                    last = 1;
                }
                if (st_dt) done = 1;
            }
            ctl->vmax_bits[0] = ctl->vmax_bits[1] = 0ull;
            if (steps_timed_out(ctl)) {
                ctl->done = 1;
            } else if (dt_mode == DT_ADVANCE) {
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

template <int NF, bool ONE, int MAXT, bool REC>
__global__ void __launch_bounds__(MAXT, 1)
    k_steps_1d(DevParams P, DevState S, double* __restrict__ cmesh, double* __restrict__ full, StepCtl* ctl,
               int npart, int nsteps, int dt_mode, Rec1DStore store)
{
    if (ctl->done) return;
    if (ctl->odd) steps_1d_body<NF, ONE, REC, true>(P, S, cmesh, full, ctl, npart, nsteps, dt_mode, store);
    else steps_1d_body<NF, ONE, REC, false>(P, S, cmesh, full, ctl, npart, nsteps, dt_mode, store);
}

// The backward sweep over recorded steps of a 1D run (emu_adjoint.cu: the
// discrete adjoint), last step first, in one cooperative launch with the
// means of k_steps_1d: the adjoint state in registers, the windows of the
// adjoint mesh and of the recorded stage mesh in shared memory, matrix
// products for the two gathers and the scatter, four grid barriers per step
// (stage 0 only gathers).  The next stage's recorded mesh and state are
// loaded between arrival and wait.  Two flavors, 128 x 80: a recorded step
// 49 -> 17 us, a backward step 62 -> 22 us (against tiles of 128 particles
// that reloaded their state and ranked their keys in every stage).  CELLS: as
// k_steps_1d, for a recorded state or an adjoint state that is not finite.
template <int NF, bool CELLS>
__device__ __forceinline__ void adjoint_1d_body(const DevParams& P, const DevState& S, const Adj1DStore& A, StepCtl* ctl,
                                                int npart, int len)
{
    using H = Herm<NF>;
    using C = Comb<NF>;
    using R = Rec1D<NF>;
    constexpr int NH = NF * NF, NV = C::NV, HV = NV / 2;
    extern __shared__ __align__(16) double smem[];
    double* const sm_lam = smem;                              // window of the adjoint mesh
    double* const sm_fwd = smem + (kWin + 4) * R::MR;         // and of the recorded stage mesh
    double* const srec = sm_fwd + (kWin + 4) * R::MR;
    __shared__ int swin[2][16];
    __shared__ int sref;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int pl = tid >> 1, sp = tid & 1;
    const long long p = (long long)blockIdx.x * npart + pl;
    const bool active = p < S.n;
    const long long cap = S.cap;
    const int nz = P.n[2], msize = (int)P.ncells * kCombSlots<NF>;
    const int nthreads = gridDim.x * blockDim.x, gtid = blockIdx.x * blockDim.x + tid;
    double* const rec = srec + pl * R::RW;
    double* const wrec = srec + warp * 16 * R::RW;

    double vs = 0, Ns = 0, Ls = 1, dN = 0;
    double lamY[NH] = {}, lamn[NH] = {}, lamYd[NH] = {}, ys[NH] = {}, yn[NH] = {};
    if (active) {
        vs = S.vscale[p];
        Ns = S.Nn[sp][p];
        Ls = S.Ll[sp][p];
#pragma unroll
        for (int e = 0; e < NH; e++) lamY[e] = A.lamY0[(sp * NH + e) * cap + p];
    }
    if (sp == 0) {
        rec[3] = 0.0;
        rec[R::V] = 1.0;
#pragma unroll
        for (int d = 0; d < 3; d++) rec[R::V + 1 + d] = active ? S.vhat[d][p] : 0.0;
    }
    // a recorded state's components of this thread
    auto load = [&](const double* base, double* y) {
        if (active)
#pragma unroll
            for (int e = 0; e < NH; e++) y[e] = __ldcg(base + (sp * NH + e) * cap + p);
    };
    auto stage_mesh = [&](int j, int s) { return A.rec.mst + j * A.rec.mst_stride + (s - 1) * msize; };
    auto zpos = [&](int j) { return active ? __ldcg(A.rec.seg + j * A.rec.seg_stride + (2 * NH + 2) * cap + p) : 0.0; };
    Place1D L;
    if (tid == 0) {   // (the CTA's first particle exists)
        int first;
        shape<double>(zpos(len - 1) * P.dxi[2], P.ord[2], first, L.wz);
        sref = wrapi(first, nz);
    }
    if (!__syncthreads_and(!steps_timed_out(ctl))) {
        // (a segment swept before this one in the same call gave up)
        if (tid == 0) steps_gave_up(ctl);
        return;
    }
    const bool patient = P.wait_polls >= kFirstPolls;
    unsigned nbar = 0;
    for (int j = len - 1; j >= 0; j--) {
        const double* const sst = A.rec.sst + j * A.rec.sst_stride;
        const double dt = A.dts[j];
        load(sst + 3 * (2 * NH) * cap, yn);   // Y_n
        load(sst + 2 * (2 * NH) * cap, ys);   // Y_4
        place_particles<NF, CELLS>(P, L, zpos(j), active, sp, sref, swin, rec, wrec);
        stage_window<NF>(L, sm_fwd, stage_mesh(j, 4), nz);
        __syncthreads();
#pragma unroll 1
        for (int s = 4; s >= 0; s--) {
            double lamK[NH];
            if (s == 4) {
                double ln[NH];
                renormalize_vjp<NF>(yn, Ls, P.maxError, lamY, ln);
                const double b4 = dt * (1. / 6.);
#pragma unroll
                for (int e = 0; e < NH; e++) {
                    lamn[e] = lamY[e] = ln[e];
                    lamK[e] = b4 * ln[e];
                    yn[e] = ys[e];
                }
            } else {
                // the gather of stage s + 1's adjoint mesh: G of nu; of nubar
                // with the opposite sign for real components
                const double* const lm_in = A.lm + ((s + 1) & 3) * A.lm_stride;
                stage_window<NF>(L, sm_lam, lm_in, nz);
                __syncthreads();
                double gv[NV], g[NH];
                interp_1d<NF, false, true>(P, L, sm_lam, nullptr, lm_in, rec, wrec, sp, active, gv);
                __syncwarp();
                C::hermitian(gv, g);
                const double b = dt * (s == 1 ? 1. / 6. : 1. / 3.), a = dt * (s == 3 ? 1.0 : 0.5);
#pragma unroll
                for (int e = 0; e < NH; e++) {
                    const double G = sp == 0 || H::is_im(e) ? g[e] : -g[e];
                    const double ly = lamYd[e] + Ns * G;   // lam of Y_{s+1}
                    dN += yn[e] * G;
                    lamY[e] += ly;
                    lamK[e] = b * lamn[e] + a * ly;
                    yn[e] = ys[e];   // (Y_s: the next gather's)
                }
                if (s == 0) break;
            }
            // commutator VJP and the scatter of lam_H
            double hv[NV], h[NH], lH[NH], cc[NH], cv[NV];
            interp_1d<NF, false, false>(P, L, sm_fwd, nullptr, stage_mesh(j, s), rec, wrec, sp, active, hv);
#pragma unroll
            for (int q = 0; q < NV; q++) hv[q] *= P.sqrt2GF_inv_vol;
            C::hermitian(hv, h);
            species_hamiltonian<NF>(P, h, vs, sp, h);
            commutator_vjp<NF>(h, ys, lamK, lH, lamYd, P.inv_hbar);
#pragma unroll
            for (int e = 0; e < NH; e++) {
                const double o = __shfl_xor_sync(kFull, lH[e], 1);
                cc[e] = P.sqrt2GF_inv_vol * (H::is_im(e) ? lH[e] + o : (sp == 0 ? lH[e] - o : o - lH[e]));
            }
            C::values(cc, cv);
            __syncwarp();   // (the pair's reads of the interpolated values)
#pragma unroll
            for (int q = 0; q < HV; q++) {
                const double x = sp == 0 ? cv[q] : cv[HV + q];
                rec[R::CV + sp * HV + q] = active ? x : 0.0;
            }
            __syncwarp();
            double* const lm_out = A.lm + (s & 3) * A.lm_stride;
            if (!CELLS && !L.wide) deposit_1d<NF, true>(L, srec, nullptr, wrec, lm_out, nz, false);
            else if (active) deposit_1d_cells<NF, true>(P, L, rec, sp, L.wide ? L.ci0 : L.c0 + L.ci0, lm_out, false);
            // the next stage's target (last read three stages ago)
            double* const lz = A.lm + ((s + 3) & 3) * A.lm_stride;
            for (int i = gtid; i < msize; i += nthreads) lz[i] = 0.0;
            steps_arrive(ctl);
            if (s > 1) {
                stage_window<NF>(L, sm_fwd, stage_mesh(j, s - 1), nz);
                load(s == 2 ? A.rec.seg + j * A.rec.seg_stride : sst + (s - 3) * (2 * NH) * cap, ys);   // Y_{s-1}
            }
            nbar++;
            if (!steps_wait(ctl, nbar * gridDim.x, patient, P.wait_polls)) {
                if (tid == 0) steps_gave_up(ctl);
                return;
            }
        }
    }
    if (active) {
#pragma unroll
        for (int e = 0; e < NH; e++) A.lamY0[(sp * NH + e) * cap + p] = lamY[e];
        A.lamN[sp * cap + p] += dN;
    }
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&ctl->blocks_done, 1u) == gridDim.x - 1) {
            __threadfence();
            ctl->blocks_done = 0u;
            ctl->bar_count = 0u;
        }
    }
}

template <int NF, int MAXT>
__global__ void __launch_bounds__(MAXT, 1)
    k_adjoint_1d(DevParams P, DevState S, Adj1DStore A, StepCtl* ctl, int npart, int len)
{
    if (ctl->odd | ctl->odd_lam) adjoint_1d_body<NF, true>(P, S, A, ctl, npart, len);
    else adjoint_1d_body<NF, false>(P, S, A, ctl, npart, len);
}

// particles per CTA: spread over the SMs, whole warps of 16, at least 64 (a
// smaller CTA only adds barrier arrivals) and at most 256 (512 threads)
int particles_per_cta(long long n, int nsm)
{
    const long long per = (n + nsm - 1) / nsm;
    return (int)std::max<long long>(64, (per + 15) / 16 * 16);
}

bool one_cta(const DevParams& P, long long n) { return n <= kOnePart && P.ncells <= kOneCells; }

int device_sms()
{
    int dev = 0, nsm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        nsm = 0;
    cudaGetLastError();
    return nsm;
}

// the kernel for a CTA of npart particles: the fewer threads, the more
// registers each (three flavors spill at 128)
using Steps1DKernel = void (*)(DevParams, DevState, double*, double*, StepCtl*, int, int, int, Rec1DStore);
template <int NF, bool REC>
Steps1DKernel steps1d_kernel(bool one, int npart)
{
    if constexpr (!REC)
        if (one) return k_steps_1d<NF, true, 256, false>;
    if (npart <= 128) return k_steps_1d<NF, false, 256, REC>;
    if (npart <= 192) return k_steps_1d<NF, false, 384, REC>;
    return k_steps_1d<NF, false, 512, REC>;
}

template <int NF>
cudaError_t launch_t(const DevParams& P, const DevState& S, double* cmesh, double* full, StepCtl* ctl, int nsteps,
                     int dt_mode, cudaStream_t st, const Rec1DStore* rec)
{
    const bool one = !rec && one_cta(P, S.n);
    int npart = one ? kOnePart : particles_per_cta(S.n, device_sms());
    const Steps1DKernel kern = rec ? steps1d_kernel<NF, true>(false, npart) : steps1d_kernel<NF, false>(one, npart);
    const int bytes = one ? steps1d_smem<NF, true>(npart) : steps1d_smem<NF, false>(npart);
    smem_optin(kern, bytes);
    DevParams Pc = P;
    DevState Sc = S;
    Rec1DStore store = rec ? *rec : Rec1DStore{};
    void* args[] = {&Pc, &Sc, &cmesh, &full, &ctl, &npart, &nsteps, &dt_mode, &store};
    return cudaLaunchCooperativeKernel((const void*)kern, dim3(grid_for(S.n, npart)), dim3(2 * npart), args, bytes, st);
}

template <int NF>
cudaError_t launch_adjoint_t(const DevParams& P, const DevState& S, const Adj1DStore& A, StepCtl* ctl, int len,
                             cudaStream_t st)
{
    using R = Rec1D<NF>;
    int npart = particles_per_cta(S.n, device_sms());
    auto kern = npart <= 128 ? k_adjoint_1d<NF, 256> : npart <= 192 ? k_adjoint_1d<NF, 384> : k_adjoint_1d<NF, 512>;
    const int bytes = 8 * (2 * (kWin + 4) * R::MR + npart * R::RW);
    smem_optin(kern, bytes);
    DevParams Pc = P;
    DevState Sc = S;
    Adj1DStore Ac = A;
    void* args[] = {&Pc, &Sc, &Ac, &ctl, &npart, &len};
    return cudaLaunchCooperativeKernel((const void*)kern, dim3(grid_for(S.n, npart)), dim3(2 * npart), args, bytes, st);
}

}  // namespace

// one-dimensional along z, at most 256 particles per SM (two flavors, 128 x
// 80: 40 -> 15 us per step; past one CTA per SM the stage kernels, which
// keep several CTAs in flight on each, take over)
bool steps_1d_fit(int nf, const DevParams& P, long long n)
{
    if (P.n[0] != 1 || P.n[1] != 1 || P.max_adaptive_speedup > 1.0) return false;
    if (P.ncells > (1 << 20)) return false;   // (mesh offsets are ints)
    if (one_cta(P, n)) return true;
    const int nsm = device_sms();
    return nsm > 0 && particles_per_cta(n, nsm) <= 256;
}

cudaError_t launch_steps_1d(int nf, const DevParams& P, const DevState& S, double* cmesh, double* full, StepCtl* ctl,
                            int nsteps, int dt_mode, cudaStream_t st, const Rec1DStore* rec)
{
    return nf == 2 ? launch_t<2>(P, S, cmesh, full, ctl, nsteps, dt_mode, st, rec)
                   : launch_t<3>(P, S, cmesh, full, ctl, nsteps, dt_mode, st, rec);
}

cudaError_t launch_adjoint_1d(int nf, const DevParams& P, const DevState& S, const Adj1DStore& A, StepCtl* ctl, int len,
                              cudaStream_t st)
{
    return nf == 2 ? launch_adjoint_t<2>(P, S, A, ctl, len, st) : launch_adjoint_t<3>(P, S, A, ctl, len, st);
}

}  // namespace emu
