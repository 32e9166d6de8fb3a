// emu_tile64.cuh -- interpolation and deposit of a CTA's 128 particles as FP64
// matrix products (m8n8k4 on the FP64 tensor cores), for the FP64 stages, the
// adjoint and the mixed path's deposits.
//
// Per particle and stage the interpolation and the deposit of a 27-cell
// stencil are 27 x 32 multiply-adds each (three flavors, Comb<NF>), about
// three quarters of the arithmetic, and both are small matrix products of
// particles that share a stencil (cell-sorted particles come in runs of about
// the number of directions per cell):
//   interpolation  G[p][q] = sum_c W[p][c] M[c][q]
//   deposit        D[c][q] = sum_p W[p][c] Q[p][q],  Q[p][(d, j)] = c_j v_d
// A product's operands are one value per lane for 256 FMAs (IEEE, at the rate
// of the FP64 pipe), so that the loads around the FMAs all but vanish: the
// former interpolation read 72 values per cell and thread, the former run
// sums 27 weights per record and lane.
//   Warp w interpolates slots 32 w .. 32 w + 31 of the CTA's 128: per distinct
// stencil it holds the cells' values (KS x NT fragments, loaded once) and
// multiplies the groups of eight particles that contain it.  Deposit: warp w
// owns the values of one 8-column tile (two flavors: half of the slots each)
// and sums whole runs of equal stencils over the CTA, so that a run costs one
// global reduction per (cell, value) and CTA.
#pragma once
#include "emu_fp64.cuh"
#include "emu_kernels.cuh"

#include <cub/block/block_radix_sort.cuh>

namespace emu {
namespace {

// Stable rank of the stencil keys held by the first NW warps of the block
// (key -1 = inactive, ranked last): the permutation a stable sort of the
// keys gives, by a counting sort over the distinct keys when the warps hold
// at most 32 (warp, key) groups (cell-sorted particles that moved a few
// cells: the usual case).  Group leaders list their keys, one warp sorts the
// list (bitonic, shuffles) and drops repeats, every thread finds its key's
// bucket by binary search, and one warp scans the (bucket, warp) counts.
// Every thread of the block calls it; the result is uniform over the block:
// false (nothing ranked, the caller sorts; the scratch is free again) when
// there are more groups.  scratch: 66 + 32 NW ints; on success it is read
// after the last barrier here, so the caller waits at a barrier before it
// writes there.
template <int NW>
__device__ __forceinline__ bool distinct_key_rank(int key, int* scratch, int& slot)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool part = w < NW;
    const unsigned lt = (1u << lane) - 1u;
    int* ngroups = scratch;                                      // (warp, key) groups listed
    int* nkeys = scratch + 1;                                    // distinct keys
    unsigned* list = reinterpret_cast<unsigned*>(scratch + 2);   // [32] group keys
    unsigned* ukey = list + 32;                                  // [32] sorted distinct keys
    int* cnt = scratch + 66;                                     // [NW][32] counts, then bases
    if (threadIdx.x == 0) *ngroups = 0;
    if (part) cnt[w * 32 + lane] = 0;
    __syncthreads();
    const unsigned k = key >= 0 ? (unsigned)key : 0xffffffffu;   // inactive last
    unsigned peers = 0u;
    if (part) {
        peers = __match_any_sync(kFull, k);
        if ((peers & lt) == 0u) {
            const int i = atomicAdd(ngroups, 1);
            if (i < 32) list[i] = k;
        }
    }
    __syncthreads();
    const int ng = *ngroups;
    if (ng > 32) {
        __syncthreads();   // every thread has read the count before the caller's sort reuses the scratch
        return false;
    }
    if (w == 0) {
        unsigned v = lane < ng ? list[lane] : 0xffffffffu;
#pragma unroll
        for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                const unsigned o = __shfl_xor_sync(kFull, v, stride);
                const bool up = (lane & size) == 0, lower = (lane & stride) == 0;
                v = (lower == up) ? min(v, o) : max(v, o);
            }
        const unsigned prev = __shfl_up_sync(kFull, v, 1);
        const bool first = lane == 0 || prev != v;
        const unsigned fm = __ballot_sync(kFull, first);
        if (first) ukey[__popc(fm & lt)] = v;
        if (lane == 0) *nkeys = __popc(fm);
    }
    __syncthreads();
    int b = 0, rank = 0;
    if (part) {
        int lo = 0, hi = *nkeys - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (ukey[mid] < k) lo = mid + 1;
            else hi = mid;
        }
        b = lo;
        rank = __popc(peers & lt);
        if ((peers & lt) == 0u) cnt[w * 32 + b] = __popc(peers);
    }
    __syncthreads();
    if (w == 0) {
        // lane = bucket: base of each (bucket, warp) in bucket-major order
        int c[NW], tot = 0;
#pragma unroll
        for (int i = 0; i < NW; i++) {
            c[i] = cnt[i * 32 + lane];
            tot += c[i];
        }
        int inc = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(kFull, inc, o);
            if (lane >= o) inc += t;
        }
        int base = inc - tot;
#pragma unroll
        for (int i = 0; i < NW; i++) {
            cnt[i * 32 + lane] = base;
            base += c[i];
        }
    }
    __syncthreads();
    if (part) slot = cnt[w * 32 + b] + rank;
    return true;
}

// Stencils of up to 4 KS cells; WX, WY, WZ fixed widths, or 0: any widths
// (run time) whose product is at most 4 KS.
template <int NF, int WX, int WY, int WZ, int KS_>
struct Tile64 {
    static constexpr int KS = KS_, WP = 4 * KS, MT = (WP + 7) / 8;
    static constexpr bool FIXED = WX > 0;
    static constexpr int NV = Comb<NF>::NV, NG = Comb<NF>::NG, NT = NG / 8, NCS = kCombSlots<NF>;
    // record row: weights, then NVAL values; a length of 4 or 12 mod 16 words
    // puts the rows of four particles into different banks
    template <int NVAL>
    __host__ __device__ static constexpr int row()
    {
        int r = WP + NVAL;
        while (r % 16 != 4 && r % 16 != 12) r++;
        return r;
    }
    static constexpr int VS = kBlock + 4;   // stride of the per-slot arrays
    static_assert(8 * MT <= WP + NV, "a tile's last rows stay inside the record");
};

// the number of stencil cells (widths at run time)
__device__ __forceinline__ int stencil_cells(const DevParams& P) { return P.w[0] * P.w[1] * P.w[2]; }

// cell offset of stencil cell c from the first cell (no wrap), and wrapped
template <class T, int WX, int WY>
__device__ __forceinline__ void stencil_decode(const DevParams& P, int c, int& ii, int& jj, int& kk)
{
    const int w0 = T::FIXED ? WX : P.w[0], w1 = T::FIXED ? WY : P.w[1];
    if (c >= stencil_cells(P)) c = 0;   // (padding: zero weight, any cell)
    ii = c % w0;
    jj = (c / w0) % w1;
    kk = c / (w0 * w1);
}

// A stencil's cells for one lane: cell index of stencil cell c of the stencil
// whose first cell is the key
struct KeyCells {
    int bx, by, bz;
    bool inside;   // no cell wraps
    __device__ __forceinline__ KeyCells(const DevParams& P, int key)
    {
        bx = key % P.n[0];
        const int r = key / P.n[0];
        by = r % P.n[1];
        bz = r / P.n[1];
        inside = bx + P.w[0] <= P.n[0] && by + P.w[1] <= P.n[1] && bz + P.w[2] <= P.n[2];
    }
    // (a stencil wider than a periodic dimension wraps more than once)
    template <class T, int WX, int WY>
    __device__ __forceinline__ int wrapped(const DevParams& P, int c) const
    {
        int ii, jj, kk;
        stencil_decode<T, WX, WY>(P, c, ii, jj, kk);
        return (((bz + kk) % P.n[2]) * P.n[1] + (by + jj) % P.n[1]) * P.n[0] + (bx + ii) % P.n[0];
    }
};

// The CTA's slice of NS state arrays (128 consecutive particles each) into
// L2, while the tile is interpolated (capacities are whole tiles: 16-byte
// aligned, in bounds).  32^3 cells x 96: 647 -> 636 us for stage 1; 90 x 77 x
// 60: 83 -> 77 us.
template <int NS>
__device__ __forceinline__ void prefetch_slices(const double* a, long long cap, int t)
{
    if (t >= 0 && t < NS)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a + t * cap + (long long)blockIdx.x * kBlock),
                     "r"(kBlock * 8)
                     : "memory");
}

// phase A of a tile: this thread's weights (and zeros up to WP) into record
// row `rec`; inactive threads write zeros
template <class T, int WX, int WY, int WZ>
__device__ __forceinline__ void write_weights(const DevParams& P, double* rec, bool active, const Stencil<double>& st)
{
    if constexpr (T::FIXED) {
        double w[T::WP];
#pragma unroll
        for (int kk = 0; kk < WZ; kk++)
#pragma unroll
            for (int jj = 0; jj < WY; jj++)
#pragma unroll
                for (int ii = 0; ii < WX; ii++)
                    w[(kk * WY + jj) * WX + ii] = active ? (st.wx[ii] * st.wy[jj]) * st.wz[kk] : 0.0;
#pragma unroll
        for (int c = WX * WY * WZ; c < T::WP; c++) w[c] = 0.0;
#pragma unroll
        for (int c = 0; c < T::WP; c += 2) *reinterpret_cast<double2*>(rec + c) = make_double2(w[c], w[c + 1]);
    } else {
        int c = 0;
#pragma unroll
        for (int kk = 0; kk < 3; kk++)
#pragma unroll
            for (int jj = 0; jj < 3; jj++)
#pragma unroll
                for (int ii = 0; ii < 3; ii++)
                    if (ii < P.w[0] && jj < P.w[1] && kk < P.w[2])
                        rec[c++] = active ? (st.wx[ii] * st.wy[jj]) * st.wz[kk] : 0.0;
        for (; c < T::WP; c++) rec[c] = 0.0;
    }
}

// run starts of the 128 slots' keys (skey, -1 last), one word per warp; the
// caller has a barrier before and after
__device__ __forceinline__ void run_starts(const int* skey, unsigned* starts)
{
    const int t = threadIdx.x;
    if (t < kBlock) {
        const int k = skey[t];
        const bool first = k >= 0 && (t == 0 || skey[t - 1] != k);
        const unsigned m = __ballot_sync(kFull, first), a = __ballot_sync(kFull, k >= 0);
        if ((t & 31) == 0) {
            starts[t >> 5] = m;
            starts[4 + (t >> 5)] = __popc(a);
        }
    }
}

// The interpolated, velocity-weighted sums u_j = G_0j - v . G_dj of the
// warp's 32 slots, from the combined mesh, into the records' values
// (rec + WP + j).  sv: v per slot and dimension, rows of VS.  PLUS: G_0 + v . G_d
// (the transpose of a deposit, see emu_adjoint.cu).  LIVE: see mesh_load.
template <int NF, class T, int WX, int WY, int RW, bool PLUS = false, bool LIVE = false>
__device__ __forceinline__ void interp64(const DevParams& P, const double* mesh, double* srec, const int* skey,
                                         const double* sv)
{
    constexpr int KS = T::KS, NT = T::NT, NV = T::NV, NCS = T::NCS, WP = T::WP, VS = T::VS;
    const int lane = threadIdx.x & 31, base = threadIdx.x & ~31, row = lane >> 2, col = lane & 3;
    const int mykey = skey[base + lane];
    unsigned todo = __ballot_sync(kFull, mykey >= 0);
    int off[KS];
#pragma unroll
    for (int k = 0; k < KS; k++) {
        int ii, jj, kk;
        stencil_decode<T, WX, WY>(P, 4 * k + col, ii, jj, kk);
        off[k] = (kk * P.n[1] + jj) * P.n[0] + ii;
    }
    // two flavors: column 2 e + i of tile nt is d = 2 nt + i of value e (a
    // lane's two columns of a product are then one value's)
    const int q0 = NF == 2 ? (row & 1) * NV + (row >> 1) : row;
    while (todo) {
        const int key = __shfl_sync(kFull, mykey, __ffs(todo) - 1);
        const unsigned mine = __ballot_sync(kFull, mykey == key);
        todo &= ~mine;
        const KeyCells kc(P, key);
        double b[KS][NT];
#pragma unroll
        for (int k = 0; k < KS; k++) {
            int cell = key + off[k];
            if (!kc.inside) cell = kc.template wrapped<T, WX, WY>(P, 4 * k + col);
            const double* m = mesh + (long long)cell * NCS + q0;
#pragma unroll
            for (int nt = 0; nt < NT; nt++) b[k][nt] = mesh_load<LIVE>(m + 8 * nt);
        }
#pragma unroll
        for (int g = 0; g < 4; g++) {
            if (((mine >> (8 * g)) & 0xffu) == 0u) continue;   // (uniform)
            double* r = srec + (base + 8 * g + row) * RW;
            double c[NT][2];
#pragma unroll
            for (int nt = 0; nt < NT; nt++) c[nt][0] = c[nt][1] = 0.0;
#pragma unroll
            for (int k = 0; k < KS; k++) {
                const double a = r[4 * k + col];
#pragma unroll
                for (int nt = 0; nt < NT; nt++) dmma(c[nt][0], c[nt][1], a, b[k][nt]);
            }
            // (the rows of other stencils: not theirs)
            if ((mine >> (8 * g + row)) & 1u) {
                const int s = base + 8 * g + row;
                const double sg = PLUS ? -1.0 : 1.0;
                const double vx = sg * sv[s], vy = sg * sv[VS + s], vz = sg * sv[2 * VS + s];
                if constexpr (NF == 2) {
                    r[WP + col] = ((c[0][0] - vx * c[0][1]) - vy * c[1][0]) - vz * c[1][1];
                } else {
                    r[WP + 2 * col] = ((c[0][0] - vx * c[1][0]) - vy * c[2][0]) - vz * c[3][0];
                    r[WP + 2 * col + 1] = ((c[0][1] - vx * c[1][1]) - vy * c[2][1]) - vz * c[3][1];
                }
            }
        }
    }
}

// Run sums of one 8-column tile of values over the slots [s0, s1): value(slot,
// n) is column n of the tile; add(cell, h, col, sum) adds the sum of column
// 2 col + h to a cell.  Columns are numbered so that (n >> 1) + 4 (n & 1) is
// the value: the four lanes of a row write 32 contiguous bytes.
// DIAG: value2, of a second tile (the diagonal slots), on the rows of the
// cell tiles mt = dm, dm + dstep, ...
template <class T, int WX, int WY, int RW, bool DIAG, class Val, class Add, class Val2, class Add2>
__device__ __forceinline__ void deposit_runs64(const DevParams& P, const double* srec, const int* skey,
                                               const unsigned* starts, int s0, int s1, Val value, Add add, int dm,
                                               int dstep, Val2 value2, Add2 add2)
{
    constexpr int MT = T::MT;
    const int lane = threadIdx.x & 31, row = lane >> 2, col = lane & 3;
    const int nact = starts[4] + starts[5] + starts[6] + starts[7];
    s1 = min(s1, nact);
    int off[MT];
#pragma unroll
    for (int m = 0; m < MT; m++) {
        int ii, jj, kk;
        stencil_decode<T, WX, WY>(P, 8 * m + row, ii, jj, kk);
        off[m] = (kk * P.n[1] + jj) * P.n[0] + ii;
    }
    const int ncell = stencil_cells(P);
    for (int a = s0; a < s1;) {
        // the run [a, e): up to the next start after a
        int e = s1;
        {
            int w = (a + 1) >> 5;
            unsigned m = w < 4 ? starts[w] & (0xffffffffu << ((a + 1) & 31)) : 0u;
            while (m == 0u && ++w < 4) m = starts[w];
            if (m) e = min(e, w * 32 + __ffs(m) - 1);
        }
        const int key = skey[a];
        double c[MT][2], c2[DIAG ? MT : 1][2];
#pragma unroll
        for (int m = 0; m < MT; m++) c[m][0] = c[m][1] = 0.0;
        if constexpr (DIAG)
#pragma unroll
            for (int m = 0; m < MT; m++) c2[m][0] = c2[m][1] = 0.0;
        // slots 4 k .. 4 k + 3; masked: some belong to another run (their
        // values and weights, which need not be finite, count as zero; rows
        // past the stencil's cells hold other words of the record and are not
        // used)
        auto step = [&](int k, bool masked) {
            const int s = 4 * k + col;
            const bool in = !masked || (s >= a && s < e);
            const double* r = srec + s * RW + row;
            double b = value(s, row), b2 = 0.0;
            if (!in) b = 0.0;
            if constexpr (DIAG) {
                b2 = value2(s, row);
                if (!in) b2 = 0.0;
            }
#pragma unroll
            for (int m = 0; m < MT; m++) {
                double wgt = r[8 * m];
                if (!in) wgt = 0.0;
                dmma(c[m][0], c[m][1], wgt, b);
                if constexpr (DIAG)
                    if (m % dstep == dm) dmma(c2[m][0], c2[m][1], wgt, b2);
            }
        };
        int k = a >> 2;
        const int kend = (e + 3) >> 2, kfull = e >> 2;
        if (a & 3) step(k++, true);
#pragma unroll 4
        for (; k < kfull; k++) step(k, false);
        if (k < kend) step(k, true);
        const KeyCells kc(P, key);
#pragma unroll
        for (int m = 0; m < MT; m++) {
            if (8 * m + row < ncell) {
                int cell = key + off[m];
                if (!kc.inside) cell = kc.template wrapped<T, WX, WY>(P, 8 * m + row);
                add(cell, col, c[m][0]);
                add(cell, col + 4, c[m][1]);
                if constexpr (DIAG)
                    if (m % dstep == dm) {
                        add2(cell, col, c2[m][0]);
                        add2(cell, col + 4, c2[m][1]);
                    }
            }
        }
        a = e;
    }
}

struct NoVal {
    __device__ double operator()(int, int) const { return 0.0; }
};
struct NoAdd {
    __device__ void operator()(int, int, double) const {}
};

// the combined deposit of the CTA's records (values c_j at rec + WP + j; sv:
// v per slot; sd: with DIAG the 2 NF diagonal numbers per slot, rows of VS).
// MINUS: fluxes with -v (the transpose of an interpolation)
template <int NF, class T, int WX, int WY, int RW, bool DIAG, bool MINUS = false>
__device__ __forceinline__ void deposit_comb64(const DevParams& P, double* mesh, const double* srec, const int* skey,
                                               const unsigned* starts, const double* sv, const double* sd)
{
    constexpr int NT = T::NT, NV = T::NV, NG = T::NG, NCS = T::NCS, WP = T::WP, VS = T::VS;
    constexpr int SPLIT = 4 / NT;   // parts of the slots (two flavors: halves)
    const int w = threadIdx.x >> 5, nt = w % NT, part = w / NT;
    const int s0 = part * (kBlock / SPLIT), s1 = s0 + kBlock / SPLIT;
    auto value = [&](int s, int n) {
        const int q = (n >> 1) + 4 * (n & 1);
        const double c = srec[s * RW + WP + q % NV];
        const int d = (8 * nt + q) / NV;   // (three flavors: uniform over the warp)
        const double f = sv[(d > 0 ? d - 1 : 0) * VS + s];
        return d == 0 ? c : MINUS ? -(c * f) : c * f;
    };
    auto add = [&](int cell, int q, double x) { atomic_add_mesh(mesh + (long long)cell * NCS + 8 * nt + q, x); };
    if constexpr (DIAG) {
        auto value2 = [&](int s, int n) {
            const int q = (n >> 1) + 4 * (n & 1);
            return q < 2 * NF ? sd[(q < 2 * NF ? q : 0) * VS + s] : 0.0;
        };
        auto add2 = [&](int cell, int q, double x) {
            if (q < 2 * NF) atomic_add_mesh(mesh + (long long)cell * NCS + NG + q, x);
        };
        deposit_runs64<T, WX, WY, RW, true>(P, srec, skey, starts, s0, s1, value, add, nt, NT, value2, add2);
    } else {
        deposit_runs64<T, WX, WY, RW, false>(P, srec, skey, starts, s0, s1, value, add, 0, 1, NoVal(), NoAdd());
    }
}

// slots of a CTA's particles in key order: the rank of this thread's key
// (scratch: at least the radix sort's storage; barriers inside, the scratch
// is free on return)
__device__ __forceinline__ int rank_slots(const DevParams& P, int key, void* scratch, int* srank)
{
    using Sort = cub::BlockRadixSort<unsigned, kBlock, 1, int>;
    int slot = threadIdx.x;
    if (distinct_key_rank<kBlock / 32>(key, reinterpret_cast<int*>(scratch), slot)) {
        __syncthreads();
        return slot;
    }
    auto& tmp = *reinterpret_cast<typename Sort::TempStorage*>(scratch);
    unsigned k[1] = {key >= 0 ? (unsigned)key : (unsigned)P.ncells};   // inactive slots last
    int v[1] = {(int)threadIdx.x};
    Sort(tmp).Sort(k, v, 0, P.key_bits);
    srank[v[0]] = threadIdx.x;
    __syncthreads();
    return srank[threadIdx.x];
}

// dynamic shared memory of the FP64 tiles: records, v, diagonal numbers,
// keys, ranks, run starts
template <int NF, class T, int RW>
struct Smem64 {
    double *rec, *v, *d;
    int *key, *rank;
    unsigned* starts;
    __device__ __forceinline__ explicit Smem64(unsigned char* p)
    {
        rec = reinterpret_cast<double*>(p);
        v = rec + kBlock * RW;
        d = v + 3 * T::VS;
        key = reinterpret_cast<int*>(d + 2 * NF * T::VS);
        rank = key + kBlock;
        starts = reinterpret_cast<unsigned*>(rank + kBlock);
    }
};

}  // namespace
}  // namespace emu
