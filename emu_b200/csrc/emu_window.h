// emu_window.h -- cell windows of the warps of a 1D CTA (emu_k_steps1d.cu) and
// the trip count of a deposit over them.  Compiles for the host too, where its
// test replays it.
#pragma once

#ifdef __CUDACC__
#define EMU_WINDOW_FN __host__ __device__ __forceinline__
#else
#define EMU_WINDOW_FN inline
#endif

namespace emu {

// window cells lo..hi that a warp's stencils touch; hi < lo: none
struct CellRange {
    int lo, hi;
};

// mn, mx: first stencil cells of the warp's particles, smallest and largest
// (mn > mx, with any values: it has no particle, and nothing may be formed
// from them); base: the CTA's smallest; width: cells of a stencil
EMU_WINDOW_FN CellRange warp_cells(int mn, int mx, int base, int width)
{
    if (mx < mn) return CellRange{0, -1};
    return CellRange{mn - base, mx - base + width - 1};
}

// tiles of eight cells that cover a range (0 for an empty one)
EMU_WINDOW_FN int cell_tiles(int lo, int hi) { return hi < lo ? 0 : (hi - lo) / 8 + 1; }

}  // namespace emu
