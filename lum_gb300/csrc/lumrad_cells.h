// lumrad_cells.h — cells of a world's block arrays (host and device code).
#pragma once
#include <cstddef>

#ifdef __CUDACC__
#define LUMRAD_HD __host__ __device__ __forceinline__
#else
#define LUMRAD_HD inline
#endif

namespace lumrad {

// Cells of a world's compact grid: one more than the grid on the high side of each axis, all of
// block 0 (what a lookup past the grid reads), so that the march reads the cell a ray leaves the
// world through without testing the grid's range.
inline size_t compact_cells(int X, int Y, int Z) { return (size_t)(X + 1) * (Y + 1) * (Z + 1); }

// Cell (bx, by, bz) of an array of rows of PX and planes of PY rows.  Unsigned: a world has fewer than
// 2^31 blocks and 2047 to an axis, its compact grid more than 2^31 cells at the most (1290 x 1290 x 1290
// blocks: the last block's cell is 2,150,017,197), which a signed index does not hold.
LUMRAD_HD unsigned cell_index(int PX, int PY, int bx, int by, int bz) {
    return (unsigned)bx + (unsigned)PX * ((unsigned)by + (unsigned)PY * (unsigned)bz);
}

// GetVoxel (radiance.comp:121-143) on integer voxel coordinates.  Block coordinate = ix/16
// truncated (OpSDiv); voxel in block = ix mod 16 floored (OpSMod) = ix & 15.  The grid fetch is
// in range iff -15 <= ix < 16*X, and then ix/16 == max(ix,0) >> 4; out of range reads block 0.
// PX, PY: the row and plane lengths of the array (the compact grid's are X + 1 and Y + 1).
LUMRAD_HD bool grid_index(int X, int Y, int Z, int PX, int PY, int ix, int iy, int iz, unsigned& idx) {
    const bool in = (unsigned)ix + 15u < (unsigned)(16 * X + 15) && (unsigned)iy + 15u < (unsigned)(16 * Y + 15) &&
                    (unsigned)iz + 15u < (unsigned)(16 * Z + 15);
    idx = cell_index(PX, PY, (ix > 0 ? ix : 0) >> 4, (iy > 0 ? iy : 0) >> 4, (iz > 0 ? iz : 0) >> 4);
    return in;
}

}  // namespace lumrad
