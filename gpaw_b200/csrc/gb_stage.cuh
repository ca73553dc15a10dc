// Which grid value the linear pass (gb_pass.cu) stages in each cell of a
// plane's tile.  Plain C++, so that the host can check it for every size.
#pragma once

#ifdef __CUDACC__
#define GB_STAGE_FN __host__ __device__ __forceinline__
#else
#define GB_STAGE_FN inline
#endif

namespace gb {

constexpr int PT_ROWS = 16;   // rows of a tile, 16 threads each
constexpr int PT_HX = 4;      // halo columns staged on each side

// Row r and column c of the plane as offset r n2 + c; -1 for a zero: outside
// a zero boundary, or still outside after one period.  (A tile is staged
// whole, 16 rows and 32 or 64 columns with their halos, so on a short
// periodic side, or past its last few points, cells lie two periods out.  No
// point of the plane reads them; as offsets they would be past its end.)
GB_STAGE_FN int staged_offset(int r, int c, int n1, int n2, int per1, int per2) {
    if (per1) r += r < 0 ? n1 : r >= n1 ? -n1 : 0;
    if (per2) c += c < 0 ? n2 : c >= n2 ? -n2 : 0;
    return r >= 0 && r < n1 && c >= 0 && c < n2 ? r * n2 + c : -1;
}

}  // namespace gb
