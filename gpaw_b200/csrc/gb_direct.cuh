// The separable form of one grid's level-0 operator and the state of its
// solve: what the direct correction (gb_direct.cu) and the grouped FP64
// defect (gb_pass.cu) of the mixed solver read on the device.
#pragma once

#include "gb_internal.cuh"

namespace gb {

constexpr int DIR_KT = 12;     // table rows a warp accumulates
constexpr int DIR_W = 64;      // grid lines a CTA transforms
constexpr int DIR_P = DIR_W + 1;   // odd pitch: lanes along either index hit distinct banks
constexpr int DIR_HMAX = 192;  // modes of one parity along an axis (16 warps)

// One axis: n points, eigenvectors that are even (he of them) or odd (ho)
// under the reflection that the boundary keeps.
struct DirAxis {
    int n, per, he, ho;
    int kpe, kpo;              // he, ho rounded up to the staging chunk
    const double* fe;          // [tile][kpe][DIR_KT]: even, points -> modes
    const double* fo;
    const double* be;          // modes -> points
    const double* bo;
    const double* lam;         // he + ho eigenvalues; the axes' sum is the operator's
};

struct DirGrid {
    int n[3];
    GridBC g;
    DirAxis ax[3];
    double tiny;               // a mode with |eigenvalue| below it is left out
    // FP64 defect: stencil, tile geometry, partial sums (2 a CTA)
    double c0, cp[3][3], cm[3][3];
    int chunk, tiles_x, tiles, nblk;
    double* partial;
    double* X;                 // work grid
    double* phi;               // this call's arrays
    const double* rho;
};

struct DirCtl {
    double rho2, rel, tol;
    int maxiter, niter, active, pad;
};

// a block's share of a group: grid index and local block
struct DirBlock {
    int grid, block;
};

// d = rho - L phi of every active grid into its X, with partials of d^2 and
// rho^2 (gb_pass.cu); map NULL: one grid
int launch_defect_group(int nn, const DirGrid* grids, const DirCtl* ctl, const DirBlock* map,
                        int nblocks, cudaStream_t st);
// tile geometry of that kernel for one grid among `share` grids of a group
void defect_group_geom(const GridBC& g, int per_grid_blocks, int& chunk, int& tiles_x,
                       int& tiles, int& nblk);

}  // namespace gb
