// Host side of the direct correction (gb_direct.cu): the eigenvector tables
// of one solver, and a group of grids solved by one captured loop.
#pragma once

#include <memory>
#include <vector>

#include "gb_direct.cuh"

namespace gb {

struct DirectTables {
    DirAxis ax[3];
    double* mem = nullptr;
    ~DirectTables();
    // pe/po: row-major [point][mode] halves of each axis's eigenvectors, lam
    // their eigenvalues (even first)
    int build(const GridBC& g, const double* const pe[3], const double* const po[3],
              const double* const lam[3]);
};

struct DirectGroup {
    int n = 0, nn = 0;
    char* mem = nullptr;
    DirGrid* grids = nullptr;
    DirCtl* ctl = nullptr;
    // outcomes of the last launch, one a grid (pinned); solvers share them
    std::shared_ptr<DirCtl> results;
    // the CTAs of one launch: grids of one block shape along one axis
    struct Part {
        DirBlock* map = nullptr;   // (one grid: block index alone)
        int blocks = 0, rows = 0;
    };
    Part part[3][4], defect;
    cudaGraphExec_t exec = nullptr;
    ~DirectGroup();
    int build(const std::vector<DirGrid>& desc, int half_width, cudaStream_t cs);
    int capture(cudaStream_t cs);
    int run(cudaStream_t st);
    int solve(double* phi, const double* rho, double tol, int maxiter, cudaStream_t st);
    int eager(double* phi, const double* rho, cudaStream_t st);
    int solve_batch(double* const* user, double tol, int maxiter, cudaStream_t st);
};

}  // namespace gb
