// The coarse levels of an FP64 V-cycle as one launch (gb_coarse.cu).
#pragma once

#include "gb_internal.cuh"

namespace gb {

constexpr int COARSE_LEVELS = 8;

struct CoarseLevel {
    int n[3], per[3], ng;
    double *phi, *tmp, *rho;  // device arrays; the result is left in phi
    // 2nd-order stencil; direction k runs along axis 2 - k.  rc0 = 1 / c0
    double c0, rc0, cp[3], cm[3];
    // weighted operator: the Laplacian above (weight w[0]) and three
    // derivatives, number i along axis gaxis[i] with centre tap gc0[i]
    const double* w[4];
    int gaxis[3];
    double gc0[3], gp[3], gm[3];
    int pre, post;
    double wj;                // relaxation weight
    int rplo[3];              // restriction to the next level: input padding
    double rw;                //   and mid-point weight
    int iplo[3], iskip[3];    // interpolation from the next level: padding, skip
    double iw;
};
struct CoarsePlan {
    int nl;
    CoarseLevel lv[COARSE_LEVELS];
};

// K = 2 transfers between this level and the next; false if they are not
bool coarse_transfers(CoarseLevel& L, int kr, const XferGeom& r, int ki, const XferGeom& i,
                      const int* ncoarse);
// most points of the first level (32768 with a cluster of 16 CTAs; 0: no
// cluster fits)
int coarse_points(bool weighted);
// 0, or an error when the device has no room for the cluster (message recorded)
int launch_coarse(const CoarsePlan& plan, bool weighted, cudaStream_t st);

}  // namespace gb
