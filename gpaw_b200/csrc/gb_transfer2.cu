// Order-2 transfers (K = 2: multigrid levels and the preconditioner) of real
// FP64 grids: the same values as k_restrict and k_interpolate
// (gb_transform.cu), operation for operation.
//
// What bounds them: HBM (9 bytes a real fine point).  A coarse point needs 3
// x 3 x 3 fine ones, so there is little to share beyond what L1 holds: no
// shared memory and no barriers.  A warp takes 32 columns of a coarse row
// and marches along axis 0; a lane reads its own columns of the three fine
// rows (restriction) or its two coarse columns of two rows (interpolation)
// straight into registers, all of a plane at once, so that many loads are in
// flight, and keeps the in-plane results of the last plane.  One row a lane at
// every size: four for the restriction and two for the interpolation of large
// batches read less twice, but leave fewer warps to hide the loads.
// Restriction / interpolation in us, general kernels, then several rows, now:
// 128 x 111^3 366 / 466, 347 / 336, 316 / 305; 16 x 96^3 periodic 45 / 41,
// 55 / 39, 39 / 35; 64 x 48 x 64 x 80 periodic 52 / 53, 55 / 41, 50 / 38.
#include <algorithm>

#include "gb_internal.cuh"
#include "gb_split.cuh"

namespace gb {
namespace {

__device__ __forceinline__ bool wrap2(int& y, int n, int periodic) {
    if (y >= 0 && y < n) return true;
    if (!periodic) return false;
    y += y < 0 ? n : -n;
    return y >= 0 && y < n;
}
// 0.5 (v + w (vp + vm)), each operation rounded on its own
__device__ __forceinline__ double mid(double v, double vp, double vm, double w) {
    const double s = Num<double>::scale(Num<double>::add(vp, vm), w);
    return Num<double>::scale(Num<double>::add(v, s), 0.5);
}

__global__ void __launch_bounds__(256)
k_restrict2(const double* __restrict__ in, double* __restrict__ out, double* __restrict__ out2,
            XferGeom G, int chunk, int tiles2) {
    const int n0 = G.g.n[0], n1 = G.g.n[1], n2 = G.g.n[2];
    const int L = blockIdx.x % tiles2 * 32 + (threadIdx.x & 31);
    const int J = blockIdx.x / tiles2 * 8 + (threadIdx.x >> 5);
    const int I0 = blockIdx.y * chunk, I1 = min(G.nout[0], I0 + chunk);
    if (J >= G.nout[1] || L >= G.nout[2]) return;
    const double* a = in + (long long)blockIdx.z * n0 * n1 * n2;
    const long long ops = (long long)G.nout[1] * G.nout[2];
    const long long oat = (long long)blockIdx.z * G.nout[0] * ops + (long long)J * G.nout[2] + L;

    int col[3];      // centre, +1, -1
#pragma unroll
    for (int k = 0; k < 3; k++) {
        col[k] = 2 * L + 1 - G.plo[2] + (k == 0 ? 0 : k == 1 ? 1 : -1);
        if (!wrap2(col[k], n2, G.g.periodic[2])) col[k] = -1;
    }
    int row[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        int r = 2 * J - G.plo[1] + k;
        row[k] = wrap2(r, n1, G.g.periodic[1]) ? r * n2 : -1;
    }
    // in-plane restriction of fine plane f at this lane's point
    auto plane = [&](int f) {
        const bool ok = wrap2(f, n0, G.g.periodic[0]);
        const double* p = a + (long long)(ok ? f : 0) * n1 * n2;
        double v[3][3];
#pragma unroll
        for (int k = 0; k < 3; k++)
#pragma unroll
            for (int c = 0; c < 3; c++)
                v[k][c] = ok && (row[k] | col[c]) >= 0 ? __ldg(p + row[k] + col[c])
                                                       : Num<double>::zero();
        double t[3];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            t[k] = mid(v[k][0], v[k][1], v[k][2], G.w[0]);
            if (G.neg_in) t[k] = Num<double>::neg(t[k]);
        }
        return mid(t[1], t[2], t[0], G.w[0]);
    };
    double um = plane(2 * I0 - G.plo[0]);
    for (int I = I0; I < I1; I++) {
        const double uc = plane(2 * I + 1 - G.plo[0]);
        const double up = plane(2 * I + 2 - G.plo[0]);
        const double r = mid(uc, up, um, G.w[0]);
        const long long at = oat + I * ops;
        out[at] = r;
        if (out2) out2[at] = Num<double>::scale(r, G.scale2);
        um = up;
    }
}

__global__ void __launch_bounds__(256)
k_interp2(const double* __restrict__ in, double* __restrict__ out, XferGeom G, int chunk,
          int pairs0, int pairs1, int pairs2, int tiles2) {
    const int n0 = G.g.n[0], n1 = G.g.n[1], n2 = G.g.n[2];
    // padded coarse column and row of this lane; each gives the fine points
    // 2 m - skip and 2 m + 1 - skip
    const int M2 = blockIdx.x % tiles2 * 32 + (threadIdx.x & 31);
    const int M1 = blockIdx.x / tiles2 * 8 + (threadIdx.x >> 5);
    const int ia = blockIdx.y * chunk, ib = min(pairs0, ia + chunk);
    if (M1 >= pairs1 || M2 >= pairs2) return;
    const double* a = in + (long long)blockIdx.z * n0 * n1 * n2;
    double* o = out + (long long)blockIdx.z * G.nout[0] * G.nout[1] * G.nout[2];

    int col[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        col[k] = M2 + k - G.plo[2];
        if (M2 + k >= G.s[2] || !wrap2(col[k], n2, G.g.periodic[2])) col[k] = -1;
    }
    int row[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        int r = M1 + k - G.plo[1];
        row[k] = M1 + k < G.s[1] && wrap2(r, n1, G.g.periodic[1]) ? r * n2 : -1;
    }
    // fine rows and columns of this lane that exist
    const int f1 = 2 * M1 - G.skip0[1], f2 = 2 * M2 - G.skip0[2];
    bool ok1[2], ok2[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        ok1[k] = f1 + k >= 0 && f1 + k < G.nout[1];
        ok2[k] = f2 + k >= 0 && f2 + k < G.nout[2];
    }
    const long long ops = (long long)G.nout[1] * G.nout[2];
    const long long oat = (long long)f1 * G.nout[2] + f2;

    // in-plane interpolation of padded coarse plane m
    auto plane = [&](int m, double (&q)[2][2]) {
        int f = m - G.plo[0];
        const bool ok = m < G.s[0] && wrap2(f, n0, G.g.periodic[0]);
        const double* p = a + (long long)(ok ? f : 0) * n1 * n2;
        double v[2][2];
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int c = 0; c < 2; c++)
                v[k][c] = ok && (row[k] | col[c]) >= 0 ? __ldg(p + row[k] + col[c])
                                                       : Num<double>::zero();
#pragma unroll
        for (int k = 0; k < 2; k++) {
            v[k][1] = Num<double>::scale(Num<double>::add(v[k][0], v[k][1]), G.w[0]);
            if (G.neg_in) {
                v[k][0] = Num<double>::neg(v[k][0]);
                v[k][1] = Num<double>::neg(v[k][1]);
            }
        }
#pragma unroll
        for (int c = 0; c < 2; c++) {
            q[0][c] = v[0][c];
            q[1][c] = Num<double>::scale(Num<double>::add(v[0][c], v[1][c]), G.w[0]);
        }
    };
    auto emit = [&](int u, const double (&q)[2][2]) {
        const int f0 = u - G.skip0[0];
        if (f0 < 0 || f0 >= G.nout[0]) return;
        double* d = o + f0 * ops + oat;
        if (G.accumulate) {
            double old[2][2];
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int c = 0; c < 2; c++)
                    if (ok1[k] && ok2[c]) old[k][c] = d[(long long)k * G.nout[2] + c];
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int c = 0; c < 2; c++)
                    if (ok1[k] && ok2[c])
                        d[(long long)k * G.nout[2] + c] = Num<double>::sub(old[k][c], q[k][c]);
        } else {
#pragma unroll
            for (int k = 0; k < 2; k++)
#pragma unroll
                for (int c = 0; c < 2; c++)
                    if (ok1[k] && ok2[c]) d[(long long)k * G.nout[2] + c] = q[k][c];
        }
    };
    double q[2][2], r[2][2];
    plane(ia, q);
    for (int i = ia; i < ib; i++) {
        plane(i + 1, r);
        emit(2 * i, q);
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int c = 0; c < 2; c++)
                q[k][c] = Num<double>::scale(Num<double>::add(q[k][c], r[k][c]), G.w[0]);
        emit(2 * i + 1, q);
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
            for (int c = 0; c < 2; c++) q[k][c] = r[k][c];
    }
}

void run_restrict(const double* in, double* out, double* out2, int nin, const XferGeom& G,
                cudaStream_t st) {
    const int tiles2 = (G.nout[2] + 31) / 32;
    const int tiles = tiles2 * ((G.nout[1] + 7) / 8);
    const int chunk = G.chunk > 0
                          ? std::min(G.chunk, G.nout[0])
                          : balance_planes(G.nout[0], 2, 1, (long long)tiles * nin, 4, 0.25, 0.5);
    const long long ngin = (long long)G.g.n[0] * G.g.n[1] * G.g.n[2];
    const long long ngout = (long long)G.nout[0] * G.nout[1] * G.nout[2];
    for (int b0 = 0; b0 < nin; b0 += 65535)
        k_restrict2<<<dim3(tiles, (G.nout[0] + chunk - 1) / chunk, std::min(65535, nin - b0)), 256,
                      0, st>>>(in + b0 * ngin, out + b0 * ngout,
                               out2 ? out2 + b0 * ngout : nullptr, G, chunk, tiles2);
}

void run_interp(const double* in, double* out, int nin, const XferGeom& G, cudaStream_t st) {
    int pairs[3];
    for (int c = 0; c < 3; c++) pairs[c] = G.s[c] - 1 + G.skip1[c];
    const int tiles2 = (pairs[2] + 31) / 32;
    const int tiles = tiles2 * ((pairs[1] + 7) / 8);
    const int chunk = G.chunk > 0 ? std::min(G.chunk, pairs[0])
                                  : balance_planes(pairs[0], 1, 1, (long long)tiles * nin, 3,
                                                   0.4, 0.5);
    const long long ngin = (long long)G.g.n[0] * G.g.n[1] * G.g.n[2];
    const long long ngout = (long long)G.nout[0] * G.nout[1] * G.nout[2];
    for (int b0 = 0; b0 < nin; b0 += 65535)
        k_interp2<<<dim3(tiles, (pairs[0] + chunk - 1) / chunk, std::min(65535, nin - b0)), 256, 0,
                    st>>>(in + b0 * ngin, out + b0 * ngout, G, chunk, pairs[0], pairs[1], pairs[2],
                          tiles2);
}

}  // namespace

int launch_transfer2(bool interpolate, const double* in, double* out, double* out2, int nin,
                     const XferGeom& G, cudaStream_t st) {
    if ((long long)G.g.n[1] * G.g.n[2] >= (1ll << 31) ||
        (long long)G.nout[1] * G.nout[2] >= (1ll << 31))
        return -1;
    if (interpolate) run_interp(in, out, nin, G, st);
    else run_restrict(in, out, out2, nin, G, st);
    return 0;
}

}  // namespace gb
