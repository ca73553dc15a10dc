// The coarse levels of an FP64 multigrid V-cycle (iterate2 from some level
// on, gpaw/poisson.py:500-537, starting from phi = 0) in one launch, for the
// plain and the weighted (dielectric) operator: weighted-Jacobi sweeps, the
// residual, the K = 2 restriction and interpolation (axis 2, then 1, then 0,
// c/bmgs/restrict.cpp:137-156, c/bmgs/interpolate.cpp:70-99).  Every value is
// computed with the same operations in the same order as by the per-level
// kernels, so the V-cycle is bit-identical to them.
//
// What bounds it: a chain of some fifty dependent passes over 31^3 points and
// fewer, each well under a microsecond of work but three and more as a launch
// of its own (launch, ramp, drain).  One thread block cluster of 16 CTAs
// (one GPC) runs them back to back: its hardware barrier replaces the kernel
// boundary, and the levels' arrays, a megabyte, stay in L2.  A level of at
// most 1024 points is left to the first CTA alone, with block barriers and
// its L1.  A thread keeps its points of a level in registers through the
// level's sweeps: coordinates, value, right-hand side, weights.  A sweep that
// starts from zero reads no neighbours.
// 63^3 grid (levels 31^3 .. 1^3): 80 us a V-cycle (dielectric 104) against 12
// launches for 31^3 and a 54 us single-CTA kernel for 15^3 down, about 105 us.
// After other work, the levels no longer in L2: about 108 (dielectric 136).
#include "gb_coarse.cuh"
#include "gb_objects.cuh"

namespace gb {
namespace {

constexpr int CT = 512;         // threads of a CTA
constexpr int LOCAL_POINTS = 1024;
constexpr int MAXP = 4;         // points a thread

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive;\n" ::: "memory");
    asm volatile("barrier.cluster.wait;\n" ::: "memory");
}
template <bool LOCAL>
__device__ __forceinline__ void sync_all() {
    if (LOCAL) __syncthreads();
    else cluster_sync();
}
// values that other CTAs wrote in this launch come from L2; a level of one
// CTA's own from its L1
template <bool LOCAL>
__device__ __forceinline__ double get(const double* p) {
    return LOCAL ? *p : __ldcg(p);
}

// a / b correctly rounded, from y = RN(1 / b): q = RN(a y) corrected twice by
// its exact remainder (P. Markstein, IBM J. Res. Dev. 34, 111 (1990): the
// first correction is within an ulp, the second rounds correctly); outside
// the range where the remainders are exact, the division itself.
__device__ __forceinline__ double quotient(double a, double b, double y) {
    const double m = fabs(a);
    if (!(m > 1e-200 && m < 1e200)) return __ddiv_rn(a, b);
    double q = __dmul_rn(a, y);
    q = __fma_rn(__fma_rn(-b, q, a), y, q);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}

// index along one axis after the boundary condition; -1 reads zero
__device__ __forceinline__ int at_axis(int j, int n, int per) {
    if (j >= 0 && j < n) return j;
    if (!per) return -1;
    j = j < 0 ? j + n : j - n;
    return (j >= 0 && j < n) ? j : -1;
}
__device__ __forceinline__ void split(int p, int n1, int n2, int& i0, int& i1, int& i2) {
    i0 = p / (n1 * n2);
    p -= i0 * n1 * n2;
    i1 = p / n2;
    i2 = p - i1 * n2;
}

// this thread's points of a level: first, first + stride, ...
struct Points {
    int n, first, stride;
    int nb[MAXP][6];          // neighbours +1, -1 along axis 2, 1, 0; -1: zero
    double v[MAXP], r[MAXP];
};

template <bool LOCAL>
__device__ __forceinline__ void take(Points& P, const CoarseLevel& L, int first, int stride) {
    P.n = 0;
    P.first = first;
    P.stride = stride;
    const int n1 = L.n[1], n2 = L.n[2];
#pragma unroll
    for (int k = 0; k < MAXP; k++) {
        const int p = first + k * stride;
        if (p >= L.ng) continue;
        P.n = k + 1;
        int i[3], s = 1;
        split(p, n1, n2, i[0], i[1], i[2]);
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const int c = 2 - d, n = L.n[c];
            const int up = at_axis(i[c] + 1, n, L.per[c]), dn = at_axis(i[c] - 1, n, L.per[c]);
            P.nb[k][2 * d] = up < 0 ? -1 : p + (up - i[c]) * s;
            P.nb[k][2 * d + 1] = dn < 0 ? -1 : p + (dn - i[c]) * s;
            s *= n;
        }
        P.r[k] = get<LOCAL>(L.rho + p);
    }
}
// the weights of point p (constant during the launch: from L1)
template <bool W>
__device__ __forceinline__ void weights(double (&w)[4], const CoarseLevel& L, int p) {
    if (W)
#pragma unroll
        for (int q = 0; q < 4; q++) w[q] = __ldg(L.w[q] + p);
}

// The operator at a point with value v and neighbours a (+1, -1 along axis
// 2, 1, 0).  CENTRE: with the centre taps (the apply), else without (the
// off-diagonal part of a sweep).
template <bool W, bool CENTRE>
__device__ __forceinline__ double stencil(const CoarseLevel& L, double v, const double (&a)[6],
                                          const double* w) {
    double x = 0.0;
    if (CENTRE) x = __dadd_rn(x, __dmul_rn(v, L.c0));
#pragma unroll
    for (int d = 0; d < 3; d++) {
        x = __dadd_rn(x, __dmul_rn(a[2 * d], L.cp[d]));
        x = __dadd_rn(x, __dmul_rn(a[2 * d + 1], L.cm[d]));
    }
    if (!W) return x;
    double t = __dadd_rn(0.0, __dmul_rn(x, w[0]));
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const int ax = L.gaxis[i];
        const double up = ax == 0 ? a[4] : ax == 1 ? a[2] : a[0];
        const double dn = ax == 0 ? a[5] : ax == 1 ? a[3] : a[1];
        double y = 0.0;
        if (CENTRE) y = __dadd_rn(y, __dmul_rn(v, L.gc0[i]));
        y = __dadd_rn(y, __dmul_rn(up, L.gp[i]));
        y = __dadd_rn(y, __dmul_rn(dn, L.gm[i]));
        t = __dadd_rn(t, __dmul_rn(y, w[i + 1]));
    }
    return t;
}
template <bool W>
__device__ __forceinline__ double diagonal(const CoarseLevel& L, const double* w) {
    if (!W) return L.c0;
    double d = __dadd_rn(0.0, __dmul_rn(w[0], L.c0));
#pragma unroll
    for (int i = 0; i < 3; i++) d = __dadd_rn(d, __dmul_rn(w[i + 1], L.gc0[i]));
    return d;
}

// n sweeps of the values in P.v, which buffer `cur` holds (`zero`: they are
// zero, and nothing holds them); returns the buffer with the result
template <bool W, bool LOCAL>
__device__ __forceinline__ double* relax(const CoarseLevel& L, Points& P, double* cur, int n,
                                         bool zero) {
    const double w1 = 1.0 - L.wj;
    for (int it = 0; it < n; it++) {
        const double* A = cur;
        cur = cur == L.phi ? L.tmp : L.phi;
        double a[MAXP][6];
#pragma unroll
        for (int k = 0; k < MAXP; k++)
#pragma unroll
            for (int d = 0; d < 6; d++)
                a[k][d] = k < P.n && P.nb[k][d] >= 0 && !(zero && it == 0)
                              ? get<LOCAL>(A + P.nb[k][d]) : 0.0;
#pragma unroll
        for (int k = 0; k < MAXP; k++)
            if (k < P.n) {
                double w[4];
                weights<W>(w, L, P.first + k * P.stride);
                const double x = stencil<W, false>(L, P.v[k], a[k], w);
                const double num = __dmul_rn(L.wj, __dsub_rn(P.r[k], x));
                const double q = W ? __ddiv_rn(num, diagonal<W>(L, w))
                                   : quotient(num, L.c0, L.rc0);
                P.v[k] = __dadd_rn(__dmul_rn(w1, P.v[k]), q);
                cur[P.first + k * P.stride] = P.v[k];
            }
        sync_all<LOCAL>();
    }
    return cur;
}

// mid-point restriction of one line, K = 2: 0.5 (a + w (a+ + a-))
__device__ __forceinline__ double middle(double v, double vp, double vm, double w) {
    return __dmul_rn(0.5, __dadd_rn(v, __dmul_rn(w, __dadd_rn(vp, vm))));
}

template <bool LOCAL>
__device__ __forceinline__ void restrict_to(const CoarseLevel& F, const CoarseLevel& C,
                                            const double* A, int first, int stride) {
    const int n1 = F.n[1], n2 = F.n[2];
    for (int p = first; p < C.ng; p += stride) {
        int c[3], j[3][3];     // per axis: the centre, +1, -1
        split(p, C.n[1], C.n[2], c[0], c[1], c[2]);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int m = 2 * c[a] + 1 - F.rplo[a];
            j[a][0] = at_axis(m, F.n[a], F.per[a]);
            j[a][1] = at_axis(m + 1, F.n[a], F.per[a]);
            j[a][2] = at_axis(m - 1, F.n[a], F.per[a]);
        }
        double v[3][3][3];
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++)
#pragma unroll
                for (int e = 0; e < 3; e++)
                    v[a][b][e] = (j[0][a] | j[1][b] | j[2][e]) < 0
                                     ? 0.0
                                     : get<LOCAL>(A + (j[0][a] * n1 + j[1][b]) * n2 + j[2][e]);
        double u[3];
#pragma unroll
        for (int a = 0; a < 3; a++) {
            double t[3];
#pragma unroll
            for (int b = 0; b < 3; b++) t[b] = middle(v[a][b][0], v[a][b][1], v[a][b][2], F.rw);
            u[a] = middle(t[0], t[1], t[2], F.rw);
        }
        C.rho[p] = middle(u[0], u[1], u[2], F.rw);
    }
}

// P.v -= interpolation of the next level's phi: per axis (2, 1, 0) an even
// fine index copies, an odd one is w (a(k) + a(k+1)) (c/bmgs/interpolate.cpp:
// 10-46, K = 2)
template <bool LOCAL>
__device__ __forceinline__ void interpolate_sub(const CoarseLevel& F, const CoarseLevel& C,
                                                Points& P) {
    const int m1 = C.n[1], m2 = C.n[2];
#pragma unroll
    for (int k = 0; k < MAXP; k++) {
        if (k >= P.n) break;
        int f[3], j[3][2];
        bool odd[3];
        split(P.first + k * P.stride, F.n[1], F.n[2], f[0], f[1], f[2]);
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const int u = f[a] + F.iskip[a];
            odd[a] = u & 1;
            j[a][0] = at_axis((u >> 1) - F.iplo[a], C.n[a], C.per[a]);
            j[a][1] = odd[a] ? at_axis((u >> 1) + 1 - F.iplo[a], C.n[a], C.per[a]) : -1;
        }
        double v[2][2][2];
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int e = 0; e < 2; e++)
                    v[a][b][e] = (j[0][a] | j[1][b] | j[2][e]) < 0
                                     ? 0.0
                                     : get<LOCAL>(C.phi + (j[0][a] * m1 + j[1][b]) * m2 + j[2][e]);
        double q[2];
#pragma unroll
        for (int a = 0; a < 2; a++) {
            double l[2];
#pragma unroll
            for (int b = 0; b < 2; b++)
                l[b] = odd[2] ? __dmul_rn(F.iw, __dadd_rn(v[a][b][0], v[a][b][1])) : v[a][b][0];
            q[a] = odd[1] ? __dmul_rn(F.iw, __dadd_rn(l[0], l[1])) : l[0];
        }
        const double x = odd[0] ? __dmul_rn(F.iw, __dadd_rn(q[0], q[1])) : q[0];
        P.v[k] = __dsub_rn(P.v[k], x);
    }
}

__device__ __forceinline__ double* other(const CoarseLevel& L, double* b) {
    return b == L.phi ? L.tmp : L.phi;
}
// the buffer a level starts in, so that all its sweeps end in phi
__device__ __forceinline__ double* start(const CoarseLevel& L, bool last) {
    const int flips = last ? L.post : L.pre + L.post;
    return (flips & 1) ? L.tmp : L.phi;
}
template <bool LOCAL>
__device__ __forceinline__ void fill_zero(Points& P, double* b) {
#pragma unroll
    for (int k = 0; k < MAXP; k++)
        if (k < P.n) b[P.first + k * P.stride] = 0.0;
    sync_all<LOCAL>();
}

template <bool W, bool LOCAL>
__device__ __forceinline__ void go_down(const CoarseLevel& L, const CoarseLevel& C, int first,
                                        int stride) {
    Points P;
    take<LOCAL>(P, L, first, stride);
#pragma unroll
    for (int k = 0; k < MAXP; k++) P.v[k] = 0.0;
    double* cur = start(L, false);
    if (L.pre == 0) fill_zero<LOCAL>(P, cur);
    cur = relax<W, LOCAL>(L, P, cur, L.pre, true);
    double* res = other(L, cur);
#pragma unroll
    for (int k = 0; k < MAXP; k++)
        if (k < P.n) {
            double a[6], w[4];
            weights<W>(w, L, first + k * stride);
#pragma unroll
            for (int d = 0; d < 6; d++)
                a[d] = P.nb[k][d] >= 0 ? get<LOCAL>(cur + P.nb[k][d]) : 0.0;
            res[first + k * stride] =
                __dsub_rn(stencil<W, true>(L, P.v[k], a, w), P.r[k]);
        }
    sync_all<LOCAL>();
    restrict_to<LOCAL>(L, C, res, first, stride);
    sync_all<LOCAL>();
}

template <bool W, bool LOCAL>
__device__ __forceinline__ void go_up(const CoarseLevel& L, const CoarseLevel* C, int first,
                                      int stride) {
    Points P;
    take<LOCAL>(P, L, first, stride);
    double* cur = start(L, !C);
    if (!C) {
#pragma unroll
        for (int k = 0; k < MAXP; k++) P.v[k] = 0.0;
        if (L.post == 0) fill_zero<LOCAL>(P, cur);
        relax<W, LOCAL>(L, P, cur, L.post, true);
        return;
    }
    if (L.pre & 1) cur = other(L, cur);
#pragma unroll
    for (int k = 0; k < MAXP; k++) P.v[k] = k < P.n ? get<LOCAL>(cur + first + k * stride) : 0.0;
    interpolate_sub<LOCAL>(L, *C, P);
#pragma unroll
    for (int k = 0; k < MAXP; k++)
        if (k < P.n) cur[first + k * stride] = P.v[k];
    sync_all<LOCAL>();
    relax<W, LOCAL>(L, P, cur, L.post, false);
}

template <bool W>
__global__ void __launch_bounds__(CT, 1) k_coarse(const __grid_constant__ CoarsePlan plan) {
    const int rank = blockIdx.x, tid = threadIdx.x;
    const int first = rank * CT + tid, stride = gridDim.x * CT;
    const int last = plan.nl - 1;
    int shared = 0;              // levels that the whole cluster works on
    while (shared < plan.nl && plan.lv[shared].ng > LOCAL_POINTS) shared++;
    for (int l = 0; l < min(shared, last); l++)
        go_down<W, false>(plan.lv[l], plan.lv[l + 1], first, stride);
    if (shared == plan.nl) go_up<W, false>(plan.lv[last], nullptr, first, stride);
    else {
        if (rank == 0) {
            for (int l = shared; l < last; l++)
                go_down<W, true>(plan.lv[l], plan.lv[l + 1], tid, CT);
            for (int l = last; l >= shared; l--)
                go_up<W, true>(plan.lv[l], l == last ? nullptr : &plan.lv[l + 1], tid, CT);
        }
        cluster_sync();
    }
    for (int l = min(shared, last) - 1; l >= 0; l--)
        go_up<W, false>(plan.lv[l], &plan.lv[l + 1], first, stride);
}

// CTAs of the cluster: 16 where the device schedules such a cluster, else 8
// (the portable size)
template <bool W>
int cluster_size() {
    static const int size = [] {
        cudaFuncSetAttribute(k_coarse<W>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        for (int c : {16, 8}) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(c);
            cfg.blockDim = dim3(CT);
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = c;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, k_coarse<W>, &cfg) == cudaSuccess && n > 0)
                return c;
            cudaGetLastError();
        }
        return 0;
    }();
    return size;
}

template <bool W>
int launch(const CoarsePlan& plan, cudaStream_t st) {
    const int c = cluster_size<W>();
    if (c == 0) return fail(GB_ECUDA, "coarse levels: no cluster of 8 CTAs fits the device");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(CT);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    GB_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_coarse<W>, plan));
    return 0;
}

}  // namespace

bool coarse_transfers(CoarseLevel& L, int kr, const XferGeom& r, int ki, const XferGeom& i,
                      const int* ncoarse) {
    if (kr != 2 || ki != 2) return false;
    for (int c = 0; c < 3; c++) {
        if (r.g.n[c] != L.n[c] || r.g.periodic[c] != L.per[c] || r.nout[c] != ncoarse[c] ||
            i.g.n[c] != ncoarse[c] || i.g.periodic[c] != L.per[c] || i.nout[c] != L.n[c])
            return false;
        L.rplo[c] = r.plo[c];
        L.iplo[c] = i.plo[c];
        L.iskip[c] = i.skip0[c];
    }
    L.rw = r.w[0];
    L.iw = i.w[0];
    return true;
}

int coarse_points(bool weighted) {
    return (weighted ? cluster_size<true>() : cluster_size<false>()) * CT * MAXP;
}

int launch_coarse(const CoarsePlan& plan, bool weighted, cudaStream_t st) {
    return weighted ? launch<true>(plan, st) : launch<false>(plan, st);
}

}  // namespace gb
