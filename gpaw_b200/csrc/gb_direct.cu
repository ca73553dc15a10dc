// Direct correction of the mixed Poisson solver: e = L^-1 d in FP64 by fast
// diagonalisation (R. E. Lynch, J. R. Rice, D. H. Thomas, Numer. Math. 6,
// 185 (1964)).
//
// The level-0 operator of an orthorhombic grid is a sum of one-dimensional
// stencils, L = T0 + T1 + T2, so L^-1 = Q diag(1 / (l0 + l1 + l2)) Q^T with
// Q = Q0 x Q1 x Q2 the eigenvectors of each axis's n x n matrix.  One
// correction is six products with those matrices: forward along axis 2, 1,
// 0, the division, and back along 0, 1, 2.  It solves the discrete problem
// to rounding, so the defect-correction loop around it stops after one
// correction (a second only repairs rounding), where the FP32 V-cycles need
// about fourteen of some thirty passes each.
//
// Folding: every axis matrix commutes with the reflection j <-> n - 1 - j
// (zero boundary) or j <-> -j (periodic), so its eigenvectors are even or
// odd.  Sums and differences of mirrored points give two products of half
// the size: half the multiplications.
//
// Work: n0 n1 n2 (n0 + n1 + n2) FP64 fused multiply-adds a correction (4.0 G
// on 191^3); bound by the FP64 pipe (64 a clock and SM).  A CTA takes 64
// grid lines and keeps them in shared memory (98 KB at n = 191: two CTAs an
// SM, one loads while the other multiplies), folded in place; a warp owns 12
// output rows x 64 lines, a thread 6 x 4 of them: 24 multiply-adds for 3
// 16-byte and 4 8-byte shared reads that touch 2 x 16 and 16 x 8 distinct
// bytes.  The warp's slice of the matrix streams from L2 through a private
// two-stage ring of cp.async copies, so the product needs no block barrier.
// The middle kernel does the forward axis-0 product, the division and the
// backward product on lines that never leave the CTA; every pass is in
// place.
//
// All kernels serve a group of grids (a batch) at once: block -> (grid,
// lines) through a table; blocks of converged grids return at once.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <utility>
#include <vector>

#include "gb_direct.cuh"
#include "gb_direct_host.cuh"
#include "gb_objects.cuh"

namespace gb {
namespace {

constexpr int CH = 8;                          // matrix columns a ring stage holds
constexpr int STAGE = CH * DIR_KT;             // doubles

enum : int { F2 = 0, F1 = 1, M0 = 2, B1 = 3, B2 = 4 };

// 8 columns x 12 rows of a warp's matrix slice: 48 copies of 16 bytes
__device__ __forceinline__ void stage_table(double* ring, const double* tab, int lane) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(ring);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + 16 * lane),
                 "l"(tab + 2 * lane));
    if (lane < 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + 16 * (lane + 32)),
                     "l"(tab + 2 * (lane + 32)));
    asm volatile("cp.async.commit_group;\n" ::);
}

__device__ __forceinline__ void copy8(double* dst, const double* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(
                     (unsigned)__cvta_generic_to_shared(dst)),
                 "l"(src));
}

// acc[i][v] = sum_j tab[j][6 h + i] A[j * ap][l + 16 v], with h and l the
// half-warp and the lane in it; the first chunk was staged into ring[0] by
// the caller (and is the latest or the only pending copy group but the
// caller's empty ones)
__device__ __forceinline__ void product(double (&acc)[6][4], const double* tab, int kp,
                                        const double* A, int ap, double* ring, int lane) {
#pragma unroll
    for (int i = 0; i < 6; i++)
#pragma unroll
        for (int v = 0; v < 4; v++) acc[i][v] = 0.0;
    const int nc = kp / CH;
    const double* a = A + (lane & 15);
    for (int c = 0; c < nc; c++) {
        if (c + 1 < nc)
            stage_table(ring + ((c + 1) & 1) * STAGE, tab + (size_t)(c + 1) * STAGE, lane);
        else
            asm volatile("cp.async.commit_group;\n" ::);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncwarp();
        const double* t = ring + (c & 1) * STAGE + 6 * (lane >> 4);
#pragma unroll
        for (int j = 0; j < CH; j++) {
            double x[4];
#pragma unroll
            for (int v = 0; v < 4; v++) x[v] = a[16 * v];
            a += ap;
#pragma unroll
            for (int i = 0; i < 6; i += 2) {
                const double2 m = *reinterpret_cast<const double2*>(t + j * DIR_KT + i);
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    acc[i][v] = fma(m.x, x[v], acc[i][v]);
                    acc[i + 1][v] = fma(m.y, x[v], acc[i + 1][v]);
                }
            }
        }
        __syncwarp();
    }
}

// rows of the line block in shared memory: the n points; when a padded half
// would reach past them (n < 15), the odd half gets rows of its own
__host__ __device__ __forceinline__ int dir_rows(const DirAxis& a) {
    if (a.kpe <= a.n && a.kpo <= a.n) return a.n;
    return (a.kpe > a.n ? a.kpe : a.n) + a.kpo;
}

// One pass over the lines along one axis.  The block S[row][line] holds the
// points j (load), then the folded halves: even index j in row j, odd index
// q in row R - 1 - q (where its mirror point was), then the modes in the
// same rows, and back.  TWO: the even half is multiplied first, then the
// odd one (a warp has a tile of each); otherwise different warps take them
// side by side.
template <int PASS, int NW, bool TWO>
__global__ void __launch_bounds__(32 * NW, NW >= 16 ? 1 : 16 / NW)
k_direct(const DirGrid* __restrict__ grids, const DirCtl* ctl, const DirBlock* __restrict__ map) {
    constexpr int AX = (PASS == F2 || PASS == B2) ? 2 : PASS == M0 ? 0 : 1;
    constexpr int NT = 32 * NW, NJ = NT / DIR_W;
    constexpr bool FWD = PASS == F2 || PASS == F1 || PASS == M0;
    DirBlock bk{0, (int)blockIdx.x};
    if (map) bk = map[blockIdx.x];
    if (!ctl[bk.grid].active) return;
    const DirGrid& G = grids[bk.grid];
    const DirAxis& ax = G.ax[AX];
    const int n = ax.n, he = ax.he, ho = ax.ho, kpe = ax.kpe, kpo = ax.kpo;
    const int off = ax.per ? 1 : 0;         // odd index q: points q + off and mir - q - off
    const int mir = ax.per ? n : n - 1;
    const int R = dir_rows(ax);
    const int n1 = G.n[1], n2 = G.n[2];
    const long long lines = (long long)G.n[0] * n1 * n2 / n;
    const long long q0 = (long long)bk.block * DIR_W;
    const int nl = (int)min((long long)DIR_W, lines - q0);
    extern __shared__ __align__(16) double dir_smem[];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    double* ring = dir_smem + wid * 2 * STAGE;   // rings first: 16-byte aligned
    double* S = dir_smem + NW * 2 * STAGE;
    double* const SO = S + (size_t)(R - 1) * DIR_P;   // odd index q: SO - q * DIR_P
    double* X = G.X;

    // this warp's tiles (12 rows of one half)
    const int nte = (he + DIR_KT - 1) / DIR_KT;
    const int tile_o = TWO ? wid : wid - nte;
    const bool has_e = wid * DIR_KT < he;
    const bool has_o = tile_o >= 0 && tile_o * DIR_KT < ho;
    const double* te = (FWD ? ax.fe : ax.be) + (size_t)wid * kpe * DIR_KT;
    const double* to = (FWD ? ax.fo : ax.bo) + (size_t)(TWO ? wid : max(tile_o, 0)) * kpo * DIR_KT;

    // ---- load.  Line w starts at base and runs with stride s (axes 0, 1)
    const long long s = AX == 0 ? (long long)n1 * n2 : n2;
    const int w = tid & (DIR_W - 1), jl = tid / DIR_W;
    long long base = 0;
    if (AX == 0) base = q0 + w;
    else if (AX == 1) {
        const long long q = q0 + w;
        base = q / n2 * ((long long)n1 * n2) + q % n2;
    }
    // modes are stored even first: mode k >= he is odd index k - he
    if (R > n || nl < DIR_W) {
        for (int e = tid; e < R * DIR_P; e += NT) S[e] = 0.0;
        __syncthreads();
    }
    if constexpr (AX != 2) {
        if (w < nl) {
            const double* src = X + base + jl * s;
            double* d = S + jl * DIR_P + w;
            if constexpr (FWD) {
                for (int j = jl; j < n; j += NJ, src += NJ * s, d += NJ * DIR_P) copy8(d, src);
            } else {
                for (int j = jl; j < n; j += NJ, src += NJ * s, d += NJ * DIR_P)
                    copy8(j < he ? d : SO - (j - he) * DIR_P + w, src);
            }
        }
    } else {
        for (int r = wid; r < nl; r += NW) {
            const double* row = X + (q0 + r) * n;
            for (int j = lane; j < n; j += 32)
                copy8(FWD || j < he ? S + j * DIR_P + r : SO - (j - he) * DIR_P + r, row + j);
        }
    }
    asm volatile("cp.async.commit_group;\n" ::);
    if (TWO || has_e) {
        if (has_e) stage_table(ring, te, lane);
    } else if (has_o) {
        stage_table(ring, to, lane);
    }
    if (has_e || (!TWO && has_o))
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    else
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    if constexpr (FWD) {
        for (int q = jl; q < ho; q += NJ) {
            double* e = S + (q + off) * DIR_P + w;
            double* o = SO - q * DIR_P + w;
            const double a = *e, b = S[(mir - q - off) * DIR_P + w];
            *e = a + b;
            *o = a - b;
        }
        __syncthreads();
    }

    // ---- products, written over their own input once every warp read it
    const int l = lane & 15, h6 = 6 * (lane >> 4);
    const int ke = wid * DIR_KT + h6, ko = tile_o * DIR_KT + h6;
    double acc[6][4];
    auto put = [&](double* D, int pitch, int k0, int h) {
#pragma unroll
        for (int i = 0; i < 6; i++)
            if (k0 + i < h)
#pragma unroll
                for (int v = 0; v < 4; v++) D[(k0 + i) * pitch + l + 16 * v] = acc[i][v];
    };
    // M0: modes divided by their eigenvalue; a singular mode is left out
    auto divide = [&](const double* lam, int k0, int h) {
        double l12[4];
#pragma unroll
        for (int v = 0; v < 4; v++) {
            const int q = (int)min(q0 + l + 16 * v, lines - 1);
            l12[v] = G.ax[1].lam[q / n2] + G.ax[2].lam[q % n2];
        }
#pragma unroll
        for (int i = 0; i < 6; i++) {
            const double l0 = k0 + i < h ? lam[k0 + i] : 1.0;
#pragma unroll
            for (int v = 0; v < 4; v++) {
                const double x = l0 + l12[v];
                acc[i][v] = fabs(x) > G.tiny ? acc[i][v] / x : 0.0;
            }
        }
    };
    // both halves through tables ea and oa (the first chunk of the first
    // product staged); `next`: stage the first chunk of the following product
    auto halves = [&](const double* ea, const double* oa, bool div, const double* next_e,
                      const double* next_o) {
        if constexpr (TWO) {
            if (has_e) {
                product(acc, ea, kpe, S, DIR_P, ring, lane);
                if (has_o) stage_table(ring, oa, lane);
                if (div) divide(ax.lam, ke, he);
            }
            __syncthreads();
            if (has_e) put(S, DIR_P, ke, he);
            __syncthreads();    // the odd half's padding reads even rows (times zero)
            if (has_o) {
                product(acc, oa, kpo, SO, -DIR_P, ring, lane);
                if (div) divide(ax.lam + he, ko, ho);
            }
            if (next_e && has_e) stage_table(ring, next_e, lane);
            __syncthreads();
            if (has_o) put(SO, -DIR_P, ko, ho);
        } else {
            if (has_e) {
                product(acc, ea, kpe, S, DIR_P, ring, lane);
                if (next_e) stage_table(ring, next_e, lane);
                if (div) divide(ax.lam, ke, he);
            } else if (has_o) {
                product(acc, oa, kpo, SO, -DIR_P, ring, lane);
                if (next_o) stage_table(ring, next_o, lane);
                if (div) divide(ax.lam + he, ko, ho);
            }
            __syncthreads();
            if (has_e) put(S, DIR_P, ke, he);
            else if (has_o) put(SO, -DIR_P, ko, ho);
        }
        __syncthreads();
    };
    if constexpr (PASS == M0) {
        const double* be = ax.be + (size_t)wid * kpe * DIR_KT;
        const double* bo = ax.bo + (size_t)(TWO ? wid : max(tile_o, 0)) * kpo * DIR_KT;
        halves(te, to, true, be, bo);
        halves(be, bo, false, nullptr, nullptr);
    } else {
        halves(te, to, false, nullptr, nullptr);
    }

    // ---- store: modes (forward) or unfolded points (backward)
    if constexpr (PASS != F2 && PASS != F1) {
        for (int q = jl; q < ho; q += NJ) {
            double* e = S + (q + off) * DIR_P + w;
            const double a = *e, b = SO[-q * DIR_P + w];
            *e = a + b;
            S[(mir - q - off) * DIR_P + w] = a - b;
        }
        __syncthreads();
    }
    constexpr bool MODES = PASS == F2 || PASS == F1;
    auto at = [&](int j) { return MODES && j >= he ? SO - (j - he) * DIR_P : S + j * DIR_P; };
    if constexpr (AX != 2) {
        if (w < nl) {
            double* dst = X + base + jl * s;
#pragma unroll 4
            for (int j = jl; j < n; j += NJ, dst += NJ * s) *dst = at(j)[w];
        }
    } else if constexpr (MODES) {
        for (int r = wid; r < nl; r += NW) {
            double* row = X + (q0 + r) * n;
#pragma unroll 4
            for (int j = lane; j < n; j += 32) row[j] = at(j)[r];
        }
    } else {
        // phi += correction: the block's rows are one run of nl * n values;
        // eight at a time so that their loads overlap
        double* dst = G.phi + q0 * n;
        const int total = nl * n;
        for (int e0 = tid; e0 < total; e0 += 8 * NT) {
            double old[8];
#pragma unroll
            for (int u = 0; u < 8; u++)
                if (e0 + u * NT < total) old[u] = dst[e0 + u * NT];
#pragma unroll
            for (int u = 0; u < 8; u++) {
                const int e = e0 + u * NT;
                if (e < total) {
                    const int r = e / n;
                    dst[e] = old[u] + S[(e - r * n) * DIR_P + r];
                }
            }
        }
    }
}

// This call's arrays and limits of one grid ...
__global__ void k_direct_set(DirGrid* grids, DirCtl* ctl, double* phi, const double* rho,
                             double tol, int maxiter) {
    grids[0].phi = phi;
    grids[0].rho = rho;
    ctl[0] = DirCtl{0.0, 0.0, tol, maxiter, 0, 1, 0};
}
// ... and of a batch: user[2 i] = phi_i, user[2 i + 1] = rho_i
__global__ void k_direct_set_batch(DirGrid* grids, DirCtl* ctl, double* const* user, int n,
                                   double tol, int maxiter) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    grids[i].phi = user[2 * i];
    grids[i].rho = user[2 * i + 1];
    ctl[i] = DirCtl{0.0, 0.0, tol, maxiter, 0, 1, 0};
}

// After a defect, one block a grid: rel = |d| / |rho|; a grid stays active
// while rel > tol and fewer than maxiter corrections ran.  `count` adds the
// correction just finished (0: the initial defect, which also gives |rho|).
__global__ void __launch_bounds__(256)
k_direct_check(const DirGrid* __restrict__ grids, DirCtl* ctl, int count) {
    DirCtl& c = ctl[blockIdx.x];
    if (!c.active) return;
    const DirGrid& G = grids[blockIdx.x];
    double d2 = 0.0, r2 = 0.0;
    for (int i = threadIdx.x; i < G.nblk; i += 256) {
        d2 += G.partial[2 * i];
        if (count == 0) r2 += G.partial[2 * i + 1];
    }
    d2 = block_sum(d2);
    if (count == 0) r2 = block_sum(r2);
    if (threadIdx.x == 0) {
        if (count == 0) c.rho2 = r2;
        const double rel = c.rho2 > 0.0 ? sqrt(d2 / c.rho2) : 0.0;
        c.rel = rel;
        c.niter += count;
        c.active = rel > c.tol && c.niter < c.maxiter;
    }
}

// the loop goes on while any grid is active
__global__ void __launch_bounds__(256)
k_direct_cond(const DirCtl* ctl, int n, cudaGraphConditionalHandle h) {
    int any = 0;
    for (int i = threadIdx.x; i < n; i += 256) any |= ctl[i].active;
    any = __syncthreads_or(any);
    if (threadIdx.x == 0) cudaGraphSetConditional(h, any ? 1u : 0u);
}

int round_up(int x, int m) { return (x + m - 1) / m * m; }

size_t class_smem(int rows, int nw) {
    return ((size_t)rows * DIR_P + (size_t)nw * 2 * STAGE) * sizeof(double);
}

// Block shape of an axis: both halves side by side in 4 or 8 warps while
// their tiles fit (n <= 48, n <= 96), then one after the other in 8 or 16
// (n <= 192, n <= 384).  16 warps an SM either way (128 registers a thread),
// so the smallest block that holds the tiles gives the most blocks to
// overlap one's loads with another's products.
int axis_class(const DirAxis& a) {
    const int te = (a.he + DIR_KT - 1) / DIR_KT, to = (a.ho + DIR_KT - 1) / DIR_KT;
    if (te + to <= 4) return 0;
    if (te + to <= 8) return 1;
    return te <= 8 ? 2 : 3;
}

template <int PASS, int NW, bool TWO>
int launch_class(const DirectGroup& g, int ax, int cls, cudaStream_t st) {
    const DirectGroup::Part& p = g.part[ax][cls];
    if (p.blocks == 0) return 0;
    // (set on every call: cheap, and safe from several threads)
    GB_CUDA_TRY(cudaFuncSetAttribute(k_direct<PASS, NW, TWO>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    k_direct<PASS, NW, TWO><<<p.blocks, 32 * NW, class_smem(p.rows, NW), st>>>(g.grids, g.ctl,
                                                                             p.map);
    GB_LAUNCH_CHECK();
    return 0;
}

template <int PASS>
int launch_pass_of(const DirectGroup& g, cudaStream_t st) {
    constexpr int AX = (PASS == F2 || PASS == B2) ? 2 : PASS == M0 ? 0 : 1;
    if (int rc = launch_class<PASS, 16, true>(g, AX, 3, st)) return rc;
    if (int rc = launch_class<PASS, 8, true>(g, AX, 2, st)) return rc;
    if (int rc = launch_class<PASS, 8, false>(g, AX, 1, st)) return rc;
    return launch_class<PASS, 4, false>(g, AX, 0, st);
}

int group_defect(const DirectGroup& g, int count, cudaGraphConditionalHandle* h,
                 cudaStream_t st) {
    if (int rc = launch_defect_group(g.nn, g.grids, g.ctl, g.defect.map, g.defect.blocks, st))
        return fail(GB_ECUDA, "mixed: defect of the direct solver (%d)", rc);
    GB_LAUNCH_CHECK();
    k_direct_check<<<g.n, 256, 0, st>>>(g.grids, g.ctl, count);
    if (h) k_direct_cond<<<1, 256, 0, st>>>(g.ctl, g.n, *h);
    GB_LAUNCH_CHECK();
    return 0;
}

int group_correction(const DirectGroup& g, cudaStream_t st) {
    if (int rc = launch_pass_of<F2>(g, st)) return rc;
    if (int rc = launch_pass_of<F1>(g, st)) return rc;
    if (int rc = launch_pass_of<M0>(g, st)) return rc;
    if (int rc = launch_pass_of<B1>(g, st)) return rc;
    return launch_pass_of<B2>(g, st);
}

}  // namespace

// ------------------------------------------------------------- one grid
DirectTables::~DirectTables() { dfree(mem); }

int DirectTables::build(const GridBC& g, const double* const pe[3], const double* const po[3],
                        const double* const lam[3]) {
    std::vector<double> host;
    size_t at[3][5];
    for (int a = 0; a < 3; a++) {
        DirAxis& A = ax[a];
        A.n = g.n[a];
        A.per = g.periodic[a];
        A.he = A.per ? A.n / 2 + 1 : (A.n + 1) / 2;
        A.ho = A.n - A.he;
        A.kpe = round_up(A.he, CH);
        A.kpo = round_up(A.ho, CH);
        for (int t = 0; t < 4; t++) {
            const bool odd = t & 1, back = t >= 2;
            const double* P = odd ? po[a] : pe[a];     // [point][mode]
            const int h = odd ? A.ho : A.he, kp = odd ? A.kpo : A.kpe;
            const int tiles = (h + DIR_KT - 1) / DIR_KT;
            at[a][t] = host.size();
            host.resize(host.size() + (size_t)tiles * kp * DIR_KT, 0.0);
            double* T = host.data() + at[a][t];
            for (int k = 0; k < h; k++)
                for (int j = 0; j < h; j++)
                    T[((size_t)(k / DIR_KT) * kp + j) * DIR_KT + k % DIR_KT] =
                        back ? P[(size_t)k * h + j] : P[(size_t)j * h + k];
        }
        at[a][4] = host.size();
        host.insert(host.end(), lam[a], lam[a] + A.n);
        if (host.size() & 1) host.push_back(0.0);      // tables start on 16 bytes
    }
    GB_CUDA_TRY(pool_malloc(&mem, host.size() * sizeof(double)));
    GB_CUDA_TRY(cudaMemcpy(mem, host.data(), host.size() * sizeof(double),
                           cudaMemcpyHostToDevice));
    for (int a = 0; a < 3; a++) {
        ax[a].fe = mem + at[a][0];
        ax[a].fo = mem + at[a][1];
        ax[a].be = mem + at[a][2];
        ax[a].bo = mem + at[a][3];
        ax[a].lam = mem + at[a][4];
    }
    return 0;
}

// ------------------------------------------------------------- the group
DirectGroup::~DirectGroup() {
    if (exec) cudaGraphExecDestroy(exec);
    dfree(mem);
}

int DirectGroup::build(const std::vector<DirGrid>& desc, int half_width, cudaStream_t cs) {
    n = (int)desc.size();
    nn = half_width;
    std::vector<DirGrid> d(desc);
    // CTAs of each pass and of the defect: the grids' blocks in a row, the
    // largest grids first so that the last wave is made of small ones
    std::vector<int> order(n);
    for (int i = 0; i < n; i++) order[i] = i;
    auto pts = [&](int i) { return (long long)d[i].n[0] * d[i].n[1] * d[i].n[2]; };
    std::stable_sort(order.begin(), order.end(),
                     [&](int a, int b) { return pts(a) > pts(b); });
    size_t npart = 0;
    std::vector<size_t> psum(n);
    // CTAs of the defect: one wave (3 an SM) for one grid, three waves over
    // the uneven grids of a batch
    long long total = 0;
    for (int i = 0; i < n; i++) total += pts(i);
    for (int i = 0; i < n; i++) {
        const int share = (int)std::max<long long>(1, 148ll * 3 * (n > 1 ? 3 : 1) * pts(i) / total);
        defect_group_geom(d[i].g, share, d[i].chunk, d[i].tiles_x, d[i].tiles, d[i].nblk);
        psum[i] = npart;
        npart += 2 * (size_t)d[i].nblk;
    }
    std::vector<std::pair<Part*, std::vector<DirBlock>>> maps;
    auto fill = [&](Part& p, auto blocks_of) {
        std::vector<DirBlock> m;
        for (int i : order) {
            const long long nb = blocks_of(i);
            for (long long b = 0; b < nb; b++) m.push_back(DirBlock{i, (int)b});
        }
        p.blocks = (int)m.size();
        if (n > 1 && !m.empty()) maps.emplace_back(&p, std::move(m));
    };
    for (int a = 0; a < 3; a++)
        for (int c = 0; c < 4; c++)
            fill(part[a][c], [&](int i) -> long long {
                const DirAxis& A = d[i].ax[a];
                if (axis_class(A) != c) return 0;
                part[a][c].rows = std::max(part[a][c].rows, dir_rows(A));
                return (pts(i) / A.n + DIR_W - 1) / DIR_W;
            });
    fill(defect, [&](int i) -> long long { return d[i].nblk; });
    // one allocation: grids, control blocks, partial sums, block tables
    auto al = [](size_t x) { return (x + 255) / 256 * 256; };
    const size_t off_ctl = al(n * sizeof(DirGrid)), off_part = off_ctl + al(n * sizeof(DirCtl));
    size_t size = off_part + al(npart * sizeof(double));
    for (auto& m : maps) size += al(m.second.size() * sizeof(DirBlock));
    GB_CUDA_TRY(pool_malloc(&mem, size));
    DirCtl* host = nullptr;
    GB_CUDA_TRY(pool_malloc_host(&host, n * sizeof(DirCtl)));
    results.reset(host, [](DirCtl* p) { hfree(p); });
    grids = (DirGrid*)mem;
    ctl = (DirCtl*)(mem + off_ctl);
    for (int i = 0; i < n; i++) d[i].partial = (double*)(mem + off_part) + psum[i];
    GB_CUDA_TRY(cudaMemcpyAsync(grids, d.data(), n * sizeof(DirGrid), cudaMemcpyHostToDevice, cs));
    GB_CUDA_TRY(cudaMemsetAsync(ctl, 0, n * sizeof(DirCtl), cs));
    size_t at = off_part + al(npart * sizeof(double));
    for (auto& m : maps) {
        m.first->map = (DirBlock*)(mem + at);
        GB_CUDA_TRY(cudaMemcpyAsync(m.first->map, m.second.data(),
                                    m.second.size() * sizeof(DirBlock), cudaMemcpyHostToDevice,
                                    cs));
        at += al(m.second.size() * sizeof(DirBlock));
    }
    // every kernel once, outside a capture (loads them and sets their
    // attributes): no grid is active, so nothing is read or written
    if (int rc = group_defect(*this, 0, nullptr, cs)) return rc;
    if (int rc = group_correction(*this, cs)) return rc;
    GB_CUDA_TRY(cudaStreamSynchronize(cs));
    return capture(cs);
}

// Graph:  defect, check -> WHILE { correction; defect; check }
int DirectGroup::capture(cudaStream_t cs) {
    cudaGraph_t graph;
    GB_CUDA_TRY(cudaGraphCreate(&graph, 0));
    struct Drop {
        cudaGraph_t g;
        ~Drop() { cudaGraphDestroy(g); }
    } drop{graph};
    cudaGraphConditionalHandle h;
    GB_CUDA_TRY(cudaGraphConditionalHandleCreate(&h, graph, 0, 0));
    cudaGraph_t gout = nullptr;
    GB_CUDA_TRY(cudaStreamBeginCaptureToGraph(cs, graph, nullptr, nullptr, 0,
                                              cudaStreamCaptureModeThreadLocal));
    int rc = group_defect(*this, 0, &h, cs);
    cudaStreamCaptureStatus stat;
    const cudaGraphNode_t* deps = nullptr;
    size_t ndeps = 0;
    cudaGraphNode_t tail = nullptr;
    if (!rc && cudaStreamGetCaptureInfo(cs, &stat, nullptr, nullptr, &deps, &ndeps) ==
                   cudaSuccess && ndeps == 1)
        tail = deps[0];
    cudaError_t ce = cudaStreamEndCapture(cs, &gout);
    if (rc) return rc;
    if (ce != cudaSuccess || !tail)
        return fail(GB_ECUDA, "mixed: capture of the defect: %s", cudaGetErrorString(ce));
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t wnode;
    GB_CUDA_TRY(cudaGraphAddNode(&wnode, graph, &tail, 1, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    GB_CUDA_TRY(cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0,
                                              cudaStreamCaptureModeThreadLocal));
    rc = group_correction(*this, cs);
    if (!rc) rc = group_defect(*this, 1, &h, cs);
    ce = cudaStreamEndCapture(cs, &gout);
    if (rc) return rc;
    if (ce != cudaSuccess)
        return fail(GB_ECUDA, "mixed: capture of the correction: %s", cudaGetErrorString(ce));
    GB_CUDA_TRY(cudaGraphInstantiate(&exec, graph, 0));
    return 0;
}

int DirectGroup::run(cudaStream_t st) {
    GB_CUDA_TRY(cudaGraphLaunch(exec, st));
    GB_CUDA_TRY(cudaMemcpyAsync(results.get(), ctl, n * sizeof(DirCtl), cudaMemcpyDeviceToHost,
                                st));
    return 0;
}

int DirectGroup::solve(double* phi, const double* rho, double tol, int maxiter,
                       cudaStream_t st) {
    k_direct_set<<<1, 1, 0, st>>>(grids, ctl, phi, rho, tol, maxiter);
    GB_LAUNCH_CHECK();
    return run(st);
}

int DirectGroup::eager(double* phi, const double* rho, cudaStream_t st) {
    k_direct_set<<<1, 1, 0, st>>>(grids, ctl, phi, rho, 0.0, 1);
    if (int rc = group_defect(*this, 0, nullptr, st)) return rc;
    if (int rc = group_correction(*this, st)) return rc;
    return group_defect(*this, 1, nullptr, st);
}

int DirectGroup::solve_batch(double* const* user, double tol, int maxiter, cudaStream_t st) {
    k_direct_set_batch<<<(n + 127) / 128, 128, 0, st>>>(grids, ctl, user, n, tol, maxiter);
    GB_LAUNCH_CHECK();
    return run(st);
}

}  // namespace gb
