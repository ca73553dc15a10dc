// FP64 stencil pass for general stencils (any offsets up to range 6: the
// Laplacians and gradients of non-orthorhombic cells, Mehrstellen
// operators), real and complex, with the epilogues of gb_internal.cuh.
//
// Same arithmetic as the reference's bmgs_fd over its padded buffer
// (c/bmgs/fd.cpp:9-33): x = 0, then x += v(tap) c(tap) in the caller's order,
// every product and sum rounded on its own.
//
// 24 x 72 x 72 x 100 complex, hexagonal, nn = 3: 613 us one thread a point
// through L1 (every warp straddled a periodic edge), 323 us with fixed 32 x 16
// tiles, 274 us with tiles that divide the plane evenly.
//
// What bounds it: every tap is one shared-memory read (16 bytes a complex
// point: 25 taps of a hexagonal cell's nn = 3 Laplacian take 3.1 clocks of an
// SM a point, against 1.4 for its HBM traffic), so the other work of a tap
// has to be small.  A CTA owns a column tile of up to 512 points (its sides
// divide the plane evenly) and a chunk of planes along axis 0; planes with
// their halo (corners too) stream by cp.async into a ring of 2 R + 2 stages.
// A thread owns two points of the tile, so a
// tap's address (its byte offset from a kernel parameter, wrapped at the
// ring's end by one unsigned minimum) serves both.  Wrap-around is folded
// into the copy's source, and Bloch phases are applied once a cell, right
// after it lands, axis by axis as the reference fills its halo
// (c/bc.cpp:108-112, 242-257).
#include <algorithm>
#include <type_traits>

#include "gb_objects.cuh"
#include "gb_split.cuh"

namespace gb {
namespace {

constexpr int GT = 256;         // threads; two points each
// CTAs an SM, and the cells of a staged plane that this leaves room for
template <class T, int R>
constexpr int gen_blocks() {
    return sizeof(T) == 16 ? (R <= 3 ? 2 : 1) : (R <= 4 ? 3 : 2);
}
template <class T, int R>
constexpr int gen_cells() {
    const int fit = (226 * 1024 / gen_blocks<T, R>() - 1024) / ((2 * R + 2) * (int)sizeof(T));
    return fit < 1536 ? fit : 1536;
}

// a stencil as byte offsets into the ring
struct Taps {
    int n;
    double coef[GB_MAX_COEFS];
    unsigned off[GB_MAX_COEFS];    // stage offset (mod the ring) + in-plane offset
};

template <int BYTES>
__device__ __forceinline__ void tap_copy(unsigned dst, const void* src, bool valid) {
    const int n = valid ? BYTES : 0;      // 0: zero fill, nothing is read
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src),
                     "r"(n));
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src),
                     "r"(n));
}

__device__ __forceinline__ bool into(int& y, int n, int periodic) {
    if (y >= 0 && y < n) return true;
    if (!periodic) return false;
    y += y < 0 ? n : -n;
    return y >= 0 && y < n;
}

// R: the stencil's range, at most this; MODE as in gb_internal.cuh
template <class T, int R, int MODE>
__global__ void __launch_bounds__(GT, gen_blocks<T, R>())
k_general(const T* __restrict__ in, T* __restrict__ out, GridBC g, Phases P,
          const __grid_constant__ Taps s, int chunk, int tiles_x, int tw, int th, Epi ep) {
    constexpr bool CPLX = sizeof(T) == 16;
    constexpr int S = 2 * R + 2, NC = (gen_cells<T, R>() + GT - 1) / GT;
    constexpr unsigned EB = sizeof(T);
    const int PX = tw + 2 * R, E = PX * (th + 2 * R);
    const unsigned PB = E * EB, RING = S * PB;
    extern __shared__ __align__(16) unsigned char gen_smem[];
    const unsigned ring = (unsigned)__cvta_generic_to_shared(gen_smem);

    const int n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
    const long long ps = (long long)n1 * n2, grid0 = (long long)blockIdx.z * n0 * ps;
    const int tid = threadIdx.x;
    const int x0 = (blockIdx.x % tiles_x) * tw, y0 = (blockIdx.x / tiles_x) * th;
    // this thread's points: number tid and tid + 256 of the tile, row by row
    const int ra = min(tid / tw, th - 1), ca_ = tid % tw;
    const int rb = min((tid + GT) / tw, th - 1), cb_ = (tid + GT) % tw;
    const int pa = blockIdx.y * chunk, pb = min(n0, pa + chunk);
    const T* a = in + grid0;

    // this thread's cells: in-plane source (-1: zero) and phase code (bits
    // 0-1 axis 1, bits 2-3 axis 2: 1 past the high edge, 2 past the low one)
    int goff[NC];
    unsigned long long code = 0;
#pragma unroll
    for (int i = 0; i < NC; i++) {
        const int e = tid + GT * i;
        goff[i] = -1;
        if (e < E) {
            int r = y0 - R + e / PX, c = x0 - R + e % PX;
            const unsigned c1 = r >= n1 ? 1u : r < 0 ? 2u : 0u;
            const unsigned c2 = c >= n2 ? 1u : c < 0 ? 2u : 0u;
            if (into(r, n1, g.periodic[1]) && into(c, n2, g.periodic[2])) {
                goff[i] = r * n2 + c;
                if (CPLX && P.use) code |= (unsigned long long)(c1 | (c2 << 2)) << (4 * i);
            }
        }
    }
    auto issue = [&](int p, int slot) {       // plane p (may lie past an edge)
        if (p < pb + R) {
            int pl = p;
            const bool ok = into(pl, n0, g.periodic[0]);
            const T* src = a + (ok ? pl : 0) * ps;
            const unsigned dst = ring + slot * PB + tid * EB;
#pragma unroll
            for (int i = 0; i < NC; i++)
                if (tid + GT * i < E) {
                    const bool v = ok && goff[i] >= 0;
                    tap_copy<(int)EB>(dst + i * GT * EB, v ? src + goff[i] : a, v);
                }
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    auto phases = [&](int p, int slot) {      // of this thread's landed cells
        if constexpr (CPLX) {
            const bool pw = P.use && (p < 0 || p >= n0) && g.periodic[0] && p < pb + R;
            if (!pw && !code) return;
            const double2 ph0 = p >= n0 ? P.ph[0][0] : P.ph[0][1];
            T* st = reinterpret_cast<T*>(gen_smem) + slot * E + tid;
#pragma unroll
            for (int i = 0; i < NC; i++) {
                const unsigned c = (unsigned)(code >> (4 * i)) & 15u;
                if (goff[i] < 0 || !(pw || c)) continue;
                T v = st[GT * i];
                if (pw) v = cmul(ph0, v);
                if (c & 3u) v = cmul((c & 3u) == 1 ? P.ph[1][0] : P.ph[1][1], v);
                if (c >> 2) v = cmul((c >> 2) == 1 ? P.ph[2][0] : P.ph[2][1], v);
                st[GT * i] = v;
            }
        }
    };

    const bool live0 = tid < tw * th && x0 + ca_ < n2 && y0 + ra < n1;
    const bool live1 = tid + GT < tw * th && x0 + cb_ < n2 && y0 + rb < n1;
    const long long at0 = (long long)(y0 + ra) * n2 + x0 + ca_;
    constexpr bool AUX = MODE != EPI_APPLY;
    const T* aux = !AUX || MODE == EPI_POT ? nullptr : (const T*)ep.aux + grid0 + at0;
    const double* pot = MODE == EPI_POT ? (const double*)ep.aux + at0 : nullptr;
    T* o = out ? out + grid0 + at0 : nullptr;
    const long long second = (long long)(rb - ra) * n2 + cb_ - ca_;   // second point
    const int delta = ((rb - ra) * PX + cb_ - ca_) * (int)EB;
    double sq = 0.0;

    // planes pa - R .. pa + R, all landed but the last
    for (int j = 0; j < 2 * R + 1; j++) issue(pa - R + j, j);
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    for (int j = 0; j < 2 * R; j++) phases(pa - R + j, j);
    int slot = R;             // of the centre plane
    for (int p = pa; p < pb; p++) {
        // operands of the epilogue: in flight during the taps
        T ca0 = Num<T>::zero(), ca1 = Num<T>::zero();
        double cp0 = 0.0, cp1 = 0.0;
        if constexpr (AUX) {
            const long long q = p * ps;
            if constexpr (MODE == EPI_POT) {
                if (live0) cp0 = pot[q];
                if (live1) cp1 = pot[q + second];
            } else {
                if (live0) ca0 = aux[q];
                if (live1) ca1 = aux[q + second];
            }
        }
        int front = slot + R;
        if (front >= S) front -= S;
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        phases(p + R, front);
        __syncthreads();
        // the plane after it goes where plane p - R - 1 was
        issue(p + R + 1, front + 1 == S ? 0 : front + 1);
        // byte address of the first point relative to the ring, one ring up
        // for the offsets that point back
        const unsigned cen = slot * PB + ((ra + R) * PX + ca_ + R) * EB;
        T xa = Num<T>::zero(), xb = Num<T>::zero(), va, vb;
        auto read = [&](unsigned at, T& u, T& v) {
            const unsigned char* b = gen_smem + at;
            u = *reinterpret_cast<const T*>(b);
            v = *reinterpret_cast<const T*>(b + delta);
        };
        read(cen, va, vb);
#pragma unroll 6
        for (int c = MODE == EPI_JACOBI ? 1 : 0; c < s.n; c++) {
            T u, v;
            const unsigned t = cen + s.off[c];
            read(min(t, t - RING), u, v);
            xa = Num<T>::add(xa, Num<T>::scale(u, s.coef[c]));
            xb = Num<T>::add(xb, Num<T>::scale(v, s.coef[c]));
        }
        auto finish = [&](T& r, T vc, T ca, double cp) {
            if constexpr (MODE == EPI_POT) {
                r = Num<T>::add(r, Num<T>::scale(vc, cp));
            } else if constexpr (MODE == EPI_RESID) {
                r = Num<T>::sub(r, ca);
            } else if constexpr (MODE == EPI_JACOBI) {
                if constexpr (!CPLX)
                    r = __dadd_rn(__dmul_rn(1.0 - ep.w, vc),
                                  __ddiv_rn(__dmul_rn(ep.w, __dsub_rn(ca, r)), s.coef[0]));
            } else if constexpr (MODE == EPI_PRECOND) {
                r = Num<T>::sub(vc, Num<T>::scale(Num<T>::sub(r, ca), ep.sc));
                if (ep.negate) r = Num<T>::neg(r);
            }
        };
        if constexpr (AUX) {
            finish(xa, va, ca0, cp0);
            finish(xb, vb, ca1, cp1);
            if (MODE == EPI_RESID) {
                if (live0) sq += sqnorm(xa);
                if (live1) sq += sqnorm(xb);
            }
        }
        if (MODE != EPI_RESID || out) {
            if (live0) o[p * ps] = xa;
            if (live1) o[p * ps + second] = xb;
        }
        slot = slot + 1 == S ? 0 : slot + 1;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if (MODE == EPI_RESID && ep.partial) {
        sq = block_sum(sq);
        if (tid == 0)
            ep.partial[((long long)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] =
                sq;
    }
}

struct Geom {
    int tw, th, tiles_x, tiles, chunk, nchunk;
};

// Tile: the even split of the plane into tw x th pieces of at most 512 points
// (two a thread) whose staged plane fits, with the least work: a tap reads
// shared memory for all 512 points, a staged cell is written once.  (A fixed
// 32 x 16 tile computes 1.42 times the points of a 72 x 100 plane.)  Chunk of
// axis 0: least waves x planes (24 x 72 x 72 x 100 hexagonal 274 us; 294 with the
// stencils' share and half a wave for an unfinished one).
Geom geom(const GridBC& g, int R, int ncoefs, int nin, int cells, int blocks) {
    Geom G{};
    long long best = -1;
    for (int kx = 1; kx <= g.n[2]; kx++) {
        const int tw = (g.n[2] + kx - 1) / kx;
        if (tw > 512) continue;
        int th = std::min(512 / tw, cells / (tw + 2 * R) - 2 * R);
        if (th < 1) continue;
        const int ky = (g.n[1] + th - 1) / th;
        th = (g.n[1] + ky - 1) / ky;
        const long long cost = (long long)((g.n[2] + tw - 1) / tw) * ky *
                               (512ll * ncoefs + 2ll * (tw + 2 * R) * (th + 2 * R));
        if (best < 0 || cost < best) {
            best = cost;
            G.tw = tw;
            G.th = th;
        }
        if (tw <= 8) break;
    }
    G.tiles_x = (g.n[2] + G.tw - 1) / G.tw;
    G.tiles = G.tiles_x * ((g.n[1] + G.th - 1) / G.th);
    G.chunk = balance_planes(g.n[0], 1, 2 * R, (long long)G.tiles * nin, blocks, 0.0, 1.0);
    G.nchunk = (g.n[0] + G.chunk - 1) / G.chunk;
    return G;
}

template <class T, int R, int MODE>
int launch_r(const void* in, void* out, int nin, const GridBC& g, const Phases& P,
             const Stencil& st, const Epi& ep, cudaStream_t stream) {
    constexpr int S = 2 * R + 2;
    const Geom G = geom(g, R, st.ncoefs, nin, gen_cells<T, R>(), gen_blocks<T, R>());
    const int PX = G.tw + 2 * R, E = PX * (G.th + 2 * R);
    const int smem = S * E * (int)sizeof(T);
    if (cudaFuncSetAttribute(k_general<T, R, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             smem) != cudaSuccess)
        return -2;
    Taps s;
    s.n = st.ncoefs;
    for (int c = 0; c < st.ncoefs; c++) {
        s.coef[c] = st.coef[c];
        const int stage = st.off[c][0] < 0 ? st.off[c][0] + S : st.off[c][0];
        s.off[c] = (unsigned)((stage * E + st.off[c][1] * PX + st.off[c][2]) * (int)sizeof(T));
    }
    const long long ng = (long long)g.n[0] * g.n[1] * g.n[2];
    for (int b0 = 0; b0 < nin; b0 += 65535) {
        const int nb = std::min(65535, nin - b0);
        Epi e = ep;
        if (e.aux && MODE != EPI_POT) e.aux = (const T*)ep.aux + b0 * ng;
        if (e.partial) e.partial = ep.partial + (long long)b0 * G.tiles * G.nchunk;
        k_general<T, R, MODE><<<dim3(G.tiles, G.nchunk, nb), GT, smem, stream>>>(
            (const T*)in + b0 * ng, out ? (T*)out + b0 * ng : nullptr, g, P, s, G.chunk,
            G.tiles_x, G.tw, G.th, e);
    }
    return 0;
}

template <class T, int MODE>
int launch_m(const void* in, void* out, int nin, const GridBC& g, const Phases& P,
             const Stencil& st, const Epi& ep, cudaStream_t stream) {
    switch (st.range) {
        case 0:
        case 1: return launch_r<T, 1, MODE>(in, out, nin, g, P, st, ep, stream);
        case 2: return launch_r<T, 2, MODE>(in, out, nin, g, P, st, ep, stream);
        case 3: return launch_r<T, 3, MODE>(in, out, nin, g, P, st, ep, stream);
        case 4: return launch_r<T, 4, MODE>(in, out, nin, g, P, st, ep, stream);
        case 5: return launch_r<T, 5, MODE>(in, out, nin, g, P, st, ep, stream);
        case 6: return launch_r<T, 6, MODE>(in, out, nin, g, P, st, ep, stream);
    }
    return -1;
}

}  // namespace

template <class T>
int launch_general(int mode, const void* in, void* out, int nin, const GridBC& g,
                   const Phases& P, const Stencil& st, const Epi& ep, cudaStream_t stream) {
    if ((long long)g.n[1] * g.n[2] >= (1ll << 31)) return -1;
    switch (mode) {
        case EPI_APPLY: return launch_m<T, EPI_APPLY>(in, out, nin, g, P, st, ep, stream);
        case EPI_RESID: return launch_m<T, EPI_RESID>(in, out, nin, g, P, st, ep, stream);
        case EPI_PRECOND: return launch_m<T, EPI_PRECOND>(in, out, nin, g, P, st, ep, stream);
        case EPI_POT: return launch_m<T, EPI_POT>(in, out, nin, g, P, st, ep, stream);
        case EPI_JACOBI:
            if constexpr (sizeof(T) == 8)
                return launch_m<T, EPI_JACOBI>(in, out, nin, g, P, st, ep, stream);
    }
    return -1;
}
template int launch_general<double>(int, const void*, void*, int, const GridBC&, const Phases&,
                                    const Stencil&, const Epi&, cudaStream_t);
template int launch_general<double2>(int, const void*, void*, int, const GridBC&, const Phases&,
                                     const Stencil&, const Epi&, cudaStream_t);

template <class T>
static int blocks_of(const GridBC& g, int range, int ncoefs, int nin) {
    auto of = [&](auto R_) {
        constexpr int R = decltype(R_)::value;
        const Geom G = geom(g, R, ncoefs, nin, gen_cells<T, R>(), gen_blocks<T, R>());
        return G.tiles * G.nchunk;
    };
    switch (range) {
        case 2: return of(std::integral_constant<int, 2>{});
        case 3: return of(std::integral_constant<int, 3>{});
        case 4: return of(std::integral_constant<int, 4>{});
        case 5: return of(std::integral_constant<int, 5>{});
        case 6: return of(std::integral_constant<int, 6>{});
    }
    return of(std::integral_constant<int, 1>{});
}

int general_blocks(const GridBC& g, int range, int ncoefs, int nin, int elem_bytes) {
    return elem_bytes == 16 ? blocks_of<double2>(g, range, ncoefs, nin)
                            : blocks_of<double>(g, range, ncoefs, nin);
}

}  // namespace gb
