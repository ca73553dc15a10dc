// C ABI of gpaw_b200 (declared in include/gpaw_b200.h): object lifetimes,
// argument checks that mirror the reference's, and the host-side sequencing
// of the kernels in gb_fd.cu and gb_transform.cu.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "gb_coarse.cuh"
#include "gb_objects.cuh"
#include "gb_tma.cuh"

using namespace gb;

// ------------------------------------------------------------------- errors
static thread_local std::string g_err;

int gb::fail(int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    g_err = buf;
    return code;
}


extern "C" int gb_version(void) { return 100; }
extern "C" const char* gb_last_error(void) { return g_err.c_str(); }

// ------------------------------------------------------------ tensor maps
namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
    // through the runtime's driver entry point table: no link against libcuda
    static EncodeTiledFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return (EncodeTiledFn) nullptr;
        return (EncodeTiledFn)f;
    }();
    return fn;
}
}  // namespace

int gb::make_plane_map16(CUtensorMap* map, const void* base, long long nb, int n0, int n1,
                         int n2, int box_rows, int box_cols, const char** why) {
    EncodeTiledFn enc = encode_tiled();
    if (!enc) {
        *why = "cuTensorMapEncodeTiled is not available";
        return -1;
    }
    // 8-byte words: a 16-byte element is two of them
    const cuuint64_t dims[4] = {(cuuint64_t)2 * n2, (cuuint64_t)n1, (cuuint64_t)n0,
                                (cuuint64_t)nb};
    const cuuint64_t strides[3] = {(cuuint64_t)n2 * 16, (cuuint64_t)n1 * n2 * 16,
                                   (cuuint64_t)n0 * n1 * n2 * 16};
    const cuuint32_t box[4] = {(cuuint32_t)(2 * box_cols), (cuuint32_t)box_rows, 1, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, const_cast<void*>(base), dims,
                     strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        *why = "cuTensorMapEncodeTiled refused the plane map";
        return -1;
    }
    return 0;
}

extern "C" int gb_device_fault(int* code) {
    if (!code) return fail(GB_EINVAL, "device_fault: NULL argument");
    *code = 0;
    int (*units[])(int*) = {take_fault_transform, take_fault_cfd, take_fault_mixed};
    for (auto take : units) {
        int c = 0;
        if (take(&c)) return fail(GB_ECUDA, "device_fault: cannot read the flag");
        if (c && !*code) *code = c;
    }
    return 0;
}

// ----------------------------------------------------------- kernel trace
// Profiling aid for composite entry points: while a trace is open, each
// kernel of gb_fd_precond is preceded by a CUDA event on the call's stream,
// and one more event follows the last kernel.
namespace {
struct Trace {
    std::mutex mu;
    bool on = false;
    std::vector<cudaEvent_t> ev;
    std::vector<const char*> label;
    int used = 0;
};
Trace g_trace;
}  // namespace

void gb::trace_mark(const char* label, cudaStream_t st) {
    if (!g_trace.on) return;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
        return;
    std::lock_guard<std::mutex> lock(g_trace.mu);
    if (!g_trace.on || g_trace.used >= (int)g_trace.ev.size()) return;
    if (cudaEventRecord(g_trace.ev[g_trace.used], st) != cudaSuccess) return;
    g_trace.label[g_trace.used++] = label;
}

extern "C" int gb_trace_begin(int capacity) {
    if (capacity < 2 || capacity > 1 << 16) return fail(GB_EINVAL, "trace: capacity 2..65536");
    std::lock_guard<std::mutex> lock(g_trace.mu);
    for (cudaEvent_t e : g_trace.ev) cudaEventDestroy(e);
    g_trace.ev.assign(capacity, nullptr);
    g_trace.label.assign(capacity, nullptr);
    for (int i = 0; i < capacity; i++)
        GB_CUDA_TRY(cudaEventCreate(&g_trace.ev[i]));
    g_trace.used = 0;
    g_trace.on = true;
    return 0;
}

extern "C" int gb_trace_end(int max, float* ms, const char** labels, int* count) {
    std::lock_guard<std::mutex> lock(g_trace.mu);
    g_trace.on = false;
    const int n = std::max(0, g_trace.used - 1);
    if (count) *count = n;
    if (g_trace.used > 0) GB_CUDA_TRY(cudaEventSynchronize(g_trace.ev[g_trace.used - 1]));
    for (int i = 0; i < n && i < max; i++) {
        float t = 0.f;
        GB_CUDA_TRY(cudaEventElapsedTime(&t, g_trace.ev[i], g_trace.ev[i + 1]));
        if (ms) ms[i] = t;
        if (labels) labels[i] = g_trace.label[i];
    }
    for (cudaEvent_t e : g_trace.ev) cudaEventDestroy(e);
    g_trace.ev.clear();
    g_trace.label.clear();
    g_trace.used = 0;
    return 0;
}

extern "C" int gb_operator_new(const double* coefs, const int64_t* offsets, int ncoefs,
                               const int64_t size[3], int range, const int64_t neighbors[6],
                               int real, int cfd, gb_operator** out) {
    if (!out || !coefs || !offsets || !size || !neighbors)
        return fail(GB_EINVAL, "Operator: NULL argument");
    *out = nullptr;
    if (ncoefs < 1 || ncoefs > GB_MAX_COEFS)
        return fail(GB_EINVAL, "Operator: %d coefficients (1..%d supported)", ncoefs, GB_MAX_COEFS);
    if (range < 0) return fail(GB_EINVAL, "Operator: negative range");
    for (int c = 0; c < 3; c++)
        if (size[c] < 1 || size[c] > (1 << 20)) return fail(GB_EINVAL, "Operator: bad size");
    if ((double)size[0] * size[1] * size[2] >= 2147483647.0)
        return fail(GB_EINVAL, "Operator: grid has 2^31 points or more");
    gb_operator* op = new gb_operator();
    memset(&op->st, 0, sizeof op->st);
    op->st.ncoefs = ncoefs;
    op->st.range = range;
    op->st.cfd = cfd ? 1 : 0;
    op->real = real ? 1 : 0;
    for (int c = 0; c < 3; c++) {
        op->g.n[c] = (int)size[c];
        const int64_t lo = neighbors[2 * c], hi = neighbors[2 * c + 1];
        if (lo > 0 || hi > 0) {
            delete op;
            return fail(GB_EINVAL, "Operator: neighbour ranks > 0 need domain decomposition");
        }
        // both sides periodic or both zero on a single domain
        op->g.periodic[c] = (lo == 0 && hi == 0) ? 1 : 0;
        if ((lo == 0) != (hi == 0)) {
            delete op;
            return fail(GB_EINVAL, "Operator: mixed periodic/zero on one axis");
        }
        if (op->g.periodic[c] && size[c] < range) {
            delete op;
            return fail(GB_EINVAL, "Stencil longer than domain");
        }
    }
    // Split each flat padded offset into (o0, o1, o2) with |o_c| <= range.
    op->diag = 0.0;
    for (int p = 0; p < ncoefs; p++) {
        const long long f = offsets[p];
        int o[3];
        if (!split_offset(f, size, range, o)) {
            delete op;
            return fail(GB_EINVAL, "Operator: offset %lld does not fit range %d", f, range);
        }
        op->st.coef[p] = coefs[p];
        op->st.off[p][0] = o[0];
        op->st.off[p][1] = o[1];
        op->st.off[p][2] = o[2];
        op->st.flat[p] = ((long long)o[0] * size[1] + o[1]) * size[2] + o[2];
        if (f == 0) op->diag = coefs[p];
    }
    const char* path = getenv("GPAW_B200_FD_PATH");
    const bool force_generic = path && strcmp(path, "generic") == 0;
    // (the plane-marching kernels sum axis 2, then 1, then 0: the order of
    // every Laplacian; axis-aligned stencils in another order are general)
    op->tiled = !force_generic && to_cfd_stencil(op->st, op->cs, op->nn) &&
                op->cs.axis[0] == 2 && op->cs.axis[1] == 1 && op->cs.axis[2] == 0;
    bool axis_aligned = true;
    for (int p = 0; p < ncoefs; p++) {
        const int* o = op->st.off[p];
        axis_aligned = axis_aligned && (o[0] != 0) + (o[1] != 0) + (o[2] != 0) <= 1;
    }
    op->general = !force_generic && range <= 6 && (!cfd || axis_aligned);
    *out = op;
    return 0;
}

extern "C" void gb_operator_free(gb_operator* op) { delete op; }

extern "C" double gb_operator_get_diagonal_element(const gb_operator* op) {
    return op ? op->diag : 0.0;
}

extern "C" int gb_operator_path(const gb_operator* op) {
    return !op ? 0 : op->tiled ? 2 : op->general ? 1 : 0;
}

extern "C" int gb_operator_reserve(gb_operator* op, int64_t nin, int dtype) {
    if (!op) return fail(GB_EINVAL, "NULL operator");
    return op->scratch.ensure((size_t)(nin < 1 ? 1 : nin) * op->ng() * elem_size(dtype));
}

static int check_dtype(const gb_operator* op, int dtype) {
    if (dtype != GB_F64 && dtype != GB_C128) return fail(GB_EINVAL, "unsupported dtype %d", dtype);
    if ((dtype == GB_F64) != (op->real != 0))
        return fail(GB_EINVAL, "dtype does not match the operator (real=%d)", op->real);
    return 0;
}

extern "C" int gb_operator_apply(gb_operator* op, const void* in, void* out, int64_t nin,
                                 int dtype, const double* phases, void* stream) {
    if (!op || !in || !out) return fail(GB_EINVAL, "apply: NULL argument");
    if (int e = check_dtype(op, dtype)) return e;
    if (nin < 0) return fail(GB_EINVAL, "apply: negative batch");
    if (nin == 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    Phases P;
    read_phases(dtype, phases, P);
    const size_t bytes = (size_t)nin * op->ng() * elem_size(dtype);
    if (ranges_overlap(in, out, bytes)) {
        if (int e = op->scratch.ensure(bytes)) return e;
        GB_CUDA_TRY(cudaMemcpyAsync(op->scratch.ptr, in, bytes, cudaMemcpyDeviceToDevice, st));
        in = op->scratch.ptr;
    }
    if (int rc = op_sweep(op, EPI_APPLY, in, out, nullptr, (int)nin, dtype, P, 0, 0, 0, nullptr, st))
        return rc;
    GB_LAUNCH_CHECK();
    return 0;
}

extern "C" int gb_operator_apply_potential(gb_operator* op, const void* in, void* out,
                                           int64_t nin, int dtype, const double* phases,
                                           const double* v, void* stream) {
    if (!op || !in || !out || !v) return fail(GB_EINVAL, "apply_potential: NULL argument");
    if (int e = check_dtype(op, dtype)) return e;
    if (nin < 0) return fail(GB_EINVAL, "apply_potential: negative batch");
    if (nin == 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    Phases P;
    read_phases(dtype, phases, P);
    const size_t bytes = (size_t)nin * op->ng() * elem_size(dtype);
    const char* vb = (const char*)v;
    const char* ob = (const char*)out;
    if (vb < ob + bytes && ob < vb + (size_t)op->ng() * sizeof(double))
        return fail(GB_EINVAL, "apply_potential: v must not overlap out");
    if (ranges_overlap(in, out, bytes)) {
        if (int e = op->scratch.ensure(bytes)) return e;
        GB_CUDA_TRY(cudaMemcpyAsync(op->scratch.ptr, in, bytes, cudaMemcpyDeviceToDevice, st));
        in = op->scratch.ptr;
    }
    if (int rc = op_sweep(op, EPI_POT, in, out, v, (int)nin, dtype, P, 0, 0, 0, nullptr, st))
        return rc;
    GB_LAUNCH_CHECK();
    return 0;
}

extern "C" int gb_operator_set_chunk(gb_operator* op, int chunk) {
    if (!op) return fail(GB_EINVAL, "set_chunk: NULL operator");
    if (chunk < 0) return fail(GB_EINVAL, "set_chunk: chunk must be >= 0");
    op->chunk = chunk;
    return 0;
}

extern "C" int gb_transformer_set_chunk(gb_transformer* t, int chunk) {
    if (!t) return fail(GB_EINVAL, "set_chunk: NULL transformer");
    if (chunk < 0) return fail(GB_EINVAL, "set_chunk: chunk must be >= 0");
    t->G.chunk = chunk;
    return 0;
}

extern "C" int gb_operator_residual(gb_operator* op, const void* phi, const void* rho, void* r,
                                    int64_t nin, int dtype, const double* phases, double scale,
                                    double* norm2, void* stream) {
    if (!op || !phi || !rho) return fail(GB_EINVAL, "residual: NULL argument");
    if (int e = check_dtype(op, dtype)) return e;
    if (nin <= 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    Phases P;
    read_phases(dtype, phases, P);
    const size_t bytes = (size_t)nin * op->ng() * elem_size(dtype);
    if (r && (ranges_overlap(phi, r, bytes)))
        return fail(GB_EINVAL, "residual: r must not overlap phi");
    double* partial = nullptr;
    const int nblk = op_resid_blocks(op, (int)nin, (int)elem_size(dtype));
    if (norm2) {
        if (int e = op->partial.ensure((size_t)nin * nblk * sizeof(double))) return e;
        partial = (double*)op->partial.ptr;
    }
    if (int rc = op_sweep(op, EPI_RESID, phi, r, rho, (int)nin, dtype, P, 0, 0, 0, partial, st))
        return rc;
    GB_LAUNCH_CHECK();
    if (norm2) {
        launch_reduce_partials(partial, nblk, (int)nin, scale, norm2, st);
        GB_LAUNCH_CHECK();
    }
    return 0;
}

// The relaxation itself, with its scratch grid X (op->ng() doubles) given by
// the caller: the operator's own buffer (gb_operator_relax) or the fixed
// device array of gb_operator_relax_noalloc.
static int relax_with_scratch(gb_operator* op, int method, double* f, const double* s,
                              int nrelax, double w, double* X, cudaStream_t st) {
    const size_t bytes = (size_t)op->ng() * sizeof(double);
    if (method == 1) {
        // Gauss-Seidel by wavefronts; wrapped reads see the sweep's start.
        const int r = op->st.range;
        int wa = 1, wb = 1;
        if (!op->st.cfd) {
            wb = 2 * r + 1;
            wa = (wb + 1) * r + 1;
        }
        const GridBC& g = op->g;
        const int nt = wa * (g.n[0] - 1) + wb * (g.n[1] - 1) + g.n[2];
        const bool periodic = g.periodic[0] || g.periodic[1] || g.periodic[2];
        const double inv0 = 1.0 / op->st.coef[0];
        for (int it = 0; it < nrelax; it++) {
            if (periodic) GB_CUDA_TRY(cudaMemcpyAsync(X, f, bytes, cudaMemcpyDeviceToDevice, st));
            for (int t = 0; t < nt; t++)
                launch_gs_wave(f, periodic ? X : f, s, g, op->st, t, wa, wb, inv0, st);
            GB_LAUNCH_CHECK();
        }
        return 0;
    }
    // weighted Jacobi: ping-pong so that the last sweep lands in f
    const double* src = f;
    if (nrelax % 2 == 1) {
        GB_CUDA_TRY(cudaMemcpyAsync(X, f, bytes, cudaMemcpyDeviceToDevice, st));
        src = X;
    }
    Phases P0;
    memset(&P0, 0, sizeof P0);
    for (int it = 0; it < nrelax; it++) {
        double* dst = (src == f) ? X : f;
        if (int rc = op_sweep(op, EPI_JACOBI, src, dst, s, 1, GB_F64, P0, w, 0, 0, nullptr, st))
            return rc;
        src = dst;
    }
    GB_LAUNCH_CHECK();
    return 0;
}

static int relax_impl(gb_operator* op, int method, double* f, const double* s, int nrelax,
                      double w, cudaStream_t st) {
    if (nrelax <= 0) return 0;
    if (int e = op->scratch.ensure((size_t)op->ng() * sizeof(double))) return e;
    return relax_with_scratch(op, method, f, s, nrelax, w, (double*)op->scratch.ptr, st);
}

extern "C" int gb_operator_relax(gb_operator* op, int method, double* f, const double* s,
                                 int nrelax, double w, void* stream) {
    if (!op || !f || !s) return fail(GB_EINVAL, "relax: NULL argument");
    if (!op->real) return fail(GB_EINVAL, "relax: float64 operators only");
    if (method != 1 && method != 2) return fail(GB_EINVAL, "relax: method must be 1 or 2");
    return relax_impl(op, method, f, s, nrelax, w, (cudaStream_t)stream);
}

// -------------------------------------------------------------- Transformer

static void lagrange_weights(int k, double* w) {
    // Weights of the order-k Lagrange interpolant at the mid-point, for the
    // node pairs at distance 1/2, 3/2, ... (exact binary fractions, equal to
    // the constants of c/bmgs/restrict.cpp:37-57).
    for (int j = k / 2; j < k; j++) {
        double num = 1.0, den = 1.0;
        const double xj = (2.0 * j - k + 1) / 2.0;
        for (int m = 0; m < k; m++) {
            if (m == j) continue;
            const double xm = (2.0 * m - k + 1) / 2.0;
            num *= (0.0 - xm);
            den *= (xj - xm);
        }
        w[j - k / 2] = num / den;
    }
}

extern "C" int gb_transformer_new(const int64_t size_in[3], const int64_t size_out[3], int k,
                                  const int64_t pads[6], const int64_t npads[6],
                                  const int64_t skip[6], const int64_t neighbors[6], int real,
                                  int interpolate, gb_transformer** out) {
    if (!out || !size_in || !size_out || !pads || !npads || !skip || !neighbors)
        return fail(GB_EINVAL, "Transformer: NULL argument");
    *out = nullptr;
    if (k != 2 && k != 4 && k != 6 && k != 8)
        return fail(GB_EINVAL, "Transformer: k must be 2, 4, 6 or 8");
    gb_transformer* t = new gb_transformer();
    memset(&t->G, 0, sizeof t->G);
    t->k = k;
    t->interpolate = interpolate ? 1 : 0;
    t->real = real ? 1 : 0;
    XferGeom& G = t->G;
    const int e = interpolate ? k - 1 : 2 * k - 3;
    for (int c = 0; c < 3; c++) {
        const int64_t lo = neighbors[2 * c], hi = neighbors[2 * c + 1];
        if (lo > 0 || hi > 0 || (lo == 0) != (hi == 0)) {
            delete t;
            return fail(GB_EINVAL, "Transformer: single-domain neighbours only");
        }
        G.g.n[c] = (int)size_in[c];
        G.g.periodic[c] = (lo == 0) ? 1 : 0;
        if (pads[2 * c] < 0 || pads[2 * c + 1] < 0) {
            delete t;
            return fail(GB_EINVAL, "Transformer: negative padding");
        }
        if (G.g.periodic[c] && (npads[2 * c] != pads[2 * c + 1] || npads[2 * c + 1] != pads[2 * c] ||
                                pads[2 * c] > size_in[c] || pads[2 * c + 1] > size_in[c])) {
            delete t;
            return fail(GB_EINVAL, "Transformer: periodic padding wider than the grid");
        }
        G.plo[c] = (int)pads[2 * c];
        G.s[c] = (int)(size_in[c] + pads[2 * c] + pads[2 * c + 1]);
        G.nout[c] = (int)size_out[c];
        G.skip0[c] = interpolate ? (int)skip[2 * c] : 0;
        G.skip1[c] = interpolate ? (int)skip[2 * c + 1] : 0;
        const int expect = interpolate ? 2 * (G.s[c] - e + G.skip1[c]) - G.skip0[c] - G.skip1[c]
                                       : (G.s[c] - e) / 2;
        if (expect != size_out[c]) {
            delete t;
            return fail(GB_EINVAL, "Transformer: output size %lld does not match input geometry (%d)",
                        (long long)size_out[c], expect);
        }
    }
    lagrange_weights(k, G.w);
    t->ngin = (long long)size_in[0] * size_in[1] * size_in[2];
    t->ngout = (long long)size_out[0] * size_out[1] * size_out[2];
    *out = t;
    return 0;
}

extern "C" void gb_transformer_free(gb_transformer* t) { delete t; }

extern "C" int gb_transformer_apply(gb_transformer* t, const void* in, void* out, int64_t nin,
                                    int dtype, const double* phases, void* stream) {
    if (!t || !in || !out) return fail(GB_EINVAL, "transformer apply: NULL argument");
    if (dtype != GB_F64 && dtype != GB_C128) return fail(GB_EINVAL, "unsupported dtype");
    if ((dtype == GB_F64) != (t->real != 0))
        return fail(GB_EINVAL, "dtype does not match the transformer (real=%d)", t->real);
    if (nin <= 0) return 0;
    const size_t es = elem_size(dtype);
    const char* ib = (const char*)in;
    const char* ob = (const char*)out;
    if (ib < ob + nin * t->ngout * es && ob < ib + nin * t->ngin * es)
        return fail(GB_EINVAL, "transformer apply: input and output overlap");
    Phases P;
    read_phases(dtype, phases, P);
    return transform_impl(t, in, out, nullptr, nin, dtype, P, 0, 0, 0.0, (cudaStream_t)stream);
}

namespace gb {
int density_work_doubles(int nin);
int launch_density(int k, const double* in, double* out, int nin, const XferGeom& G,
                   const double* const w[3], double dv, double dvf, double* work,
                   cudaStream_t st);
}  // namespace gb

extern "C" int64_t gb_density_work(int64_t nin) {
    return nin > 0 && nin <= 65535 ? density_work_doubles((int)nin) : 0;
}

extern "C" int gb_density_interpolate(gb_transformer* t, const double* in, double* out,
                                      int64_t nin, const double* const* weights, double dv,
                                      double dv_fine, double* work, void* stream) {
    if (!t || !in || !out || !weights || !weights[0] || !weights[1] || !weights[2] || !work)
        return fail(GB_EINVAL, "density interpolate: NULL argument");
    if (!t->interpolate || !t->real)
        return fail(GB_EINVAL, "density interpolate: a real interpolator is needed");
    if (nin <= 0) return 0;
    if (nin > 65535) return fail(GB_EINVAL, "density interpolate: at most 65535 grids");
    const char* ib = (const char*)in;
    const char* ob = (const char*)out;
    if (ib < ob + nin * t->ngout * 8 && ob < ib + nin * t->ngin * 8)
        return fail(GB_EINVAL, "density interpolate: input and output overlap");
    const int rc = launch_density(t->k, in, out, (int)nin, t->G, weights, dv, dv_fine, work,
                                  (cudaStream_t)stream);
    if (rc == -2) return fail(GB_ECUDA, "transformer: could not raise the shared-memory limit");
    if (rc) return fail(GB_EINVAL, "transformer: unsupported order");
    GB_LAUNCH_CHECK();
    return 0;
}

// --------------------------------------------------------------- fd_precond
extern "C" int gb_fd_precond(gb_transformer* rest0, gb_transformer* rest1, gb_transformer* intp1,
                             gb_transformer* intp2, gb_operator* kin0, gb_operator* kin1,
                             gb_operator* kin2, void* d0, void* q0, void* r1, void* d1, void* q1,
                             void* r2, void* d2, void* q2, const void* residuals,
                             const void* nresiduals, int64_t nin, int dtype, double step,
                             const double* phases, void* stream) {
    if (!rest0 || !rest1 || !intp1 || !intp2 || !kin0 || !kin1 || !kin2)
        return fail(GB_EINVAL, "fd_precond: NULL object");
    if (!d0 || !q0 || !r1 || !d1 || !q1 || !r2 || !d2 || !q2 || !residuals)
        return fail(GB_EINVAL, "fd_precond: NULL array");
    if (int e = check_dtype(kin0, dtype)) return e;
    if (int e = check_dtype(kin1, dtype)) return e;
    if (int e = check_dtype(kin2, dtype)) return e;
    if (rest0->ngin != kin0->ng() || rest0->ngout != kin1->ng() || rest1->ngin != kin1->ng() ||
        rest1->ngout != kin2->ng() || intp2->ngin != kin2->ng() || intp2->ngout != kin1->ng() ||
        intp1->ngin != kin1->ng() || intp1->ngout != kin0->ng() || rest0->interpolate ||
        rest1->interpolate || !intp1->interpolate || !intp2->interpolate)
        return fail(GB_EINVAL, "fd_precond: level sizes do not match");
    if (nin <= 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    Phases P;
    read_phases(dtype, phases, P);
    const int n = (int)nin;
    const double s4 = 4 * step, s16 = 16 * step;
    // real grids of at least 2^18 points: the pass kernel (two points a
    // thread from 16-byte shared-memory reads, the same arithmetic) unless
    // GPAW_B200_PASS=0.  128 x 112^3 (C4): 1.64 -> 1.16 ms for the level-0
    // step; on the 56^3 level it was slower (0.13 -> 0.16 ms).
    static const bool pass = [] {
        const char* e = getenv("GPAW_B200_PASS");
        return !(e && atoi(e) == 0);
    }();
    auto step_launch = [&](gb_operator* op, const void* d, const void* r, void* o, double sc,
                           int negate) {
        if (pass && dtype == GB_F64 && op->tiled && d != o && r != o &&
            op->ng() >= (1ll << 18)) {
            const int rc = launch_pass_precond(op->g, op->cs, op->nn, (const double*)d,
                                               (double*)o, (const double*)r, n, sc, negate, st);
            if (rc == 0) {
                GB_LAUNCH_CHECK();
                return 0;
            }
            if (rc == -2) return fail(GB_ECUDA, "precond: could not raise the shared-memory limit");
        }
        return op_sweep(op, EPI_PRECOND, d, o, r, n, dtype, P, 0, sc, negate, nullptr, st);
    };
    int rc;
    // r1 = restrict(-R); d1 = 4 s r1
    trace_mark("restrict0 r1,d1 = R(-R), 4s r1", st);
    if (nresiduals)
        rc = transform_impl(rest0, nresiduals, r1, d1, nin, dtype, P, 0, 0, s4, st);
    else
        rc = transform_impl(rest0, residuals, r1, d1, nin, dtype, P, 1, 0, s4, st);
    if (rc) return rc;
    // q1 = K1 d1 - r1; r2 = restrict(q1); d2 = 16 s r2
    trace_mark("kin1 q1 = K1 d1 - r1", st);
    if ((rc = op_sweep(kin1, EPI_RESID, d1, q1, r1, n, dtype, P, 0, 0, 0, nullptr, st))) return rc;
    GB_LAUNCH_CHECK();
    trace_mark("restrict1 r2,d2 = R(q1), 16s r2", st);
    if ((rc = transform_impl(rest1, q1, r2, d2, nin, dtype, P, 0, 0, s16, st))) return rc;
    // d2' = d2 - 16 s (K2 d2 - r2)   (into q2)
    trace_mark("kin2 q2 = d2 - 16s(K2 d2 - r2)", st);
    if ((rc = step_launch(kin2, d2, r2, q2, s16, 0))) return rc;
    GB_LAUNCH_CHECK();
    // d1 -= interpolate(d2')
    trace_mark("interp2 d1 -= I(q2)", st);
    if ((rc = transform_impl(intp2, q2, d1, nullptr, nin, dtype, P, 0, 1, 0.0, st))) return rc;
    // d1' = d1 - 4 s (K1 d1 - r1)   (into q1)
    trace_mark("kin1 q1 = d1 - 4s(K1 d1 - r1)", st);
    if ((rc = step_launch(kin1, d1, r1, q1, s4, 0))) return rc;
    GB_LAUNCH_CHECK();
    // q0 = interpolate(-d1')
    trace_mark("interp1 q0 = I(-q1)", st);
    if ((rc = transform_impl(intp1, q1, q0, nullptr, nin, dtype, P, 1, 0, 0.0, st))) return rc;
    // d0 = -(q0 - s (K0 q0 - R))
    trace_mark("kin0 d0 = -(q0 - s(K0 q0 - R))", st);
    if ((rc = step_launch(kin0, q0, residuals, d0, step, 1))) return rc;
    GB_LAUNCH_CHECK();
    trace_mark("end", st);
    return 0;
}

// --------------------------------------------------------------- FD Poisson
struct SolveCtl {
    double eps;
    double err;
    int maxiter;
    int niter;
};

// After each V-cycle: niter += 1; keep looping while err > eps and
// niter < maxiter (gpaw/poisson.py:484-486).
__global__ void k_solve_check(SolveCtl* ctl, const double* err, cudaGraphConditionalHandle h) {
    const int n = ctl->niter + 1;
    ctl->niter = n;
    ctl->err = err[0];
    cudaGraphSetConditional(h, (err[0] > ctl->eps && n < ctl->maxiter) ? 1u : 0u);
}

__global__ void k_solve_init(SolveCtl* ctl, double eps, int maxiter) {
    ctl->eps = eps;
    ctl->maxiter = maxiter;
    ctl->niter = 0;
    ctl->err = 0.0;
}

struct gb_poisson {
    int L;  // coarsest level index
    int tail_lf = -1;           // first level of the fused coarse V-cycle (-1: none)
    gb::CoarsePlan tail;
    std::vector<gb_operator*> ops;
    std::vector<gb_transformer*> rst, itp;
    std::vector<int> pre, post;
    std::vector<double> w;
    int method;
    double dv;
    std::vector<double*> phi, rho, res;  // per level (phi[0], rho[0] from the caller)
    double* partial = nullptr;
    double* err_dev = nullptr;
    double* err_host = nullptr;
    double* mean_dev = nullptr;
    // device-resident solve: own copies of phi0/rho0, a control block and a
    // graph holding   while (err > eps && niter < maxiter) { V-cycle }
    double* phi0 = nullptr;
    double* rho0 = nullptr;
    SolveCtl* ctl = nullptr;
    SolveCtl* ctl_host = nullptr;
    cudaStream_t cap = nullptr;
    cudaGraphExec_t solve_exec = nullptr;
    int last_maxiter = 0;
    ~gb_poisson() {
        if (solve_exec) cudaGraphExecDestroy(solve_exec);
        if (cap) cudaStreamDestroy(cap);
        dfree(phi0);
        dfree(rho0);
        dfree(ctl);
        if (ctl_host) hfree(ctl_host);
        for (size_t l = 1; l < phi.size(); l++) dfree(phi[l]);
        for (size_t l = 1; l < rho.size(); l++) dfree(rho[l]);
        for (double* p : res) dfree(p);
        dfree(partial);
        dfree(err_dev);
        dfree(mean_dev);
        if (err_host) hfree(err_host);
    }
};

// Pick the first level of the fused coarse V-cycle (gb_coarse.cu): the
// coarsest run of levels (below level 0) whose operators are 2nd-order
// axis-aligned Laplacians, whose transfers are K = 2, that relax by weighted
// Jacobi and whose first level holds at most coarse_points() points (four a
// thread; the 63^3 level of a 127^3 grid is faster over all SMs).
// GPAW_B200_POISSON_TAIL=0 keeps every level on the per-level kernels (same
// results).
static void plan_tail(gb_poisson* p) {
    p->tail_lf = -1;
    memset(&p->tail, 0, sizeof p->tail);
    const char* env = getenv("GPAW_B200_POISSON_TAIL");
    if ((env && atoi(env) == 0) || p->method != 2 || p->L < 1) return;
    std::vector<gb::CoarseLevel> lv(p->L + 1);
    int lf = -1;
    for (int l = p->L; l >= 1; l--) {
        const gb_operator* op = p->ops[l];
        if (!op->tiled || op->nn != 1 || !op->real || op->ng() > gb::coarse_points(false) ||
            !(op->cs.axis[0] == 2 && op->cs.axis[1] == 1 && op->cs.axis[2] == 0) ||
            p->L - l + 1 > gb::COARSE_LEVELS)
            break;
        gb::CoarseLevel& V = lv[l];
        memset(&V, 0, sizeof V);
        V.ng = (int)op->ng();
        for (int c = 0; c < 3; c++) {
            V.n[c] = op->g.n[c];
            V.per[c] = op->g.periodic[c];
            V.cp[c] = op->cs.cp[c][0];
            V.cm[c] = op->cs.cm[c][0];
        }
        V.c0 = op->cs.c0;
        V.rc0 = 1.0 / op->cs.c0;
        V.pre = p->pre[l];
        V.post = p->post[l];
        V.wj = p->w[l];
        if (l < p->L &&
            !gb::coarse_transfers(V, p->rst[l]->k, p->rst[l]->G, p->itp[l]->k, p->itp[l]->G,
                                  p->ops[l + 1]->g.n))
            break;
        lf = l;
    }
    if (lf < 0) return;
    p->tail.nl = p->L - lf + 1;
    for (int l = lf; l <= p->L; l++) p->tail.lv[l - lf] = lv[l];
    p->tail_lf = lf;
}

extern "C" int gb_poisson_new(int nlevels, gb_operator* const* operators,
                              gb_transformer* const* restrictors,
                              gb_transformer* const* interpolators, const int* presmooths,
                              const int* postsmooths, const double* weights, int relax_method,
                              double dv, gb_poisson** out) {
    if (!out || !operators || nlevels < 1 || !presmooths || !postsmooths || !weights)
        return fail(GB_EINVAL, "Poisson: bad arguments");
    if (nlevels > 1 && (!restrictors || !interpolators))
        return fail(GB_EINVAL, "Poisson: missing transformers");
    if (relax_method != 1 && relax_method != 2)
        return fail(GB_EINVAL, "Poisson: relax method must be 1 (GS) or 2 (J)");
    *out = nullptr;
    gb_poisson* p = new gb_poisson();
    p->L = nlevels - 1;
    p->method = relax_method;
    p->dv = dv;
    for (int l = 0; l < nlevels; l++) {
        if (!operators[l] || !operators[l]->real) {
            delete p;
            return fail(GB_EINVAL, "Poisson: level %d operator missing or complex", l);
        }
        p->ops.push_back(operators[l]);
        p->pre.push_back(presmooths[l]);
        p->post.push_back(postsmooths[l]);
        p->w.push_back(weights[l]);
    }
    for (int l = 0; l < p->L; l++) {
        gb_transformer* r = restrictors[l];
        gb_transformer* i = interpolators[l];
        if (!r || !i || r->interpolate || !i->interpolate || !r->real || !i->real ||
            r->ngin != p->ops[l]->ng() || r->ngout != p->ops[l + 1]->ng() ||
            i->ngin != p->ops[l + 1]->ng() || i->ngout != p->ops[l]->ng()) {
            delete p;
            return fail(GB_EINVAL, "Poisson: transformer %d does not match the levels", l);
        }
        p->rst.push_back(r);
        p->itp.push_back(i);
    }
    plan_tail(p);
    p->phi.assign(nlevels, nullptr);
    p->rho.assign(nlevels, nullptr);
    p->res.assign(nlevels, nullptr);
    for (int l = 0; l < nlevels; l++) {
        const size_t bytes = (size_t)p->ops[l]->ng() * sizeof(double);
        cudaError_t e = pool_malloc(&p->res[l], bytes);
        if (e == cudaSuccess && l > 0) e = pool_malloc(&p->phi[l], bytes);
        if (e == cudaSuccess && l > 0) e = pool_malloc(&p->rho[l], bytes);
        if (e != cudaSuccess) {
            delete p;
            return fail(GB_ECUDA, "Poisson: cudaMalloc: %s", cudaGetErrorString(e));
        }
        if (int rc = gb_operator_reserve(p->ops[l], 1, GB_F64)) {
            delete p;
            return rc;
        }
    }
    const int nblk = std::max(residual_blocks(p->ops[0]->g), op_resid_blocks(p->ops[0], 1, 8));
    cudaError_t e = pool_malloc(&p->partial, (size_t)nblk * sizeof(double));
    if (e == cudaSuccess) e = pool_malloc(&p->err_dev, sizeof(double));
    if (e == cudaSuccess) e = pool_malloc(&p->mean_dev, sizeof(double));
    if (e == cudaSuccess) e = pool_malloc_host(&p->err_host, sizeof(double));
    const size_t bytes0 = (size_t)p->ops[0]->ng() * sizeof(double);
    if (e == cudaSuccess) e = pool_malloc(&p->phi0, bytes0);
    if (e == cudaSuccess) e = pool_malloc(&p->rho0, bytes0);
    if (e == cudaSuccess) e = pool_malloc(&p->ctl, sizeof(SolveCtl));
    if (e == cudaSuccess) e = pool_malloc_host(&p->ctl_host, sizeof(SolveCtl));
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&p->cap, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        delete p;
        return fail(GB_ECUDA, "Poisson: allocation: %s", cudaGetErrorString(e));
    }
    for (int k = 0; k < p->tail.nl; k++) {
        gb::CoarseLevel& V = p->tail.lv[k];
        V.phi = p->phi[p->tail_lf + k];
        V.rho = p->rho[p->tail_lf + k];
        V.tmp = p->res[p->tail_lf + k];
    }
    *out = p;
    return 0;
}

extern "C" void gb_poisson_free(gb_poisson* p) { delete p; }

extern "C" int gb_poisson_fused_levels(const gb_poisson* p) {
    return (p && p->tail_lf >= 0) ? p->tail.nl : 0;
}

// iterate2 (gpaw/poisson.py:500-537), recursive over levels.
static int vcycle(gb_poisson* p, int l, cudaStream_t st) {
    if (l == p->tail_lf) return launch_coarse(p->tail, false, st);   // starts from phi_l = 0
    gb_operator* op = p->ops[l];
    Phases P;
    memset(&P, 0, sizeof P);
    if (l < p->L) {
        if (int rc = relax_impl(op, p->method, p->phi[l], p->rho[l], p->pre[l], p->w[l], st))
            return rc;
        if (int rc = op_sweep(op, EPI_RESID, p->phi[l], p->res[l], p->rho[l], 1, GB_F64, P, 0, 0, 0,
                              nullptr, st))
            return rc;
        GB_LAUNCH_CHECK();
        if (int rc = transform_impl(p->rst[l], p->res[l], p->rho[l + 1], nullptr, 1, GB_F64, P, 0,
                                    0, 0.0, st))
            return rc;
        if (l + 1 != p->tail_lf)
            GB_CUDA_TRY(cudaMemsetAsync(p->phi[l + 1], 0,
                                        (size_t)p->ops[l + 1]->ng() * sizeof(double), st));
        if (int rc = vcycle(p, l + 1, st)) return rc;
        // phi_l -= interpolate(phi_{l+1})
        if (int rc = transform_impl(p->itp[l], p->phi[l + 1], p->phi[l], nullptr, 1, GB_F64, P, 0,
                                    1, 0.0, st))
            return rc;
    }
    if (int rc = relax_impl(op, p->method, p->phi[l], p->rho[l], p->post[l], p->w[l], st))
        return rc;
    if (l == 0) {
        const int nblk = op_resid_blocks(op, 1, 8);
        if (int rc = op_sweep(op, EPI_RESID, p->phi[0], p->res[0], p->rho[0], 1, GB_F64, P, 0, 0, 0,
                              p->partial, st))
            return rc;
        GB_LAUNCH_CHECK();
        launch_reduce_partials(p->partial, nblk, 1, p->dv, p->err_dev, st);
        GB_LAUNCH_CHECK();
    }
    return 0;
}

extern "C" int gb_poisson_iterate(gb_poisson* p, double* phi, const double* rho, double* error,
                                  void* stream) {
    if (!p || !phi || !rho) return fail(GB_EINVAL, "Poisson iterate: NULL argument");
    cudaStream_t st = (cudaStream_t)stream;
    p->phi[0] = phi;
    p->rho[0] = (double*)rho;  // never written
    if (int rc = vcycle(p, 0, st)) return rc;
    GB_CUDA_TRY(cudaMemcpyAsync(p->err_host, p->err_dev, sizeof(double), cudaMemcpyDeviceToHost, st));
    GB_CUDA_TRY(cudaStreamSynchronize(st));
    if (error) *error = *p->err_host;
    return 0;
}

__global__ void k_sub_scalar(double* a, long long n, const double* v, double count) {
    // phi_ave = sum(phi) / prod(N_c); phi -= phi_ave  (gpaw/poisson.py:492-496)
    const double m = v[0] / count;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        a[i] = a[i] - m;
}

__global__ void k_block_sums(const double* a, long long n, double* partial) {
    double v = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x)
        v += a[i];
    v = block_sum(v);
    if (threadIdx.x == 0) partial[blockIdx.x] = v;
}

static int mean_removal(gb_poisson* p, double* phi, cudaStream_t st) {
    const GridBC& g = p->ops[0]->g;
    if (!(g.periodic[0] && g.periodic[1] && g.periodic[2])) return 0;
    const long long n = p->ops[0]->ng();
    const int nb = (int)std::min<long long>(1024, (n + 255) / 256);
    k_block_sums<<<nb, 256, 0, st>>>(phi, n, p->partial);
    launch_reduce_partials(p->partial, nb, 1, 1.0, p->mean_dev, st);
    k_sub_scalar<<<nb, 256, 0, st>>>(phi, n, p->mean_dev, (double)n);
    GB_LAUNCH_CHECK();
    return 0;
}

// Capture the whole solve_neutral loop once per executor into a graph with
// a conditional WHILE node: the V-cycle and a check kernel that sets the
// loop condition, then the periodic mean removal.  It works on the
// executor's own phi0/rho0, so one graph serves every call.
static int build_solve_graph(gb_poisson* p) {
    cudaStream_t cs = p->cap;
    // one uncaptured V-cycle first: sets kernel attributes, touches scratch
    GB_CUDA_TRY(cudaMemsetAsync(p->phi0, 0, (size_t)p->ops[0]->ng() * 8, cs));
    GB_CUDA_TRY(cudaMemsetAsync(p->rho0, 0, (size_t)p->ops[0]->ng() * 8, cs));
    p->phi[0] = p->phi0;
    p->rho[0] = p->rho0;
    if (int rc = vcycle(p, 0, cs)) return rc;
    if (int rc = mean_removal(p, p->phi0, cs)) return rc;
    GB_CUDA_TRY(cudaStreamSynchronize(cs));

    cudaGraph_t graph;
    GB_CUDA_TRY(cudaGraphCreate(&graph, 0));
    cudaGraphConditionalHandle h;
    GB_CUDA_TRY(cudaGraphConditionalHandleCreate(&h, graph, 1, cudaGraphCondAssignDefault));
    cudaGraphNodeParams cp = {};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t wnode;
    GB_CUDA_TRY(cudaGraphAddNode(&wnode, graph, nullptr, 0, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    GB_CUDA_TRY(cudaStreamBeginCaptureToGraph(cs, body, nullptr, nullptr, 0,
                                              cudaStreamCaptureModeThreadLocal));
    int rc = vcycle(p, 0, cs);
    if (!rc) k_solve_check<<<1, 1, 0, cs>>>(p->ctl, p->err_dev, h);
    cudaGraph_t body_out = nullptr;
    cudaError_t ce = cudaStreamEndCapture(cs, &body_out);
    if (rc) {
        cudaGraphDestroy(graph);
        return rc;
    }
    if (ce != cudaSuccess) {
        cudaGraphDestroy(graph);
        return fail(GB_ECUDA, "Poisson: capture of the V-cycle: %s", cudaGetErrorString(ce));
    }
    // mean removal after the loop (periodic grids)
    GB_CUDA_TRY(cudaStreamBeginCaptureToGraph(cs, graph, &wnode, nullptr, 1,
                                              cudaStreamCaptureModeThreadLocal));
    rc = mean_removal(p, p->phi0, cs);
    cudaGraph_t g2 = nullptr;
    ce = cudaStreamEndCapture(cs, &g2);
    if (rc || ce != cudaSuccess) {
        cudaGraphDestroy(graph);
        return rc ? rc : fail(GB_ECUDA, "Poisson: capture: %s", cudaGetErrorString(ce));
    }
    cudaError_t ie = cudaGraphInstantiate(&p->solve_exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ie != cudaSuccess) return fail(GB_ECUDA, "Poisson: instantiate: %s", cudaGetErrorString(ie));
    return 0;
}

extern "C" int gb_poisson_solve_neutral_async(gb_poisson* p, double* phi, const double* rho,
                                              double eps, int maxiter, void* stream) {
    if (!p || !phi || !rho) return fail(GB_EINVAL, "Poisson solve: NULL argument");
    if (maxiter < 1) return fail(GB_EINVAL, "Poisson solve: maxiter must be >= 1");
    cudaStream_t st = (cudaStream_t)stream;
    if (!p->solve_exec)
        if (int rc = build_solve_graph(p)) return rc;
    const size_t bytes = (size_t)p->ops[0]->ng() * sizeof(double);
    // rhos[0][:] = rho; phis[0] = phi  (gpaw/poisson.py:476-482)
    GB_CUDA_TRY(cudaMemcpyAsync(p->rho0, rho, bytes, cudaMemcpyDeviceToDevice, st));
    GB_CUDA_TRY(cudaMemcpyAsync(p->phi0, phi, bytes, cudaMemcpyDeviceToDevice, st));
    k_solve_init<<<1, 1, 0, st>>>(p->ctl, eps, maxiter);
    GB_LAUNCH_CHECK();
    GB_CUDA_TRY(cudaGraphLaunch(p->solve_exec, st));
    GB_CUDA_TRY(cudaMemcpyAsync(phi, p->phi0, bytes, cudaMemcpyDeviceToDevice, st));
    GB_CUDA_TRY(cudaMemcpyAsync(p->ctl_host, p->ctl, sizeof(SolveCtl), cudaMemcpyDeviceToHost, st));
    p->last_maxiter = maxiter;
    return 0;
}

extern "C" int gb_poisson_result(gb_poisson* p, int* niter, double* error) {
    if (!p) return fail(GB_EINVAL, "Poisson result: NULL executor");
    const int it = p->ctl_host->niter;
    if (niter) *niter = it;
    if (error) *error = p->ctl_host->err;
    if (it >= p->last_maxiter)
        return fail(GB_ENOCONV, "Poisson solver did not converge in %d iterations!",
                    p->last_maxiter);
    return 0;
}

extern "C" int gb_poisson_solve_neutral(gb_poisson* p, double* phi, const double* rho, double eps,
                                        int maxiter, int* niter, double* error, void* stream) {
    if (int rc = gb_poisson_solve_neutral_async(p, phi, rho, eps, maxiter, stream)) return rc;
    GB_CUDA_TRY(cudaStreamSynchronize((cudaStream_t)stream));
    return gb_poisson_result(p, niter, error);
}

// ------------------------------------------------- relax without allocation
// Some callers cannot let this library call cudaMalloc: a host program that
// has handed all of HBM to its own memory pool (a cudaMalloc would fail or
// force the pool to release cached blocks), a latency-critical serving loop
// that must not risk the implicit device synchronisation cudaMalloc and
// cudaFree may perform, or a plugin host that forbids allocations outside
// its own allocator.  gb_operator_relax_noalloc serves them: the scratch
// grid that relaxation needs (the Jacobi ping-pong buffer, the Gauss-Seidel
// start-of-sweep snapshot) lives in the fixed device array below instead of
// the operator's lazily allocated buffer.
//
// The array is GB_NOALLOC_MAX_POINTS doubles (16 MiB); every GPU that loads
// the library holds it until the process exits.  All calls share it, so
// calls that overlap on the GPU (other streams, other threads) race; calls
// on one stream are ordered.  It keeps the last call's contents; nothing
// needs to start at zero, because each sweep writes every point of the
// scratch before reading it.
static __device__ __align__(256) double g_relax_scratch[GB_NOALLOC_MAX_POINTS];

namespace {
std::mutex g_noalloc_mu;
// Per device: the address of g_relax_scratch and the CUDA context it was
// looked up in.  After cudaDeviceReset (or any other re-creation of the
// primary context) the module is loaded again and the array may move, so a
// cached address is used only while the current context is the one it came
// from.
struct NoallocSlot {
    void* ptr = nullptr;
    void* ctx = nullptr;
};
NoallocSlot g_noalloc[256];

// cuCtxGetCurrent through the runtime's driver entry point table, so that
// the library needs no link against libcuda.
typedef int (*CtxGetCurrentFn)(void**);
CtxGetCurrentFn ctx_get_current() {
    static CtxGetCurrentFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return (CtxGetCurrentFn) nullptr;
        return (CtxGetCurrentFn)f;
    }();
    return fn;
}
}  // namespace

// Host code must not use g_relax_scratch's name as a device address (it is a
// host-side stand-in); the array's address is looked up with the device
// current, on the first call on that device and again whenever the current
// context has changed since.  The look-up may load the module, which a
// stream capture does not allow: if `st` is capturing and no address is
// cached for this context, the call fails with GB_EINVAL and says so.
static int noalloc_scratch(double** out, cudaStream_t st) {
    int dev = 0;
    GB_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 256) return fail(GB_EINVAL, "relax_noalloc: device index %d", dev);
    void* ctx = nullptr;
    if (CtxGetCurrentFn f = ctx_get_current()) {
        if (f(&ctx) != 0) ctx = nullptr;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    NoallocSlot& slot = g_noalloc[dev];
    if (!slot.ptr || slot.ctx != ctx) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        GB_CUDA_TRY(cudaStreamIsCapturing(st, &cs));
        if (cs != cudaStreamCaptureStatusNone)
            return fail(GB_EINVAL,
                        "relax_noalloc: the first call on a device (or after its context was "
                        "re-created) looks up the scratch array's address and must not run "
                        "inside a stream capture; call it once before capturing");
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_relax_scratch);
        if (e != cudaSuccess || !p)
            return fail(GB_ECUDA, "relax_noalloc: cudaGetSymbolAddress: %s",
                        cudaGetErrorString(e));
        slot.ptr = p;
        slot.ctx = ctx;
    }
    *out = (double*)slot.ptr;
    return 0;
}

extern "C" int gb_operator_relax_noalloc(gb_operator* op, int method, double* f,
                                         const double* s, int nrelax, double w, void* stream) {
    if (!op || !f || !s) return fail(GB_EINVAL, "relax_noalloc: NULL argument");
    if (!op->real) return fail(GB_EINVAL, "relax_noalloc: float64 operators only");
    if (method != 1 && method != 2) return fail(GB_EINVAL, "relax_noalloc: method must be 1 or 2");
    if (op->ng() > (long long)GB_NOALLOC_MAX_POINTS)
        return fail(GB_EINVAL,
                    "relax_noalloc: grid has %lld points, more than the %d this entry point "
                    "supports; use gb_operator_relax",
                    op->ng(), (int)GB_NOALLOC_MAX_POINTS);
    if (nrelax <= 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    double* X = nullptr;
    if (int rc = noalloc_scratch(&X, st)) return rc;
    return relax_with_scratch(op, method, f, s, nrelax, w, X, st);
}
