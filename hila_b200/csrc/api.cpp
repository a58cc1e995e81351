// C-ABI entry points: contexts, lattices, fields and the FP64 operators.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include <cstdlib>
#include <cstring>

#include "hw_internal.h"

namespace hw {

static thread_local std::string g_err;

void set_error(const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    g_err = buf;
}
void clear_error() { g_err.clear(); }

int DevBuf::alloc(size_t n) {
    release();
    if (n == 0) return HW_OK;
    cudaError_t e = cudaMalloc(&ptr, n);
    if (e != cudaSuccess) {
        ptr = nullptr;
        cudaGetLastError();  // reported here, not by the next launch's check too
        set_error("cudaMalloc(%zu bytes) failed: %s", n, cudaGetErrorString(e));
        return e == cudaErrorMemoryAllocation ? HW_ERR_OOM : HW_ERR_CUDA;
    }
    bytes = n;
    return HW_OK;
}
void DevBuf::release() {
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
}

static int alloc_half(HalfBuf &h, int stride) {
    h.stride = stride;
    return h.buf.alloc((size_t)12 * stride * sizeof(double2));
}

int ensure_workspace(hw_lattice *lat) {
    if (!lat->ws) lat->ws.reset(new CgWorkspace());
    CgWorkspace &w = *lat->ws;
    if (w.allocated) return HW_OK;
    int rc;
    for (HalfBuf *h : {&w.r, &w.p, &w.Dp, &w.DDp, &w.src, &w.res, &w.t})
        if ((rc = alloc_half(*h, lat->stride)) != HW_OK) return rc;
    w.allocated = true;
    return HW_OK;
}

int tune_hop(hw_lattice *lat, const hw_gauge *G) {
    if (lat->tuned) return HW_OK;
    lat->tuned = true;
    if (const char *env = std::getenv("HW_HOP_VARIANT")) {
        int v = std::atoi(env);
        lat->g.hop_variant = (v >= 0 && v < kHopVariants) ? v : 0;
        return HW_OK;
    }
    if (lat->Vh <= kHopSplitSites) {
        lat->g.hop_variant = 3;
        return HW_OK;
    }
    int rc;
    if ((rc = ensure_workspace(lat)) != HW_OK) return rc;
    hw_context *ctx = lat->ctx;
    CgWorkspace &w = *lat->ws;
    HW_CUDA(cudaMemsetAsync(w.p.buf.ptr, 0, w.p.buf.bytes, ctx->stream));
    HW_CUDA(cudaMemsetAsync(w.r.buf.ptr, 0, w.r.buf.bytes, ctx->stream));
    // each shape times whole even-odd applies (both hops: scale, then the diagonal
    // term); the best of three trials, after two untimed applies
    auto apply = [&](const Geom &g) {
        launch_hop_scale(g, G->U(), 1, +1, w.p.h(), w.t.h(), 1.0, nullptr, ctx->stream);
        launch_hop_xpay(g, G->U(), 0, +1, w.t.h(), w.p.h(), w.r.h(), -0.01, nullptr, nullptr, ctx->stream);
    };
    float best = 1e30f;
    int best_v = 0;
    for (int v = 0; v < kHopVariants - 1; v++) {
        Geom g = lat->g;
        g.hop_variant = v;
        for (int k = 0; k < 2; k++) apply(g);
        float vbest = 1e30f;
        for (int trial = 0; trial < 3; trial++) {
            HW_CUDA(cudaEventRecord(ctx->ev0, ctx->stream));
            for (int k = 0; k < 3; k++) apply(g);
            HW_CUDA(cudaEventRecord(ctx->ev1, ctx->stream));
            HW_CUDA(cudaEventSynchronize(ctx->ev1));
            float ms = 0;
            HW_CUDA(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
            vbest = std::min(vbest, ms);
        }
        if (vbest < best) {
            best = vbest;
            best_v = v;
        }
    }
    HW_CUDA(cudaGetLastError());
    lat->g.hop_variant = best_v;
    return HW_OK;
}

int ensure_stage(hw_context *ctx, size_t bytes) {
    if (ctx->stage.bytes >= bytes) return HW_OK;
    HW_CUDA(cudaStreamSynchronize(ctx->stream));
    return ctx->stage.alloc(bytes);
}

int ensure_reduction_capacity(hw_context *ctx, long nblocks) {
    const size_t need = red_doubles(nblocks);
    if (ctx->red_capacity_doubles >= need) return HW_OK;
    HW_CUDA(cudaStreamSynchronize(ctx->stream));
    ctx->red_capacity_doubles = 0;  // the old buffer is gone if the new one cannot be had
    int rc = ctx->red_partials.alloc(need * sizeof(double));
    if (rc != HW_OK) return rc;
    ctx->red_capacity_doubles = need;
    return HW_OK;
}

}  // namespace hw

using namespace hw;

extern "C" {

int hw_api_version(void) { return HW_API_VERSION; }

const char *hw_last_error(void) { return g_err.c_str(); }

int hw_device_count(int *count) {
    HW_CHECK_ARG(count, "count is null");
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess) {
        *count = 0;
        set_error("cudaGetDeviceCount: %s", cudaGetErrorString(e));
        return HW_ERR_NO_DEVICE;
    }
    *count = n;
    return HW_OK;
}

int hw_context_create(int device, hw_context **out) {
    HW_CHECK_ARG(out, "ctx out-pointer is null");
    *out = nullptr;
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
        set_error("no CUDA device available");
        return HW_ERR_NO_DEVICE;
    }
    HW_CHECK_ARG(device >= 0 && device < n, "device %d out of range (%d devices)", device, n);
    HW_CUDA(cudaSetDevice(device));
    std::unique_ptr<hw_context> c(new hw_context());
    c->device = device;
    HW_CUDA(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
    int rc;
    if ((rc = c->red_ticket.alloc(64 * sizeof(unsigned))) != HW_OK) return rc;
    HW_CUDA(cudaMemset(c->red_ticket.ptr, 0, 64 * sizeof(unsigned)));
    if ((rc = ensure_reduction_capacity(c.get(), 1 << 16)) != HW_OK) return rc;
    if ((rc = c->cg_state.alloc(sizeof(CgState))) != HW_OK) return rc;
    HW_CUDA(cudaMemset(c->cg_state.ptr, 0, sizeof(CgState)));
    HW_CUDA(cudaMallocHost(&c->cg_state_host, sizeof(CgState)));
    HW_CUDA(cudaEventCreate(&c->ev0));
    HW_CUDA(cudaEventCreate(&c->ev1));
    *out = c.release();
    clear_error();
    return HW_OK;
}

int hw_context_destroy(hw_context *ctx) {
    if (!ctx) return HW_OK;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    destroy_engines(ctx);
    if (ctx->cg_state_host) cudaFreeHost(ctx->cg_state_host);
    if (ctx->ev0) cudaEventDestroy(ctx->ev0);
    if (ctx->ev1) cudaEventDestroy(ctx->ev1);
    ctx->red_partials.release();
    ctx->red_ticket.release();
    ctx->cg_state.release();
    cudaStreamDestroy(ctx->stream);
    delete ctx;
    return HW_OK;
}

int hw_context_synchronize(hw_context *ctx) {
    HW_CHECK_ARG(ctx, "ctx is null");
    HW_CUDA(cudaSetDevice(ctx->device));
    HW_CUDA(cudaStreamSynchronize(ctx->stream));
    return HW_OK;
}

int hw_lattice_create(hw_context *ctx, const int dims[4], int t_antiperiodic, hw_lattice **out) {
    HW_CHECK_ARG(ctx && dims && out, "null argument");
    *out = nullptr;
    long V = 1;
    for (int d = 0; d < 4; d++) {
        HW_CHECK_ARG(dims[d] >= 2 && dims[d] % 2 == 0, "dims[%d] = %d: every extent must be even and >= 2", d,
                     dims[d]);
        V *= dims[d];
    }
    HW_CHECK_ARG(V / 2 < (1L << 30), "lattice too large (%ld sites)", V);
    std::unique_ptr<hw_lattice> l(new hw_lattice());
    l->ctx = ctx;
    for (int d = 0; d < 4; d++) l->dims[d] = dims[d];
    l->tap = t_antiperiodic ? 1 : 0;
    l->V = V;
    l->Vh = V / 2;
    l->stride = padded_stride(l->Vh);
    geom_setup(l->g, dims, l->tap);
    *out = l.release();
    clear_error();
    return HW_OK;
}

int hw_lattice_destroy(hw_lattice *lat) {
    if (!lat) return HW_OK;
    cudaSetDevice(lat->ctx->device);
    cudaStreamSynchronize(lat->ctx->stream);
    delete lat;
    return HW_OK;
}

int hw_lattice_volume(const hw_lattice *lat, int64_t *volume) {
    HW_CHECK_ARG(lat && volume, "null argument");
    *volume = lat->V;
    return HW_OK;
}

int hw_gauge_create(hw_lattice *lat, const double *links, int link_format, hw_gauge **out) {
    HW_CHECK_ARG(lat && links && out, "null argument");
    HW_CHECK_ARG(link_format == 18 || link_format == 12, "link_format must be 18 or 12");
    *out = nullptr;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    std::unique_ptr<hw_gauge> G(new hw_gauge());
    G->lat = lat;
    G->link_format = link_format;
    const int planes = link_format == 12 ? 6 : 9;
    int rc;
    if ((rc = G->f64.alloc((size_t)8 * planes * lat->stride * sizeof(double2))) != HW_OK) return rc;
    HW_CUDA(cudaMemsetAsync(G->f64.ptr, 0, G->f64.bytes, ctx->stream));
    // stage one direction at a time: V links of 18 doubles
    if ((rc = ensure_stage(ctx, (size_t)lat->V * 18 * sizeof(double))) != HW_OK) return rc;
    DevBuf &stage = ctx->stage;
    Geom g1 = lat->g;
    for (int dir = 0; dir < 4; dir++) {
        HW_CUDA(cudaMemcpyAsync(stage.ptr, links + (size_t)dir * lat->V * 18, (size_t)lat->V * 18 * sizeof(double),
                                cudaMemcpyHostToDevice, ctx->stream));
        for (int par = 0; par < 2; par++) {
            double2 *dst = G->f64.as<double2>() + (size_t)((par * 4 + dir) * planes) * lat->stride;
            launch_links_lex_to_eo(g1, stage.as<double>(), dst, planes, lat->stride, par, ctx->stream);
        }
    }
    HW_CUDA(cudaGetLastError());
    HW_CUDA(cudaStreamSynchronize(ctx->stream));
    *out = G.release();
    clear_error();
    return HW_OK;
}

int hw_gauge_destroy(hw_gauge *gauge) {
    if (!gauge) return HW_OK;
    cudaSetDevice(gauge->lat->ctx->device);
    cudaStreamSynchronize(gauge->lat->ctx->stream);
    delete gauge;
    return HW_OK;
}

int hw_field_create(hw_lattice *lat, hw_field **out) {
    HW_CHECK_ARG(lat && out, "null argument");
    *out = nullptr;
    HW_CUDA(cudaSetDevice(lat->ctx->device));
    std::unique_ptr<hw_field> f(new hw_field());
    f->lat = lat;
    int rc;
    for (int p = 0; p < 2; p++) {
        if ((rc = alloc_half(f->half[p], lat->stride)) != HW_OK) return rc;
        HW_CUDA(cudaMemsetAsync(f->half[p].buf.ptr, 0, f->half[p].buf.bytes, lat->ctx->stream));
    }
    HW_CUDA(cudaStreamSynchronize(lat->ctx->stream));
    *out = f.release();
    clear_error();
    return HW_OK;
}

int hw_field_destroy(hw_field *field) {
    if (!field) return HW_OK;
    cudaSetDevice(field->lat->ctx->device);
    cudaStreamSynchronize(field->lat->ctx->stream);
    delete field;
    return HW_OK;
}

int hw_field_upload(hw_field *f, const double *host, int parity) {
    HW_CHECK_ARG(f && host, "null argument");
    HW_CHECK_ARG(parity >= 1 && parity <= 3, "parity must be HW_EVEN, HW_ODD or HW_ALL");
    hw_lattice *lat = f->lat;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    const size_t bytes = (size_t)lat->V * 24 * sizeof(double);
    int rc;
    if ((rc = ensure_stage(ctx, bytes)) != HW_OK) return rc;
    DevBuf &stage = ctx->stage;
    HW_CUDA(cudaMemcpyAsync(stage.ptr, host, bytes, cudaMemcpyHostToDevice, ctx->stream));
    for (int p = 0; p < 2; p++)
        if (parity & (1 << p)) launch_spinor_lex_to_eo(lat->g, stage.as<double>(), p, f->half[p].h(), ctx->stream);
    HW_CUDA(cudaGetLastError());
    HW_CUDA(cudaStreamSynchronize(ctx->stream));
    return HW_OK;
}

int hw_field_download(const hw_field *f, double *host, int parity) {
    HW_CHECK_ARG(f && host, "null argument");
    HW_CHECK_ARG(parity >= 1 && parity <= 3, "parity must be HW_EVEN, HW_ODD or HW_ALL");
    hw_lattice *lat = f->lat;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    const size_t bytes = (size_t)lat->V * 24 * sizeof(double);
    int rc;
    if ((rc = ensure_stage(ctx, bytes)) != HW_OK) return rc;
    DevBuf &stage = ctx->stage;
    if (parity != 3) {
        // keep the host's sites of the other parity: start from the host array
        HW_CUDA(cudaMemcpyAsync(stage.ptr, host, bytes, cudaMemcpyHostToDevice, ctx->stream));
    }
    for (int p = 0; p < 2; p++)
        if (parity & (1 << p)) launch_spinor_eo_to_lex(lat->g, f->half[p].h(), p, stage.as<double>(), ctx->stream);
    HW_CUDA(cudaGetLastError());
    return copy_to_host(ctx, host, stage.ptr, bytes);
}

int hw_field_upload_eo(hw_field *f, const double *host, int parity) {
    HW_CHECK_ARG(f && host, "null argument");
    HW_CHECK_ARG(parity >= 1 && parity <= 3, "parity must be HW_EVEN, HW_ODD or HW_ALL");
    hw_lattice *lat = f->lat;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    const size_t half = (size_t)lat->Vh * 24;
    int rc;
    if ((rc = ensure_stage(ctx, half * sizeof(double))) != HW_OK) return rc;
    for (int p = 0; p < 2; p++)
        if (parity & (1 << p)) {
            HW_CUDA(cudaMemcpyAsync(ctx->stage.ptr, host + p * half, half * sizeof(double), cudaMemcpyHostToDevice,
                                    ctx->stream));
            launch_aos_to_soa((int)lat->Vh, ctx->stage.as<double>(), f->half[p].h(), ctx->stream);
        }
    HW_CUDA(cudaGetLastError());
    HW_CUDA(cudaStreamSynchronize(ctx->stream));
    return HW_OK;
}

int hw_field_download_eo(const hw_field *f, double *host, int parity) {
    HW_CHECK_ARG(f && host, "null argument");
    HW_CHECK_ARG(parity >= 1 && parity <= 3, "parity must be HW_EVEN, HW_ODD or HW_ALL");
    hw_lattice *lat = f->lat;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    const size_t half = (size_t)lat->Vh * 24;
    int rc;
    if ((rc = ensure_stage(ctx, half * sizeof(double))) != HW_OK) return rc;
    for (int p = 0; p < 2; p++)
        if (parity & (1 << p)) {
            launch_soa_to_aos((int)lat->Vh, f->half[p].h(), ctx->stage.as<double>(), ctx->stream);
            HW_CUDA(cudaGetLastError());
            if ((rc = copy_to_host(ctx, host + p * half, ctx->stage.ptr, half * sizeof(double))) != HW_OK) return rc;
        }
    return HW_OK;
}

int hw_field_zero(hw_field *f, int parity) {
    HW_CHECK_ARG(f, "null argument");
    HW_CHECK_ARG(parity >= 1 && parity <= 3, "parity must be HW_EVEN, HW_ODD or HW_ALL");
    hw_context *ctx = f->lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    for (int p = 0; p < 2; p++)
        if (parity & (1 << p)) HW_CUDA(cudaMemsetAsync(f->half[p].buf.ptr, 0, f->half[p].buf.bytes, ctx->stream));
    HW_CUDA(cudaStreamSynchronize(ctx->stream));
    return HW_OK;
}

// ------------------------------------------------------------------ operators

static int check_op(const hw_gauge *g, const hw_field *in, const hw_field *out) {
    HW_CHECK_ARG(g && in && out, "null argument");
    HW_CHECK_ARG(in->lat == g->lat && out->lat == g->lat, "fields and gauge belong to different lattices");
    return HW_OK;
}

// out_e = d in_e - kappa^2 H^{eo}_s H^{oe}_s in_e, d = 1 + m_h (d = 1: wilson.h:272-289;
// m_h > 0: Hasenbusch_operator::apply / dagger, Hasenbusch.h:39-47)
static int eo_apply(const hw_gauge *G, double kappa, const hw_field *in, hw_field *out, int sign, double d = 1.0) {
    int rc = check_op(G, in, out);
    if (rc != HW_OK) return rc;
    hw_lattice *lat = G->lat;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    if ((rc = ensure_workspace(lat)) != HW_OK) return rc;
    if ((rc = tune_hop(lat, G)) != HW_OK) return rc;
    CgWorkspace &w = *lat->ws;
    // t_o = H^{oe}_s in_e ; out_e = in_e - kappa^2 H^{eo}_s t_o ; out_o = 0  (wilson.h:272-279);
    // the second hop clears out_o as it goes (the odd half of `in` is not read)
    launch_hop_scale(lat->g, G->U(), 1, sign, in->half[0].h(), w.t.h(), 1.0, nullptr, ctx->stream);
    launch_hop_xpay(lat->g, G->U(), 0, sign, w.t.h(), in->half[0].h(), out->half[0].h(), -kappa * kappa, nullptr,
                    nullptr, ctx->stream, d, out->half[1].buf.as<double2>());
    // stream-ordered: later calls on this context see the result; downloads synchronise
    HW_CUDA(cudaGetLastError());
    return HW_OK;
}

int hw_wilson_evenodd_apply(const hw_gauge *gauge, double kappa, const hw_field *in, hw_field *out) {
    return eo_apply(gauge, kappa, in, out, +1);
}

int hw_wilson_evenodd_dagger(const hw_gauge *gauge, double kappa, const hw_field *in, hw_field *out) {
    return eo_apply(gauge, kappa, in, out, -1);
}

int hw_hasenbusch_evenodd_apply(const hw_gauge *gauge, double kappa, double mh, const hw_field *in, hw_field *out) {
    HW_CHECK_ARG(std::isfinite(mh), "mh must be finite");
    return eo_apply(gauge, kappa, in, out, +1, 1.0 + mh);
}

int hw_hasenbusch_evenodd_dagger(const hw_gauge *gauge, double kappa, double mh, const hw_field *in, hw_field *out) {
    HW_CHECK_ARG(std::isfinite(mh), "mh must be finite");
    return eo_apply(gauge, kappa, in, out, -1, 1.0 + mh);
}

int hw_wilson_apply(const hw_gauge *G, double kappa, int sign, const hw_field *in, hw_field *out) {
    int rc = check_op(G, in, out);
    if (rc != HW_OK) return rc;
    HW_CHECK_ARG(sign == 1 || sign == -1, "sign must be +1 or -1");
    HW_CHECK_ARG(in != out, "in and out must be different fields");
    hw_lattice *lat = G->lat;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    if ((rc = tune_hop(lat, G)) != HW_OK) return rc;
    // out_p = in_p - kappa H_s in_{1-p} for both parities (wilson.h:183-192)
    for (int p = 0; p < 2; p++)
        launch_hop_xpay(lat->g, G->U(), p, sign, in->half[1 - p].h(), in->half[p].h(), out->half[p].h(), -kappa,
                        nullptr, nullptr, ctx->stream);
    HW_CUDA(cudaGetLastError());
    return HW_OK;
}

int hw_wilson_hop(const hw_gauge *G, double kappa, const hw_field *in, hw_field *out, int parity, int sign, int set) {
    int rc = check_op(G, in, out);
    if (rc != HW_OK) return rc;
    HW_CHECK_ARG(parity == HW_EVEN || parity == HW_ODD, "parity must be HW_EVEN or HW_ODD");
    HW_CHECK_ARG(sign == 1 || sign == -1, "sign must be +1 or -1");
    hw_lattice *lat = G->lat;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    const int p = parity == HW_EVEN ? 0 : 1;
    if (set)
        launch_hop_scale(lat->g, G->U(), p, sign, in->half[1 - p].h(), out->half[p].h(), -kappa, nullptr,
                         ctx->stream);
    else
        launch_hop_xpay(lat->g, G->U(), p, sign, in->half[1 - p].h(), out->half[p].h(), out->half[p].h(), -kappa,
                        nullptr, nullptr, ctx->stream);
    HW_CUDA(cudaGetLastError());
    return HW_OK;
}

int hw_context_stream(hw_context *ctx, void **stream) {
    HW_CHECK_ARG(ctx && stream, "null argument");
    *stream = (void *)ctx->stream;
    return HW_OK;
}

}  // extern "C"

CgWorkspace::~CgWorkspace() {
    if (init_exec) cudaGraphExecDestroy(init_exec);
    if (loop_exec) cudaGraphExecDestroy(loop_exec);
}

LoopCgWorkspace::~LoopCgWorkspace() {
    if (loop_exec) cudaGraphExecDestroy(loop_exec);
    *total -= kept;
}

LoopCgLease::~LoopCgLease() {
    if (!ws || (done && ws->kept)) return;
    size_t bytes = ws->t.bytes;
    for (int h = 0; h < 2; h++)
        for (const hw::DevBuf *d : {&ws->r[h], &ws->p[h], &ws->Dp[h], &ws->x[h]}) bytes += d->bytes;
    if (done && (*ws->total += bytes) <= kLoopWsKeep) {
        ws->kept = bytes;
        return;
    }
    if (done) *ws->total -= bytes;
    ws.reset();
}

hw_lattice::~hw_lattice() {
    hw_field_destroy(host_b);
    hw_field_destroy(host_x);
}

extern "C" {

int hw_host_alloc(size_t bytes, void **ptr) {
    HW_CHECK_ARG(ptr, "ptr is null");
    *ptr = nullptr;
    HW_CUDA(cudaMallocHost(ptr, bytes));
    return HW_OK;
}

int hw_host_free(void *ptr) {
    if (ptr) HW_CUDA(cudaFreeHost(ptr));
    return HW_OK;
}

int hw_wilson_evenodd_solve_host(const hw_gauge *G, double kappa, const double *b_host, double *x_host,
                                 const hw_cg_params *params, hw_cg_result *result) {
    HW_CHECK_ARG(G && b_host && x_host, "null argument");
    hw_lattice *lat = G->lat;
    std::lock_guard<std::recursive_mutex> lk(lat->ctx->mu);
    int rc;
    if (!lat->host_b && (rc = hw_field_create(lat, &lat->host_b)) != HW_OK) return rc;
    if (!lat->host_x && (rc = hw_field_create(lat, &lat->host_x)) != HW_OK) return rc;
    if ((rc = hw_field_upload(lat->host_b, b_host, HW_EVEN)) != HW_OK) return rc;
    if ((rc = hw_field_zero(lat->host_x, HW_ALL)) != HW_OK) return rc;
    int st = hw_wilson_evenodd_solve(G, kappa, lat->host_b, lat->host_x, params, result);
    if (st != HW_OK && st != HW_ERR_NOT_CONVERGED) return st;
    if ((rc = hw_field_download(lat->host_x, x_host, HW_ALL)) != HW_OK) return rc;
    return st;
}

}  // extern "C"

namespace hw {
// (M_s + m_h) on EVEN half fields, stream-ordered, through the lattice's ODD
// workspace field (context lock held; workspace and hop shape ready)
void eo_apply_half(const hw_gauge *G, double kappa, HalfF64 in, HalfF64 out, int sign, double d) {
    hw_lattice *lat = G->lat;
    CgWorkspace &w = *lat->ws;
    launch_hop_scale(lat->g, G->U(), 1, sign, in, w.t.h(), 1.0, nullptr, lat->ctx->stream);
    launch_hop_xpay(lat->g, G->U(), 0, sign, w.t.h(), in, out, -kappa * kappa, nullptr, nullptr, lat->ctx->stream, d);
}
}  // namespace hw
