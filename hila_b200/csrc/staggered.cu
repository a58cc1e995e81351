// Staggered fermions (libraries/dirac/staggered.h): colour-vector fields, the
// even-odd operator, its force, and CG on its normal equations, all in FP64.
//
//   eta_d(x)  = ((sum_{d' < d} x_d') % 2) * 2 - 1      (staggered.h:14-28 as coded; its
//                                                       comment states the opposite sign)
//   hop_s v(x) = 0.5 s sum_d eta_d(x) [U_d(x) v(x+d) - U_d(x-d)^dag v(x-d)]   (:48-68)
//   M_s in    : out_o = (1/m) hop_s in_e ;  out_e = m in_e + hop_s out_o       (:224-242)
// with the fermion boundary sign on values gathered across the t boundary.
// out_o keeps (1/m) D_oe in_e, as the reference leaves it.  Fields are two
// half lattices of 3 double2 planes (stride = the lattice's padded parity size).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "cg_loop.cuh"
#include "hw_internal.h"
#include "reduce.cuh"
#include "staggered_math.cuh"
#include "storage.cuh"


namespace hw {
namespace {

constexpr int kStagBlock = 128;
constexpr int kStagVecBlock = 256;

HalfStag half_of(const hw_stag_field *f, int p) {
    return HalfStag{f->half[p].as<double2>(), f->lat->stride};
}

// out = a * 0.5 SIGN acc  (x null)   or   out = m x + 0.5 SIGN acc
template <int SIGN, class Lk>
__global__ void __launch_bounds__(kStagBlock) k_stag_hop(Geom g, Lk U, int par, HalfStag in, HalfStag x, double m,
                                                          double a, HalfStag out) {
    const int i = blockIdx.x * kStagBlock + threadIdx.x;
    if (i >= g.Vh) return;
    Cx<double> acc[3];
    stag_hop_site(g, U, par, i, in, acc);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const Cx<double> h = (0.5 * SIGN) * acc[k];
        out.st(k, i, x.p ? m * x.ld(k, i) + h : a * h);
    }
}

template <class Lk>
void stag_hop(const Geom &g, const Lk &U, int par, int sign, HalfStag in, HalfStag x, double m, double a,
              HalfStag out, cudaStream_t s) {
    const int blocks = (int)((g.Vh + kStagBlock - 1) / kStagBlock);
    if (sign > 0)
        k_stag_hop<1><<<blocks, kStagBlock, 0, s>>>(g, U, par, in, x, m, a, out);
    else
        k_stag_hop<-1><<<blocks, kStagBlock, 0, s>>>(g, U, par, in, x, m, a, out);
}

// hop over both link formats
void stag_hop_any(const hw_gauge *G, int par, int sign, HalfStag in, HalfStag x, double m, double a, HalfStag out,
                  cudaStream_t s) {
    const GaugeF64 U = G->U();
    const Geom &g = G->lat->g;
    if (U.planes == 9)
        stag_hop(g, LinksF64x18{U.p, U.stride}, par, sign, in, x, m, a, out, s);
    else
        stag_hop(g, LinksF64x12{U.p, U.stride}, par, sign, in, x, m, a, out, s);
}

// M_s: out_o = (1/m) hop in_e ; out_e = m in_e + hop out_o
void stag_eo_apply(const hw_gauge *G, double mass, HalfStag in_e, HalfStag out_e, HalfStag out_o, int sign,
                   cudaStream_t s) {
    stag_hop_any(G, 1, sign, in_e, HalfStag{nullptr, 0}, 0.0, 1.0 / mass, out_o, s);
    stag_hop_any(G, 0, sign, out_o, in_e, mass, 0.0, out_e, s);
}

// ---- layout: host lexicographic [V][3] complex <-> half lattices
__global__ void k_stag_layout(Geom g, int par, double2 *lex, HalfStag f, int to_eo) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.Vh) return;
    int c[4];
    site_coords(g, i, par, c);
    const size_t s = c[0] + (size_t)g.L[0] * (c[1] + (size_t)g.L[1] * (c[2] + (size_t)g.L[2] * c[3]));
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (to_eo)
            f.p[(size_t)k * f.stride + i] = lex[s * 3 + k];
        else
            lex[s * 3 + k] = f.p[(size_t)k * f.stride + i];
    }
}

// ---- CG on the normal equations, resident on the device (the body of a CUDA-graph WHILE
// node, as solver_f64.cpp): t = (1/m) D p, Dp = m p + D t with |Dp|^2 -> alpha, t = (1/m)
// D^dag Dp, then r -= alpha M^dag Dp, x += alpha p with |r|^2 -> beta and the stopping
// decision, and p = r + beta p.  (A host loop over the operator, dot products and axpys with
// two host synchronisations per iteration and its workspace allocated per call took 98 us
// per iteration at 14x18x12x26.)  Partial sums are added in block order.

// t = a 0.5 s hop in
struct StagScale {
    static constexpr int NRED = 0;
    HalfStag out;
    double a;
    const CgState *st;
    __device__ bool skip() const { return st && st->status != CG_RUNNING; }
    __device__ void operator()(int i, const Cx<double> (&h)[3], double *) const {
#pragma unroll
        for (int k = 0; k < 3; k++) out.st(k, i, a * h[k]);
    }
    __device__ void operator()(const double *) const {}
};

// Dp = m p + h; ALPHA: |Dp|^2 -> alpha
template <bool ALPHA>
struct StagMul {
    static constexpr int NRED = ALPHA ? 1 : 0;
    HalfStag p, Dp;
    double m;
    CgState *st;
    __device__ bool skip() const { return ALPHA && st->status != CG_RUNNING; }
    __device__ void operator()(int i, const Cx<double> (&h)[3], double *red) const {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const Cx<double> v = m * p.ldp(k, i) + h[k];
            Dp.st(k, i, v);
            red[0] += norm2(v);
        }
    }
    __device__ void operator()(const double *tot) const {
        cg_alpha(st, tot[0]);
    }
};

// r = p = b - (m Dp + h); |r|^2, |b|^2 -> the start of the iteration
struct StagInit {
    static constexpr int NRED = 2;
    HalfStag Dp, b, r, p;
    double m, acc2;
    int maxiter;
    CgState *st;
    __device__ bool skip() const { return false; }
    __device__ void operator()(int i, const Cx<double> (&h)[3], double *red) const {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const Cx<double> bv = b.ldp(k, i);
            const Cx<double> v = bv - (m * Dp.ldp(k, i) + h[k]);
            r.st(k, i, v);
            p.st(k, i, v);
            red[0] += norm2(v);
            red[1] += norm2(bv);
        }
    }
    __device__ void operator()(const double *tot) const {
        cg_start(st, tot[0], tot[1], acc2, maxiter);
    }
};

// r -= alpha (m Dp + h), x += alpha p; |r|^2 -> beta, status
struct StagUpdate {
    static constexpr int NRED = 1;
    HalfStag Dp, r, x, p;
    double m;
    CgState *st;
    __device__ bool skip() const { return st->status != CG_RUNNING; }
    __device__ void operator()(int i, const Cx<double> (&h)[3], double *red) const {
        const double alpha = st->alpha;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            const Cx<double> rv = r.ldp(k, i) - alpha * (m * Dp.ldp(k, i) + h[k]);
            r.st(k, i, rv);
            x.st(k, i, x.ldp(k, i) + alpha * p.ldp(k, i));
            red[0] += norm2(rv);
        }
    }
    __device__ void operator()(const double *tot) const {
        cg_step(st, tot[0]);
    }
};

// |b - (m Dp + h)|^2
struct StagResidual {
    static constexpr int NRED = 1;
    HalfStag Dp, b;
    double m;
    CgState *st;
    __device__ bool skip() const { return false; }
    __device__ void operator()(int i, const Cx<double> (&h)[3], double *red) const {
#pragma unroll
        for (int k = 0; k < 3; k++) red[0] += norm2(b.ldp(k, i) - (m * Dp.ldp(k, i) + h[k]));
    }
    __device__ void operator()(const double *tot) const { st->res_num2 = tot[0]; }
};

template <int SIGN, class Lk, class Epi>
__global__ void __launch_bounds__(kStagBlock) k_stag_cg(Geom g, Lk U, int par, HalfStag in, Epi epi, RedBuf red) {
    if (epi.skip()) return;
    const int i = blockIdx.x * kStagBlock + threadIdx.x;
    constexpr int NR = Epi::NRED > 0 ? Epi::NRED : 1;
    double v[NR];
#pragma unroll
    for (int k = 0; k < NR; k++) v[k] = 0.0;
    if (i < g.Vh) {
        Cx<double> acc[3];
        stag_hop_site(g, U, par, i, in, acc);
#pragma unroll
        for (int k = 0; k < 3; k++) acc[k] = (0.5 * SIGN) * acc[k];
        epi(i, acc, v);
    }
    if constexpr (Epi::NRED > 0) grid_reduce<Epi::NRED, kStagBlock>(v, red.partials, red.ticket, epi);
}

// p = r + beta p
__global__ void __launch_bounds__(kStagVecBlock) k_stag_pupdate(int Vh, HalfStag r, HalfStag p, CgState *st,
                                                               cudaGraphConditionalHandle cond) {
    if (blockIdx.x == 0 && threadIdx.x == 0) loop_next(st, cond, 1);
    if (!st->do_pupdate) return;
    const int i = blockIdx.x * kStagVecBlock + threadIdx.x;
    if (i >= Vh) return;
    const double beta = st->beta;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const Cx<double> rv = r.ldp(k, i), pv = p.ldp(k, i);
        p.st(k, i, {fma(beta, pv.re, rv.re), fma(beta, pv.im, rv.im)});
    }
}

template <class Epi>
void stag_cg(const hw_gauge *G, int par, int sign, HalfStag in, const Epi &epi, RedBuf red, cudaStream_t s) {
    const GaugeF64 U = G->U();
    const Geom &g = G->lat->g;
    const long nb = (g.Vh + kStagBlock - 1) / kStagBlock;
    const dim3 grid = Epi::NRED > 0 ? red.grid(Epi::NRED, nb) : dim3((unsigned)nb);
    const LinksF64x18 U18{U.p, U.stride};
    const LinksF64x12 U12{U.p, U.stride};
    if (U.planes == 9) {
        if (sign > 0)
            k_stag_cg<1><<<grid, kStagBlock, 0, s>>>(g, U18, par, in, epi, red);
        else
            k_stag_cg<-1><<<grid, kStagBlock, 0, s>>>(g, U18, par, in, epi, red);
    } else {
        if (sign > 0)
            k_stag_cg<1><<<grid, kStagBlock, 0, s>>>(g, U12, par, in, epi, red);
        else
            k_stag_cg<-1><<<grid, kStagBlock, 0, s>>>(g, U12, par, in, epi, red);
    }
}

// ---- force (staggered.h:70-86, 246-265); t1 = (1/m) hop_{-s} chi, t2 = (1/m) hop_s psi on ODD
//   x even: F_d = -s/2 eta_d t1(x+d) (x) psi(x) + s/2 eta_d t2(x+d) (x) chi(x)
//   x odd:  F_d =  s/2 eta_d psi(x+d) (x) t1(x) - s/2 eta_d chi(x+d) (x) t2(x)
// (eta_d(x+d) = eta_d(x): it depends on the coordinates below d only)
template <int SIGN>
__global__ void __launch_bounds__(kStagBlock) k_stag_force(Geom g, HalfStag chi, HalfStag psi, HalfStag t1,
                                                            HalfStag t2, long V, double2 *out) {
    const int par = blockIdx.y;
    const int i = blockIdx.x * kStagBlock + threadIdx.x;
    if (i >= g.Vh) return;
    const SiteNbrs n = site_neighbours(g, i, par);
    int c[4];
    site_coords(g, i, par, c);
    const long lex = c[0] + (long)g.L[0] * (c[1] + (long)g.L[1] * (c[2] + (long)g.L[2] * c[3]));
    const HalfStag &A1 = par == 0 ? t1 : psi, &B1 = par == 0 ? psi : t1;
    const HalfStag &A2 = par == 0 ? t2 : chi, &B2 = par == 0 ? chi : t2;
    const double f1 = par == 0 ? -0.5 * SIGN : 0.5 * SIGN, f2 = -f1;
#pragma unroll
    for (int d = 0; d < 4; d++) {
        const int y = n.fwd[d];
        const double e = (d == 3 && n.tfwd_wrap) ? -stag_eta(c, d) : stag_eta(c, d);
        double2 *o = out + ((size_t)d * V + lex) * 9;
#pragma unroll
        for (int a = 0; a < 3; a++) {
            const Cx<double> a1 = A1.ld(a, y), a2 = A2.ld(a, y);
#pragma unroll
            for (int b = 0; b < 3; b++) {
                const Cx<double> v = (f1 * e) * cmul(a1, conj(B1.ld(b, i))) + (f2 * e) * cmul(a2, conj(B2.ld(b, i)));
                o[a * 3 + b] = make_double2(v.re, v.im);
            }
        }
    }
}

}  // namespace
}  // namespace hw

using namespace hw;

namespace {

int check_stag_op(const hw_gauge *G, const hw_stag_field *a, const hw_stag_field *b, double mass) {
    HW_CHECK_ARG(G && a && b, "null argument");
    HW_CHECK_ARG(a->lat == G->lat && b->lat == G->lat, "fields and gauge live on different lattices");
    HW_CHECK_ARG(std::isfinite(mass) && mass != 0.0, "mass must be finite and non-zero");
    return HW_OK;
}

// the lattice's staggered workspace (five half-lattice fields); the caller holds a lease on it
int ensure_stag_ws(hw_lattice *lat) {
    if (!lat->stag_ws) lat->stag_ws.reset(new LoopCgWorkspace(lat->ctx->loop_ws_bytes));
    LoopCgWorkspace &w = *lat->stag_ws;
    int rc;
    for (DevBuf *d : {&w.r[0], &w.p[0], &w.Dp[0], &w.x[0], &w.t})
        if (!d->ptr && (rc = d->alloc((size_t)3 * lat->stride * sizeof(double2))) != HW_OK) return rc;
    return HW_OK;
}

int stag_apply(const hw_gauge *G, double mass, const hw_stag_field *in, hw_stag_field *out, int sign) {
    int rc = check_stag_op(G, in, out, mass);
    if (rc != HW_OK) return rc;
    HW_CHECK_ARG(in != out, "in and out must be different fields");
    hw_context *ctx = G->lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    stag_eo_apply(G, mass, half_of(in, 0), half_of(out, 0), half_of(out, 1), sign, ctx->stream);
    HW_CUDA(cudaGetLastError());
    return HW_OK;
}

}  // namespace

extern "C" {

int hw_stag_field_create(hw_lattice *lat, hw_stag_field **out) {
    HW_CHECK_ARG(lat && out, "null argument");
    *out = nullptr;
    std::lock_guard<std::recursive_mutex> lk(lat->ctx->mu);
    HW_CUDA(cudaSetDevice(lat->ctx->device));
    std::unique_ptr<hw_stag_field> f(new hw_stag_field());
    f->lat = lat;
    for (int p = 0; p < 2; p++) {
        int rc = f->half[p].alloc((size_t)3 * lat->stride * sizeof(double2));
        if (rc != HW_OK) return rc;
        HW_CUDA(cudaMemsetAsync(f->half[p].ptr, 0, f->half[p].bytes, lat->ctx->stream));
    }
    HW_CUDA(cudaStreamSynchronize(lat->ctx->stream));
    *out = f.release();
    return HW_OK;
}

int hw_stag_field_destroy(hw_stag_field *f) {
    if (!f) return HW_OK;
    {
        std::lock_guard<std::recursive_mutex> lk(f->lat->ctx->mu);
        cudaSetDevice(f->lat->ctx->device);
        for (auto &h : f->half) h.release();
    }
    delete f;
    return HW_OK;
}

int hw_stag_field_upload(hw_stag_field *f, const double *host, int parity) {
    HW_CHECK_ARG(f && host, "null argument");
    HW_CHECK_ARG(parity >= 1 && parity <= 3, "parity must be HW_EVEN, HW_ODD or HW_ALL");
    hw_lattice *lat = f->lat;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    const size_t bytes = (size_t)lat->V * 6 * sizeof(double);
    int rc;
    if ((rc = ensure_stage(ctx, bytes)) != HW_OK) return rc;
    HW_CUDA(cudaMemcpyAsync(ctx->stage.ptr, host, bytes, cudaMemcpyHostToDevice, ctx->stream));
    for (int p = 0; p < 2; p++)
        if (parity & (1 << p))
            k_stag_layout<<<(unsigned)((lat->Vh + 255) / 256), 256, 0, ctx->stream>>>(
                lat->g, p, ctx->stage.as<double2>(), half_of(f, p), 1);
    HW_CUDA(cudaGetLastError());
    HW_CUDA(cudaStreamSynchronize(ctx->stream));
    return HW_OK;
}

int hw_stag_field_download(const hw_stag_field *f, double *host, int parity) {
    HW_CHECK_ARG(f && host, "null argument");
    HW_CHECK_ARG(parity >= 1 && parity <= 3, "parity must be HW_EVEN, HW_ODD or HW_ALL");
    hw_lattice *lat = f->lat;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    const size_t bytes = (size_t)lat->V * 6 * sizeof(double);
    int rc;
    if ((rc = ensure_stage(ctx, bytes)) != HW_OK) return rc;
    // sites of the other parity come back as zero
    HW_CUDA(cudaMemsetAsync(ctx->stage.ptr, 0, bytes, ctx->stream));
    for (int p = 0; p < 2; p++)
        if (parity & (1 << p))
            k_stag_layout<<<(unsigned)((lat->Vh + 255) / 256), 256, 0, ctx->stream>>>(
                lat->g, p, ctx->stage.as<double2>(), half_of(f, p), 0);
    HW_CUDA(cudaGetLastError());
    return copy_to_host(ctx, host, ctx->stage.ptr, bytes);
}

int hw_stag_field_zero(hw_stag_field *f, int parity) {
    HW_CHECK_ARG(f, "null argument");
    HW_CHECK_ARG(parity >= 1 && parity <= 3, "parity must be HW_EVEN, HW_ODD or HW_ALL");
    hw_context *ctx = f->lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    for (int p = 0; p < 2; p++)
        if (parity & (1 << p)) HW_CUDA(cudaMemsetAsync(f->half[p].ptr, 0, f->half[p].bytes, ctx->stream));
    HW_CUDA(cudaStreamSynchronize(ctx->stream));
    return HW_OK;
}

int hw_staggered_evenodd_apply(const hw_gauge *gauge, double mass, const hw_stag_field *in, hw_stag_field *out) {
    return stag_apply(gauge, mass, in, out, +1);
}

int hw_staggered_evenodd_dagger(const hw_gauge *gauge, double mass, const hw_stag_field *in, hw_stag_field *out) {
    return stag_apply(gauge, mass, in, out, -1);
}

int hw_staggered_evenodd_force(const hw_gauge *gauge, double mass, const hw_stag_field *chi, const hw_stag_field *psi,
                               int sign, double *force) {
    int rc = check_stag_op(gauge, chi, psi, mass);
    if (rc != HW_OK) return rc;
    HW_CHECK_ARG(force, "null argument");
    HW_CHECK_ARG(sign == 1 || sign == -1, "sign must be +1 or -1");
    hw_lattice *lat = gauge->lat;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    const int stride = lat->stride;
    LoopCgLease lease{lat->stag_ws};
    if ((rc = ensure_stag_ws(lat)) != HW_OK) return rc;
    DevBuf own;
    void *out = nullptr;
    const size_t bytes = (size_t)36 * lat->V * sizeof(double2);
    if ((rc = force_buffer(ctx, bytes, own, &out)) != HW_OK) return rc;
    const HalfStag h1{lat->stag_ws->t.as<double2>(), stride}, h2{lat->stag_ws->Dp[0].as<double2>(), stride},
        none{nullptr, 0};
    stag_hop_any(gauge, 1, -sign, half_of(chi, 0), none, 0.0, 1.0 / mass, h1, ctx->stream);
    stag_hop_any(gauge, 1, sign, half_of(psi, 0), none, 0.0, 1.0 / mass, h2, ctx->stream);
    dim3 grid((unsigned)((lat->Vh + kStagBlock - 1) / kStagBlock), 2);
    if (sign > 0)
        k_stag_force<1><<<grid, kStagBlock, 0, ctx->stream>>>(lat->g, half_of(chi, 0), half_of(psi, 0), h1, h2,
                                                              lat->V, static_cast<double2 *>(out));
    else
        k_stag_force<-1><<<grid, kStagBlock, 0, ctx->stream>>>(lat->g, half_of(chi, 0), half_of(psi, 0), h1, h2,
                                                               lat->V, static_cast<double2 *>(out));
    HW_CUDA(cudaGetLastError());
    rc = copy_to_host(ctx, force, out, bytes);
    lease.done = rc == HW_OK;
    return rc;
}

// CG<dirac_staggered_evenodd>::apply (conjugate_gradient.h:46-104): M^dag M out = in
// on EVEN, out the initial guess; stops when |r|^2 < accuracy^2 |in|^2 (with
// true_residual set, also on the recomputed |in - M^dag M out|).  FP64.
int hw_staggered_cg_solve(const hw_gauge *gauge, double mass, const hw_stag_field *in, hw_stag_field *out,
                          const hw_cg_params *params, hw_cg_result *result) {
    int rc = check_stag_op(gauge, in, out, mass);
    if (rc != HW_OK) return rc;
    HW_CHECK_ARG(in != out, "in and out must be different fields");
    hw_cg_params P;
    hw_cg_params_default(&P);
    if (params) P = *params;
    HW_CHECK_ARG(P.accuracy > 0 && P.maxiters > 0, "bad accuracy or maxiters");
    HW_CHECK_ARG(P.precision == HW_PREC_F64, "staggered solves run in FP64");
    hw_lattice *lat = gauge->lat;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    if ((rc = ensure_reduction_capacity(ctx, (lat->Vh + kStagBlock - 1) / kStagBlock)) != HW_OK) return rc;
    LoopCgLease lease{lat->stag_ws};
    if ((rc = ensure_stag_ws(lat)) != HW_OK) return rc;
    LoopCgWorkspace &w = *lat->stag_ws;
    const int stride = lat->stride;
    const size_t hb = (size_t)3 * stride * sizeof(double2);
    auto half = [stride](const DevBuf &d) { return HalfStag{d.as<double2>(), stride}; };
    const HalfStag b = half_of(in, 0), xo = half_of(out, 0), x = half(w.x[0]), r = half(w.r[0]), p = half(w.p[0]),
                   Dp = half(w.Dp[0]), t = half(w.t);
    cudaStream_t s = ctx->stream;
    CgState *st = ctx->cg_state.as<CgState>();
    const RedBuf red = ctx->red();
    const double im = 1.0 / mass;
    LoopCgWorkspace::Key key;
    key.links = gauge->U().p;
    key.planes = gauge->U().planes;
    key.red = red.partials;
    key.par = mass;
    if (!w.loop_exec || !(key == w.key)) {
        w.key = LoopCgWorkspace::Key();
        rc = build_loop_graph(s, &w.loop_exec, [&](cudaGraphConditionalHandle cond) {
            stag_cg(gauge, 1, +1, p, StagScale{t, im, st}, red, s);
            stag_cg(gauge, 0, +1, t, StagMul<true>{p, Dp, mass, st}, red, s);
            stag_cg(gauge, 1, -1, Dp, StagScale{t, im, st}, red, s);
            stag_cg(gauge, 0, -1, t, StagUpdate{Dp, r, x, p, mass, st}, red, s);
            k_stag_pupdate<<<(unsigned)((lat->Vh + kStagVecBlock - 1) / kStagVecBlock), kStagVecBlock, 0, s>>>(
                (int)lat->Vh, r, p, st, cond);
        });
        if (rc != HW_OK) return rc;
        w.key = key;
    }
    // Dp = M x ; then the epilogue of M^dag Dp
    auto normal = [&](auto epi) {
        stag_cg(gauge, 1, +1, x, StagScale{t, im, nullptr}, red, s);
        stag_cg(gauge, 0, +1, t, StagMul<false>{x, Dp, mass, st}, red, s);
        stag_cg(gauge, 1, -1, Dp, StagScale{t, im, nullptr}, red, s);
        stag_cg(gauge, 0, -1, t, epi, red, s);
    };
    HW_CUDA(cudaEventRecord(ctx->ev0, s));
    HW_CUDA(cudaMemcpyAsync(x.p, xo.p, hb, cudaMemcpyDeviceToDevice, s));
    // r = b - A x ; p = r
    normal(StagInit{Dp, b, r, p, mass, P.accuracy * P.accuracy, P.maxiters, st});
    HW_CUDA(cudaGetLastError());
    HW_CUDA(cudaGraphLaunch(w.loop_exec, s));
    // explicit residual |b - A x| / |b| in FP64
    normal(StagResidual{Dp, b, mass, st});
    HW_CUDA(cudaMemcpyAsync(xo.p, x.p, hb, cudaMemcpyDeviceToDevice, s));
    HW_CUDA(cudaMemsetAsync(out->half[1].ptr, 0, out->half[1].bytes, s));
    HW_CUDA(cudaGetLastError());
    HW_CUDA(cudaEventRecord(ctx->ev1, s));
    CgState *h = ctx->cg_state_host;
    HW_CUDA(cudaMemcpyAsync(h, st, sizeof(CgState), cudaMemcpyDeviceToHost, s));
    HW_CUDA(cudaStreamSynchronize(s));
    lease.done = true;
    const double bb = h->src_norm2;
    const double true_res = bb > 0 ? std::sqrt(h->res_num2 / bb) : 0.0;
    int status = h->status == CG_BREAKDOWN ? HW_ERR_BREAKDOWN
                 : h->status == CG_MAXITER ? HW_ERR_NOT_CONVERGED
                                           : HW_OK;
    if (status == HW_OK && (!std::isfinite(true_res) || (P.true_residual && true_res > P.accuracy)))
        status = HW_ERR_NOT_CONVERGED;
    if (result) {
        std::memset(result, 0, sizeof(*result));
        float ms = 0.f;
        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
        result->status = status;
        result->iterations = h->iter;
        result->rr_relative = bb > 0 ? h->rr / bb : 0.0;
        result->true_residual = true_res;
        result->seconds = ms * 1e-3;
        result->kernel_launches = 8 + 5 * h->bodies;
    }
    return status;
}

}  // extern "C"
