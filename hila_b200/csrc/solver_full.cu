// CG<Dirac_Wilson>::apply (libraries/dirac/conjugate_gradient.h:46-104 on the
// unpreconditioned operator of wilson.h:146-201): M^dag M out = in on ALL sites, FP64.
//
// An iteration is three kernels resident on the device (the body of a
// CUDA-graph WHILE node, as solver_f64.cpp): K1 Dp = D p with |Dp|^2 -> alpha, K2 r -= alpha
// D^dag Dp, x += alpha p with |r|^2 -> beta and the stopping decision, both over the two
// parities in one launch, and p = r + beta p.  (A host loop over the operator, dot products
// and axpys, with two host synchronisations per iteration and its workspace allocated per
// call, took 107 us per iteration at 16^4.)  Partial sums are added in block order: the
// result does not depend on scheduling.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "cg_loop.cuh"
#include "hw_internal.h"
#include "reduce.cuh"
#include "storage.cuh"

namespace hw {
namespace {

constexpr int kFullBlock = 128;

struct Full {  // the two halves of a Wilson field
    double2 *h[2];
};

__device__ __forceinline__ Cx<double> ldf(const Full &f, int par, int stride, int c, int i) {
    const double2 v = f.h[par][(size_t)c * stride + i];
    return {v.x, v.y};
}
__device__ __forceinline__ void stf(const Full &f, int par, int stride, int c, int i, Cx<double> v) {
    f.h[par][(size_t)c * stride + i] = make_double2(v.re, v.im);
}

// out = in - k H in; ALPHA: |out|^2 -> alpha
template <bool ALPHA>
struct FullMul {
    static constexpr int NRED = ALPHA ? 1 : 0;
    Full in, out;
    double k;
    CgState *st;
    __device__ bool skip() const { return ALPHA && st->status != CG_RUNNING; }
    __device__ void operator()(int par, int stride, int i, const Spinor<double> &acc, double *red) const {
        double n2 = 0;
#pragma unroll
        for (int c = 0; c < 12; c++) {
            const Cx<double> v = ldf(in, par, stride, c, i) - k * acc.s[c / 3][c % 3];
            stf(out, par, stride, c, i, v);
            n2 += norm2(v);
        }
        red[0] = n2;
    }
    __device__ void operator()(const double *tot) {
        cg_alpha(st, tot[0]);
    }
};

// r = p = b - (Dp - k H Dp); |r|^2, |b|^2 -> the start of the iteration
struct FullInit {
    static constexpr int NRED = 2;
    Full Dp, b, r, p;
    double k, acc2;
    int maxiter;
    CgState *st;
    __device__ bool skip() const { return false; }
    __device__ void operator()(int par, int stride, int i, const Spinor<double> &acc, double *red) const {
#pragma unroll
        for (int c = 0; c < 12; c++) {
            const Cx<double> bv = ldf(b, par, stride, c, i);
            const Cx<double> v = bv - (ldf(Dp, par, stride, c, i) - k * acc.s[c / 3][c % 3]);
            stf(r, par, stride, c, i, v);
            stf(p, par, stride, c, i, v);
            red[0] += norm2(v);
            red[1] += norm2(bv);
        }
    }
    __device__ void operator()(const double *tot) {
        cg_start(st, tot[0], tot[1], acc2, maxiter);
    }
};

// r -= alpha (Dp - k H Dp), x += alpha p; |r|^2 -> beta, status
struct FullUpdate {
    static constexpr int NRED = 1;
    Full Dp, r, x, p;
    double k;
    CgState *st;
    __device__ bool skip() const { return st->status != CG_RUNNING; }
    __device__ void operator()(int par, int stride, int i, const Spinor<double> &acc, double *red) const {
        const double alpha = st->alpha;
        double n2 = 0;
#pragma unroll
        for (int c = 0; c < 12; c++) {
            const Cx<double> ddp = ldf(Dp, par, stride, c, i) - k * acc.s[c / 3][c % 3];
            const Cx<double> rv = ldf(r, par, stride, c, i) - alpha * ddp;
            stf(r, par, stride, c, i, rv);
            stf(x, par, stride, c, i, ldf(x, par, stride, c, i) + alpha * ldf(p, par, stride, c, i));
            n2 += norm2(rv);
        }
        red[0] = n2;
    }
    __device__ void operator()(const double *tot) {
        cg_step(st, tot[0]);
    }
};

// |b - (Dp - k H Dp)|^2
struct FullResidual {
    static constexpr int NRED = 1;
    Full Dp, b;
    double k;
    CgState *st;
    __device__ bool skip() const { return false; }
    __device__ void operator()(int par, int stride, int i, const Spinor<double> &acc, double *red) const {
#pragma unroll
        for (int c = 0; c < 12; c++)
            red[0] += norm2(ldf(b, par, stride, c, i) - (ldf(Dp, par, stride, c, i) - k * acc.s[c / 3][c % 3]));
    }
    __device__ void operator()(const double *tot) { st->res_num2 = tot[0]; }
};

// the hop over both parities: blocks [0, n) EVEN output sites, [n, 2n) ODD ones.  At most 128
// registers, for four blocks per SM: us per iteration (18-real links) without the bound -> with
// it, 12^4 36 -> 36, 16^4 91 -> 64 (one wave of blocks), 20^4 203 -> 207, 24^4 405 -> 374, 32^4
// 1233 -> 1087; 12 reals alike (32^4 991 -> 888).
template <int SIGN, class Lk, class Epi>
__global__ void __launch_bounds__(kFullBlock, 4) k_full_hop(Geom g, Lk U, Full in, Epi epi, RedBuf red) {
    if (epi.skip()) return;
    const int nb = gridDim.x / 2;
    const int par = (int)blockIdx.x >= nb ? 1 : 0;
    const int i = ((int)blockIdx.x - par * nb) * kFullBlock + threadIdx.x;
    constexpr int NR = Epi::NRED > 0 ? Epi::NRED : 1;
    double v[NR];
#pragma unroll
    for (int k = 0; k < NR; k++) v[k] = 0.0;
    if (i < g.Vh) {
        Spinor<double> acc;
        hop_site<SIGN>(g, par, i, SpinorF64{in.h[1 - par], U.stride}, U, acc);
        epi(par, U.stride, i, acc, v);
    }
    if constexpr (Epi::NRED > 0) grid_reduce<Epi::NRED, kFullBlock>(v, red.partials, red.ticket, epi);
}

// p = r + beta p over both halves
__global__ void __launch_bounds__(256) k_full_pupdate(long n, Full r, Full p, CgState *st,
                                                     cudaGraphConditionalHandle cond) {
    if (blockIdx.x == 0 && threadIdx.x == 0) loop_next(st, cond, 1);
    if (!st->do_pupdate) return;
    const double beta = st->beta;
    const long k = blockIdx.x * 256L + threadIdx.x;
    if (k >= n) return;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const double2 rv = r.h[h][k], pv = p.h[h][k];
        p.h[h][k] = make_double2(fma(beta, pv.x, rv.x), fma(beta, pv.y, rv.y));
    }
}

template <class Epi>
void full_hop(const hw_gauge *G, int sign, Full in, const Epi &epi, RedBuf red, cudaStream_t s) {
    const Geom &g = G->lat->g;
    const GaugeF64 U = G->U();
    const long nb = 2L * ((g.Vh + kFullBlock - 1) / kFullBlock);
    const dim3 grid = Epi::NRED > 0 ? red.grid(Epi::NRED, nb) : dim3((unsigned)nb);
    const LinksF64x18 U18{U.p, U.stride};
    const LinksF64x12 U12{U.p, U.stride};
    if (U.planes == 9) {
        if (sign > 0)
            k_full_hop<1><<<grid, kFullBlock, 0, s>>>(g, U18, in, epi, red);
        else
            k_full_hop<-1><<<grid, kFullBlock, 0, s>>>(g, U18, in, epi, red);
    } else {
        if (sign > 0)
            k_full_hop<1><<<grid, kFullBlock, 0, s>>>(g, U12, in, epi, red);
        else
            k_full_hop<-1><<<grid, kFullBlock, 0, s>>>(g, U12, in, epi, red);
    }
}

Full full_of(const DevBuf (&b)[2]) { return Full{{b[0].as<double2>(), b[1].as<double2>()}}; }

Full full_of(const hw_field *f) { return Full{{f->half[0].buf.as<double2>(), f->half[1].buf.as<double2>()}}; }

}  // namespace
}  // namespace hw

using namespace hw;

extern "C" int hw_wilson_cg_solve(const hw_gauge *gauge, double kappa, const hw_field *in, hw_field *out,
                                  const hw_cg_params *params, hw_cg_result *result) {
    HW_CHECK_ARG(gauge && in && out, "null argument");
    HW_CHECK_ARG(in->lat == gauge->lat && out->lat == gauge->lat, "fields and gauge belong to different lattices");
    HW_CHECK_ARG(in != out, "in and out must be different fields");
    hw_cg_params P;
    hw_cg_params_default(&P);
    if (params) P = *params;
    HW_CHECK_ARG(P.accuracy > 0 && P.maxiters > 0, "bad accuracy or maxiters");
    HW_CHECK_ARG(P.precision == HW_PREC_F64, "the unpreconditioned solve runs in FP64");
    hw_lattice *lat = gauge->lat;
    hw_context *ctx = lat->ctx;
    std::lock_guard<std::recursive_mutex> lk(ctx->mu);
    HW_CUDA(cudaSetDevice(ctx->device));
    int rc;
    if ((rc = ensure_reduction_capacity(ctx, 2 * ((lat->Vh + kFullBlock - 1) / kFullBlock))) != HW_OK) return rc;
    if (!lat->full_ws) lat->full_ws.reset(new LoopCgWorkspace(ctx->loop_ws_bytes));
    LoopCgLease lease{lat->full_ws};
    LoopCgWorkspace &w = *lat->full_ws;
    const size_t hb = (size_t)12 * lat->stride * sizeof(double2);
    cudaStream_t s = ctx->stream;
    for (int h = 0; h < 2; h++)
        for (DevBuf *d : {&w.r[h], &w.p[h], &w.Dp[h], &w.x[h]})
            if (!d->ptr) {
                if ((rc = d->alloc(hb)) != HW_OK) return rc;
                HW_CUDA(cudaMemsetAsync(d->ptr, 0, hb, s));  // the padding sites of p are read by its update
            }
    const Full b = full_of(in), xo = full_of(out), x = full_of(w.x), r = full_of(w.r), p = full_of(w.p),
               Dp = full_of(w.Dp);
    CgState *st = ctx->cg_state.as<CgState>();
    const RedBuf red = ctx->red();
    const long n = (long)12 * lat->stride;
    LoopCgWorkspace::Key key;
    key.links = gauge->U().p;
    key.planes = gauge->U().planes;
    key.red = red.partials;
    key.par = kappa;
    if (!w.loop_exec || !(key == w.key)) {
        w.key = LoopCgWorkspace::Key();
        rc = build_loop_graph(s, &w.loop_exec, [&](cudaGraphConditionalHandle cond) {
            full_hop(gauge, 1, p, FullMul<true>{p, Dp, kappa, st}, red, s);
            full_hop(gauge, -1, Dp, FullUpdate{Dp, r, x, p, kappa, st}, red, s);
            k_full_pupdate<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, r, p, st, cond);
        });
        if (rc != HW_OK) return rc;
        w.key = key;
    }
    HW_CUDA(cudaEventRecord(ctx->ev0, s));
    for (int h = 0; h < 2; h++) HW_CUDA(cudaMemcpyAsync(x.h[h], xo.h[h], hb, cudaMemcpyDeviceToDevice, s));
    // r = b - A x ; p = r   (conjugate_gradient.h:57-63)
    full_hop(gauge, 1, x, FullMul<false>{x, Dp, kappa, st}, red, s);
    full_hop(gauge, -1, Dp, FullInit{Dp, b, r, p, kappa, P.accuracy * P.accuracy, P.maxiters, st}, red, s);
    HW_CUDA(cudaGetLastError());
    HW_CUDA(cudaGraphLaunch(w.loop_exec, s));
    // explicit residual |b - A x| in FP64
    full_hop(gauge, 1, x, FullMul<false>{x, Dp, kappa, st}, red, s);
    full_hop(gauge, -1, Dp, FullResidual{Dp, b, kappa, st}, red, s);
    for (int h = 0; h < 2; h++) HW_CUDA(cudaMemcpyAsync(xo.h[h], x.h[h], hb, cudaMemcpyDeviceToDevice, s));
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
        result->kernel_launches = 4 + 3 * h->bodies;
    }
    return status;
}
