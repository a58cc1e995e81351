// Host-side launch interface of the CUDA kernels (no CUDA types beyond
// streams and graph handles).  Implemented in dslash_f64.cu and layout.cu.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "hop_shapes.h"
#include "wilson_math.cuh"

namespace hw {

// Launch of a kernel of a chain on one stream.  With `chain` it may become resident while the
// kernel before it drains (programmatic dependent launch); it begins with chain_begin(), which
// waits for that kernel to complete before anything is read or written.  Between the two hops
// of an operator call this hides the launch and the drain: one even-odd apply took 12.4 -> 8.5
// us at 8^4, 18.6 -> 15.5 us at 16^4 and 103 -> 98 us at 24^4 (18 reals).  Not in the body of a
// CUDA-graph loop, where the early residents of the next kernel crowd the SMs that drain
// first: an FP64 CG iteration took 52 -> 63 us at 16^4 and was no faster at 32^4.
template <class... KArgs, class... Args>
inline void launch_chain(bool chain, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                         const Args &...args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = chain ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

#ifdef __CUDACC__
// First statement of every kernel launched by launch_chain: waits for the kernels before it
// on the stream, then lets the next one become resident (its own wait holds it back).
__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// A pointer that loads through the read-only path (which the compiler may move over the
// wait) start from: its value is known only after chain_begin().
template <class T>
__device__ __forceinline__ T *chained(T *p) {
    asm volatile("" : "+l"(p)::"memory");
    return p;
}
#endif

// Device-resident scalars of one FP64 conjugate-gradient solve
// (conjugate_gradient.h:55-57 keeps the same quantities on the host).
struct CgState {
    double rr;         // |r|^2 of the current residual
    double pAp;        // |M p|^2
    double alpha, beta;
    double target_rr;  // stop when |r|^2 < target_rr
    double src_norm2;  // |in|^2 over EVEN
    double res_num2;   // last explicit residual check: |b - A x|^2
    double res_den2;   //                                |b|^2
    int iter, maxiter;
    int status;        // CG_RUNNING / CG_CONVERGED / CG_MAXITER / CG_BREAKDOWN
    int do_pupdate;    // whether the iteration's last kernel forms p (its CG update ran)
    int bodies;        // loop bodies run
};
enum : int { CG_RUNNING = 0, CG_CONVERGED = 1, CG_MAXITER = 2, CG_BREAKDOWN = 3 };

#ifdef __CUDACC__
// Keeps a graph's while loop going while the solve runs: called by one thread of an iteration's
// last kernel (the kernel always runs, so the loop ends even when the others returned early;
// the iteration counter is bounded by maxiter, so the loop is bounded).
__device__ __forceinline__ void loop_next(CgState *st, cudaGraphConditionalHandle cond, int use_cond) {
    st->bodies += 1;
    if (use_cond) cudaGraphSetConditional(cond, st->status == CG_RUNNING ? 1u : 0u);
}
#endif

// Work buffers for one grid reduction: partial sums and the arrival ticket.
struct RedBuf {
    double *partials;
    unsigned *ticket;  // one counter, zero between uses
    size_t capacity;   // doubles that partials holds
    // the grid of a reducing launch: the one asked for if its partial sums fit, else an empty
    // one, which the launch refuses (cudaErrorInvalidConfiguration)
    dim3 grid(int nred, long nblocks) const {
        return dim3((size_t)nred * nblocks <= capacity ? (unsigned)nblocks : 0u);
    }
};

// FP64 spinor half-lattice: 12 double2 planes
struct HalfF64 {
    double2 *p;
    int stride;
};

// link_planes: 9 (18 reals) or 6 (12 reals, third row rebuilt)
struct GaugeF64 {
    const double2 *p;
    int stride;
    int planes;
};

// ---- FP64 hopping-term launches. `out` has parity par, `in` the opposite.
// out = a * H_s in
void launch_hop_scale(const Geom &g, const GaugeF64 &U, int par, int sign, HalfF64 in, HalfF64 out, double a,
                      const CgState *st, cudaStream_t s);
// The x-type term of the epilogues below carries a factor d (1 + m_h for the
// Hasenbusch operator M + m_h, Hasenbusch.h:16-52; 1 for M itself).
// out = d x + b * H_s in; with red != null also |out|^2 -> st->pAp and alpha = rr/pAp.
// zero (optional): a half-lattice field on out's sites (the other parity of out) that
// the same launch clears, site i by the thread of output site i.
void launch_hop_xpay(const Geom &g, const GaugeF64 &U, int par, int sign, HalfF64 in, HalfF64 x, HalfF64 out,
                     double b, CgState *st, const RedBuf *red, cudaStream_t s, double d = 1.0,
                     double2 *zero = nullptr);
// CG update fused into the last hop of M^dagger M p:
//   DDp = d Dp + b * H_s t;  r -= alpha DDp;  x += alpha p;  |r|^2 -> st (beta, status)
void launch_hop_cg_update(const Geom &g, const GaugeF64 &U, int par, int sign, HalfF64 t, HalfF64 Dp,
                          HalfF64 r, HalfF64 x, HalfF64 p, double b, CgState *st, const RedBuf &red,
                          cudaStream_t s, double d = 1.0);
// explicit residual: res = src - (d x + b * H_s t); |res|^2 -> st->res_num2, |src|^2 -> st->res_den2
void launch_hop_residual(const Geom &g, const GaugeF64 &U, int par, int sign, HalfF64 t, HalfF64 x,
                         HalfF64 src, HalfF64 res, double b, CgState *st, const RedBuf &red, cudaStream_t s,
                         double d = 1.0);

// ---- FP64 vector kernels over one half lattice
// CG start: r = src - Ax (Ax may be null: x = 0), p = r; sets rr, src_norm2, target_rr, status
void launch_cg_init(int Vh, HalfF64 src, HalfF64 Ax, HalfF64 r, HalfF64 p, double acc2, int maxiter,
                    CgState *st, const RedBuf &red, cudaStream_t s);
// end of a loop-body iteration: p = r + beta p (beta from st) and, with use_cond, the graph's
// while loop goes on while st->status == CG_RUNNING
void launch_cg_pupdate(int Vh, HalfF64 r, HalfF64 p, CgState *st, cudaGraphConditionalHandle cond, int use_cond,
                       cudaStream_t s);
// y = a * x
void launch_scale(int Vh, HalfF64 x, HalfF64 y, double a, cudaStream_t s);

// ---- layout conversion (host canonical lexicographic AoS <-> device even-odd SoA)
void launch_spinor_lex_to_eo(const Geom &g, const double *lex, int par, HalfF64 out, cudaStream_t s);
void launch_spinor_eo_to_lex(const Geom &g, HalfF64 in, int par, double *lex, cudaStream_t s);
// checkerboard-ordered AoS [n][12] complex <-> the SoA planes of one half lattice
void launch_aos_to_soa(int n, const double *aos, HalfF64 out, cudaStream_t s);
void launch_soa_to_aos(int n, HalfF64 in, double *aos, cudaStream_t s);
// one direction of links [V][3][3] complex (lexicographic) -> the planes of (par, dir)
void launch_links_lex_to_eo(const Geom &g, const double *lex_dir, double2 *dst, int nplanes, int stride, int par,
                            cudaStream_t s);

}  // namespace hw
