// Internal host-side objects behind the opaque C-ABI handles.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "errors.h"
#include "graph_build.h"
#include "host_copy.h"
#include "kernels.h"

namespace hw {

class Engine;

// RAII device buffer
struct DevBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
    DevBuf() = default;
    DevBuf(const DevBuf &) = delete;
    DevBuf &operator=(const DevBuf &) = delete;
    ~DevBuf() { release(); }
    int alloc(size_t n);
    void release();
    template <typename T>
    T *as() const {
        return static_cast<T *>(ptr);
    }
};

// Sites per parity rounded up to 64 so every SoA plane starts 1 KiB aligned
// (for FP64 planes) and coalesced rows never straddle planes.
inline int padded_stride(long vh) { return (int)((vh + 63) / 64 * 64); }

}  // namespace hw

// ------------------------------------------------------------------ handles

struct hw_context {
    int device = 0;
    cudaStream_t stream = nullptr;
    std::recursive_mutex mu;
    hw::DevBuf red_partials;  // grid-reduction partial sums
    hw::DevBuf red_ticket;    // grid-reduction arrival counters
    hw::DevBuf cg_state;      // hw::CgState
    hw::DevBuf stage;         // lexicographic staging buffer for host transfers (grow-only)
    hw::CgState *cg_state_host = nullptr;  // pinned mirror
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    hw::HostCopier copier;  // copies into pageable memory
    std::shared_ptr<std::atomic<size_t>> loop_ws_bytes = std::make_shared<std::atomic<size_t>>(0);
    hw::RedBuf red() const {
        return hw::RedBuf{red_partials.as<double>(), red_ticket.as<unsigned>(), red_capacity_doubles};
    }
    size_t red_capacity_doubles = 0;
    hw::Engine *engines[3] = {nullptr, nullptr, nullptr};  // batched mixed-precision engines by precision
    bool engine_profile = false;  // per-phase event timing of the engines (hw_engine_profile_enable)
};

// FP64 half-lattice field buffer
struct HalfBuf {
    hw::DevBuf buf;
    int stride = 0;
    hw::HalfF64 h() const { return hw::HalfF64{buf.as<double2>(), stride}; }
};

struct hw_lattice;

// Per-lattice FP64 solver workspace (the reference allocates r, p, Dp, DDp per
// CG call, conjugate_gradient.h:49; here they live as long as the lattice).
struct CgWorkspace {
    HalfBuf r, p, Dp, DDp, src, res;  // EVEN
    HalfBuf t;                        // ODD
    // cached graphs of the last solve
    cudaGraphExec_t init_exec = nullptr, loop_exec = nullptr;
    struct Key {
        const void *links = nullptr, *in = nullptr, *out = nullptr, *red = nullptr;  // pointers in the graphs
        double kappa = 0, acc2 = 0, diag = 1;
        int maxiter = 0, mode = 0, planes = 0;
        bool operator==(const Key &o) const {
            return links == o.links && planes == o.planes && red == o.red && in == o.in && out == o.out &&
                   kappa == o.kappa && acc2 == o.acc2 && diag == o.diag && maxiter == o.maxiter && mode == o.mode;
        }
    } key;
    bool allocated = false;
    ~CgWorkspace();
};

// Workspace of a CG over device fields that keeps its loop graph (solver_full.cu,
// staggered.cu): the iterated fields and the solution are the workspace's own, so the graph
// serves every source and solution on the lattice.  After a call it stays with its lattice while
// the context's lattices keep no more than kLoopWsKeep bytes together (a Wilson 32^4 has 0.8 GB),
// else it is freed.
constexpr size_t kLoopWsKeep = size_t(1) << 30;
struct LoopCgWorkspace {
    std::shared_ptr<std::atomic<size_t>> total;  // bytes kept by the context's workspaces
    size_t kept = 0;                             // of them, this one's
    hw::DevBuf r[2], p[2], Dp[2], x[2], t;  // [0] EVEN, [1] ODD (unpreconditioned solve only)
    cudaGraphExec_t loop_exec = nullptr;
    struct Key {
        const void *links = nullptr, *red = nullptr;
        int planes = 0;
        double par = 0;  // kappa or mass
        bool operator==(const Key &o) const {
            return links == o.links && red == o.red && planes == o.planes && par == o.par;
        }
    } key;
    explicit LoopCgWorkspace(std::shared_ptr<std::atomic<size_t>> t) : total(std::move(t)) {}
    ~LoopCgWorkspace();
};

// Frees a workspace at the end of the call that used it unless it may stay; after an error it is
// freed in any case, as it may be half made.
struct LoopCgLease {
    std::unique_ptr<LoopCgWorkspace> &ws;
    bool done = false;  // set when the call has come to its end
    ~LoopCgLease();
};

struct hw_field;

struct hw_lattice {
    hw_context *ctx = nullptr;
    int dims[4] = {0, 0, 0, 0};
    int tap = 1;
    long V = 0, Vh = 0;
    int stride = 0;
    hw::Geom g{};
    std::unique_ptr<CgWorkspace> ws;
    std::unique_ptr<LoopCgWorkspace> full_ws, stag_ws;  // unpreconditioned and staggered CG
    hw_field *host_b = nullptr, *host_x = nullptr;  // fields behind the host-array solve
    bool tuned = false;  // FP64 hop launch shape chosen (g.hop_variant)
    ~hw_lattice();
};

struct hw_gauge {
    hw_lattice *lat = nullptr;
    int link_format = 18;
    hw::DevBuf f64;  // FP64 planes
    hw::GaugeF64 U() const { return hw::GaugeF64{f64.as<double2>(), lat->stride, link_format == 12 ? 6 : 9}; }
    // low-precision copies for mixed-precision solves (built on first use)
    mutable hw::DevBuf f32, f16a, f16b, f32a, f32b, f16x, f16z;
};

struct hw_field {
    hw_lattice *lat = nullptr;
    HalfBuf half[2];  // [0] EVEN, [1] ODD
};

// staggered colour-vector field (staggered.cu)
struct hw_stag_field {
    hw_lattice *lat = nullptr;
    hw::DevBuf half[2];  // [0] EVEN, [1] ODD: 3 double2 planes each
};

namespace hw {
int ensure_workspace(hw_lattice *lat);
int ensure_reduction_capacity(hw_context *ctx, long nblocks);
int ensure_stage(hw_context *ctx, size_t bytes);
// pick the fastest FP64 hop launch shape for this lattice once (HW_HOP_VARIANT overrides)
int tune_hop(hw_lattice *lat, const hw_gauge *G);
// (M_s + m_h) on EVEN half fields (d = 1 + m_h), stream-ordered through the lattice's
// ODD workspace field; context lock held, workspace and hop shape ready
void eo_apply_half(const hw_gauge *G, double kappa, HalfF64 in, HalfF64 out, int sign, double d);
// device memory for a force on its way to the host: the context's staging buffer up to
// kForceStage bytes, else `own`
constexpr size_t kForceStage = 512u << 20;
inline int force_buffer(hw_context *ctx, size_t bytes, DevBuf &own, void **out) {
    const int rc = bytes <= kForceStage ? ensure_stage(ctx, bytes) : own.alloc(bytes);
    *out = bytes <= kForceStage ? ctx->stage.ptr : own.ptr;
    return rc;
}
// device -> host after the work on the context's stream; returns when dst is complete.  The
// caller holds the context's lock.
inline int copy_to_host(hw_context *ctx, void *dst, const void *src, size_t bytes) {
    return ctx->copier.copy(ctx->device, ctx->stream, dst, src, bytes);
}
void destroy_engines(hw_context *ctx);
}  // namespace hw
