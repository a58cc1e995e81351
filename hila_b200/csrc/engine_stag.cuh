// Staggered fermions on the solver engine (engine.h lists the phases).  Included by
// engine.cu inside its anonymous namespace, after the finishers: the staggered slots
// share the Wilson slots' tables, states, finishers, per-(slot, tile) reductions and
// chunk graphs, so staggered and Wilson solves run in the same batches and through the
// same server, and a solve is bitwise the same alone and in any batch.
//
// The operator is dirac_staggered_evenodd (staggered.h:193-279) as the reference codes
// it: M_s in = m in_e + D^{eo}_s (1/m) D^{oe}_s in_e with D_s = 0.5 s hop, M^dag = M_{-s}.
// FP64 slots run in FP64 throughout, in k_stag_eng: the low-precision buffers of a slot hold
// FP64 half lattices (3 double2 planes: 48 bytes per site, the size of a Wilson FP16 buffer)
// and work items are (tile, active slot) pairs as in the Wilson FP64 phases.  Slots with FP16
// inner iterations run P1..P5 in k_stag_low and share k_stag_eng's reliable update.  The site algebra comes from
// staggered_math.cuh, which engine.cu includes at file scope.
#pragma once

// An FP16 colour-vector half lattice of a low-precision staggered slot: the three
// colours as (re, im) half pairs in the first uint4 plane of the slot's buffer (the
// fourth word unused) and a per-site scale, the largest |component| of the site.
struct HalfStag16 {
    uint4 *p;
    float *n;
    __device__ __forceinline__ static void unpack(uint4 v, float s, Cx<float> w[3]) {
        const __half2 *h = reinterpret_cast<const __half2 *>(&v);
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const float2 f = __half22float2(h[c]);
            w[c] = {f.x * s, f.y * s};
        }
    }
    __device__ __forceinline__ void ld(int i, Cx<float> w[3]) const { unpack(__ldg(p + i), __ldg(n + i), w); }
    // plain (coherent) load, for arrays the same kernel also writes
    __device__ __forceinline__ void ldp(int i, Cx<float> w[3]) const { unpack(p[i], n[i], w); }
    __device__ __forceinline__ void st(int i, const Cx<float> w[3]) const {
        float m = 0.f;
#pragma unroll
        for (int c = 0; c < 3; c++) m = fmaxf(m, fmaxf(fabsf(w[c].re), fabsf(w[c].im)));
        const float inv = m > 0.f ? 1.0f / m : 0.f;
        n[i] = m;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        __half2 *h = reinterpret_cast<__half2 *>(&v);
#pragma unroll
        for (int c = 0; c < 3; c++) h[c] = __floats2half2_rn(w[c].re * inv, w[c].im * inv);
        p[i] = v;
    }
};

// The FP32 solution increment y of a low-precision staggered slot: colour c of site i at
// y[c * stride + i] (the slot's y buffer viewed as float2 planes).
struct HalfStagY {
    float2 *p;
    int stride;
    __device__ __forceinline__ Cx<float> ld(int c, int i) const {
        const float2 v = p[(size_t)c * stride + i];
        return {v.x, v.y};
    }
    __device__ __forceinline__ void st(int c, int i, Cx<float> v) const {
        p[(size_t)c * stride + i] = make_float2(v.re, v.im);
    }
};

// A thread of the FP16 phases serves two sources at a time, in the two lanes of packed FP32
// instructions (pair.cuh); a block is two teams of kEngTile threads on the same sites, which
// take the pairs of sources in turn and share the staged links.
constexpr int kStagTeams = 2;
constexpr int kStagLowBlock = kStagTeams * kEngTile;

// the values of a pair of sources at one neighbour, as stored
struct StagRaw {
    uint4 a, b;
    float na, nb;
    __device__ __forceinline__ void load(const HalfStag16 &A, const HalfStag16 &B, int j) {
        a = __ldg(A.p + j);
        b = __ldg(B.p + j);
        na = __ldg(A.n + j);
        nb = __ldg(B.n + j);
    }
};

// One term of the hop: acc += f U v (ADJ: f U^dag v), f the site norm of v times sg.  Lane
// arithmetic is independent, so a source's result does not depend on the other; a source
// without a partner fills both lanes.
template <bool ADJ>
__device__ __forceinline__ void stag_term(const Su3<float> &u, const StagRaw &raw, float sg, Cx2 (&acc)[3]) {
    Cx2 w[3];
    float2 nw[3];  // minus the part that the product subtracts
    const __half2 *ha = reinterpret_cast<const __half2 *>(&raw.a);
    const __half2 *hb = reinterpret_cast<const __half2 *>(&raw.b);
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const float2 fa = __half22float2(ha[c]), fb = __half22float2(hb[c]);
        w[c] = {make_float2(fa.x, fb.x), make_float2(fa.y, fb.y)};
        nw[c] = neg2(ADJ ? w[c].re : w[c].im);
    }
    const float2 f = make_float2(sg * raw.na, sg * raw.nb);
#pragma unroll
    for (int a = 0; a < 3; a++) {
        Cx2 t;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const Cx<float> e = ADJ ? u.e[c][a] : u.e[a][c];
            const float2 er = bc2(e.re), ei = bc2(e.im);
            t.re = c == 0 ? mul2(er, w[c].re) : fma2(er, w[c].re, t.re);
            t.im = c == 0 ? mul2(er, w[c].im) : fma2(er, w[c].im, t.im);
            t.re = fma2(ei, ADJ ? w[c].im : nw[c], t.re);
            t.im = fma2(ei, ADJ ? nw[c] : w[c].re, t.im);
        }
        acc[a] = axpy2(acc[a], f, t);
    }
}

// stag_hop_site in FP32 for a pair of sources; the next term's values are asked for before a
// term is computed.  eta: bit d set for eta_d = +1.
__device__ __forceinline__ void stag_hop_pair(const LinksF16x18Smem<kEngTile> &U, const SiteNbrs &n, unsigned eta,
                                              int par, const HalfStag16 &A, const HalfStag16 &B, const StagRaw &first,
                                              Cx2 (&acc)[3]) {
#pragma unroll
    for (int a = 0; a < 3; a++) acc[a] = {bc2(0.f), bc2(0.f)};
    StagRaw fw = first, bw;
#pragma unroll
    for (int d = 0; d < 4; d++) {
        const float e = (eta >> d & 1u) ? 1.f : -1.f;
        Su3<float> u;
        bw.load(A, B, n.bwd[d]);
        U.load(par, d, 0, u);
        stag_term<false>(u, fw, (d == 3 && n.tfwd_wrap) ? -e : e, acc);
        if (d < 3) fw.load(A, B, n.fwd[d + 1]);
        U.load(1 - par, d, 0, u);
        stag_term<true>(u, bw, (d == 3 && n.tbwd_wrap) ? e : -e, acc);
    }
}

// the hop's input of a slot
template <int PHASE>
__device__ __forceinline__ HalfStag16 stag_low_in(const EngProblem &pr) {
    if (PHASE == PH_P1) return HalfStag16{static_cast<uint4 *>(pr.p), pr.pn};
    if (PHASE == PH_P3) return HalfStag16{static_cast<uint4 *>(pr.Dp), pr.Dpn};
    return HalfStag16{static_cast<uint4 *>(pr.t), pr.tn};
}

// Own-site operands of a low-precision staggered slot's epilogue, and the epilogue: P1..P5 in
// FP32 arithmetic on FP16 fields, acc the hop of the slot's input; red[0] receives the
// phase's |.|^2 contribution.  The operands of a pair are asked for before its hop.
template <int PHASE>
struct StagOwn {
    uint4 pv, rv, dv;  // as stored, unpacked by finish()
    float pn, rn, dn;
    Cx<float> y[3];
    __device__ __forceinline__ void load(const EngProblem &pr, int stride, int i) {
        if constexpr (PHASE == PH_P2 || PHASE == PH_P4) {
            pv = __ldg(static_cast<uint4 *>(pr.p) + i);
            pn = __ldg(pr.pn + i);
        }
        if constexpr (PHASE == PH_P4) {
            dv = __ldg(static_cast<uint4 *>(pr.Dp) + i);
            dn = __ldg(pr.Dpn + i);
            rv = static_cast<uint4 *>(pr.r)[i];
            rn = pr.rn[i];
            const HalfStagY Y{reinterpret_cast<float2 *>(pr.y), stride};
#pragma unroll
            for (int c = 0; c < 3; c++) y[c] = Y.ld(c, i);
        }
    }
    __device__ __forceinline__ void finish(const EngProblem &pr, const EngState &st, int stride, int i,
                                           const Cx<float> (&acc)[3], double *red) {
        constexpr int SIGN = (PHASE == PH_P1 || PHASE == PH_P2) ? 1 : -1;
        const float m = (float)pr.kappa;  // the mass
        Cx<float> h[3], p[3], r[3], d[3];
        if constexpr (PHASE == PH_P2 || PHASE == PH_P4) HalfStag16::unpack(pv, pn, p);
        if constexpr (PHASE == PH_P4) {
            HalfStag16::unpack(rv, rn, r);
            HalfStag16::unpack(dv, dn, d);
        }
#pragma unroll
        for (int c = 0; c < 3; c++) h[c] = (0.5f * SIGN) * acc[c];
        if constexpr (PHASE == PH_P1 || PHASE == PH_P3) {  // t = (1/m) D in
            const float im = 1.0f / m;
#pragma unroll
            for (int c = 0; c < 3; c++) h[c] = im * h[c];
            HalfStag16{static_cast<uint4 *>(pr.t), pr.tn}.st(i, h);
        } else if constexpr (PHASE == PH_P2) {  // Dp = m p + D t
#pragma unroll
            for (int c = 0; c < 3; c++) {
                h[c] = m * p[c] + h[c];
                red[0] += (double)norm2(h[c]);
            }
            HalfStag16{static_cast<uint4 *>(pr.Dp), pr.Dpn}.st(i, h);
        } else {  // P4: r -= alpha (m Dp + D t), y += alpha p
            const float alpha = (float)st.alpha;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                r[c] = r[c] - alpha * (m * d[c] + h[c]);
                red[0] += (double)norm2(r[c]);
            }
            HalfStag16{static_cast<uint4 *>(pr.r), pr.rn}.st(i, r);
            const HalfStagY Y{reinterpret_cast<float2 *>(pr.y), stride};
#pragma unroll
            for (int c = 0; c < 3; c++) Y.st(c, i, y[c] + alpha * p[c]);
        }
    }
};

// P1..P4 of the staggered slots with FP16 inner iterations: a block takes items (a tile and a
// part of its slots) from a counter; per item, the sites' eight FP16 links are copied into
// shared memory once, the block's teams take the pairs of slots in turn, and each slot's partial
// sum is formed once per tile in block_sum's order.  Bound by load latency: at 24^4 with 8
// sources P1 takes 54 us (100 MB: 15 us at the HBM's rate), P2 80, P4 98; one source a thread
// with 16 warps per SM took 62, 92 and 132.  P4 holds its pair's own-site operands during the
// hop, in 128 registers (24 warps with 80 registers: 111 us); P2 is slower that way (84 us).
template <int PHASE>
__global__ void __launch_bounds__(kStagLowBlock, PHASE == PH_P4 ? 2 : 3) k_stag_low(EngPtrs P) {
    constexpr int OUTPAR = (PHASE == PH_P1 || PHASE == PH_P3) ? 1 : 0;
    constexpr int NRED = (PHASE == PH_P2 || PHASE == PH_P4) ? 1 : 0;
    __shared__ double smem[kStagLowBlock / 32];
    __shared__ bool last;
    __shared__ int s_item;
    __shared__ int s_act[kEngMaxRhs];
    __shared__ int s_na;
    __shared__ uint4 s_lx[16 * kEngTile];
    __shared__ unsigned s_lz[8 * kEngTile];
    __shared__ double s_red[NRED > 0 ? kEngMaxRhs : 1][kEngTile / 32];
    const EngTables *T = P.T;
    const int max_tiles = T->max_tiles;
    const TileParts TP(T->parts[ITEMS_STAG]);
    const int nitems = TP.items(T->ntiles);
    const int team = threadIdx.x / kEngTile, t = threadIdx.x % kEngTile;
    const LinksF16x18Smem<kEngTile> US{s_lx, s_lz, OUTPAR, t};
    // in fixed order where each block has one item at most (as in k_eng_low)
    auto next_item = [&]() {
        if (nitems <= (int)gridDim.x) return nitems;
        if (threadIdx.x == 0) s_item = atomicAdd(P.sched + kEngPhases + PHASE, 1);
        __syncthreads();
        return s_item;
    };
    for (int item = nitems <= (int)gridDim.x ? (int)blockIdx.x : next_item(); item < nitems; item = next_item()) {
        const int tile = TP.tile(item);
        const int l = find_lattice(T, tile);
        const EngLattice &La = T->lat[l];
        const int lt = tile - La.tile0;
        const int i = lt * kEngTile + t;
        const bool valid = i < La.g.Vh;
        if (threadIdx.x < 32) {
            const int q = threadIdx.x;
            int j = 0;
            bool on = false;
            if (La.fermion == FERM_STAGGERED && q < La.nprob) {
                j = La.prob[q];
                on = active<PHASE, FERM_STAGGERED_LOW>(P.S[j]);
            }
            const unsigned m = __ballot_sync(0xffffffffu, on);
            if (on) s_act[__popc(m & ((1u << q) - 1u))] = j;
            if (q == 0) s_na = __popc(m);
        }
        __syncthreads();
        const int na = s_na;
        // every item of a lattice sees the same active slots: a lattice without any is left
        // alone (no arrival, its ticket untouched)
        int a0, a1;
        if (!TP.range(item, na, 2, a0, a1)) {
            __syncthreads();
            if (NRED > 0 && na > 0)
                arrive_and_finish<PHASE, NRED, FERM_STAGGERED_LOW, kStagLowBlock>(P, La, l, smem, last,
                                                                                 TP.items(La.ntiles));
            continue;
        }
        SiteNbrs nb;
        unsigned eta = 0;
        if (valid) {
            nb = site_neighbours(La.g, i, OUTPAR);
            US.stage<kStagTeams>(LinksF16x18{La.l16x, La.l16z, La.stride}, nb, i, team);
            int c[4];
            site_coords(La.g, i, OUTPAR, c);
#pragma unroll
            for (int d = 0; d < 4; d++) eta |= (stag_eta(c, d) > 0.0 ? 1u : 0u) << d;
        }
        const int stride = La.stride;
        bool staged = false;
        for (int a = a0; a < a1; a += 2 * kStagTeams) {
            const int mine = a + 2 * team;  // this team's pair of slots
            const bool on = valid && mine < a1;
            const bool two = mine + 1 < a1;
            const int jA = s_act[min(mine, a1 - 1)], jB = s_act[min(mine + 1, a1 - 1)];
            const EngProblem &A = T->prob[jA], &B = T->prob[jB];
            const HalfStag16 inA = stag_low_in<PHASE>(A), inB = stag_low_in<PHASE>(B);
            StagRaw first;
            if (on) first.load(inA, inB, nb.fwd[0]);
            if (!staged) {  // each team copied half of the links
                cp_async_wait_all();
                __syncthreads();
                staged = true;
            }
            double redA = 0.0, redB = 0.0;
            if (on) {
                Cx2 acc[3];
                StagOwn<PHASE> oa, ob;
                oa.load(A, stride, i);
                ob.load(B, stride, i);
                stag_hop_pair(US, nb, eta, OUTPAR, inA, inB, first, acc);
                Cx<float> ha[3], hb[3];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    ha[c] = {acc[c].re.x, acc[c].im.x};
                    hb[c] = {acc[c].re.y, acc[c].im.y};
                }
                oa.finish(A, P.S[jA], stride, i, ha, &redA);
                if (two) ob.finish(B, P.S[jB], stride, i, hb, &redB);
            }
            if constexpr (NRED > 0) {
                if (mine < a1) {
                    const double vA = warp_sum(redA), vB = warp_sum(redB);
                    if ((t & 31) == 0) {
                        s_red[mine][t >> 5] = vA;
                        if (two) s_red[mine + 1][t >> 5] = vB;
                    }
                }
            }
        }
        if constexpr (NRED > 0) {
            __syncthreads();
            if (threadIdx.x >= a0 && threadIdx.x < a1) {
                double sum = 0;
#pragma unroll
                for (int w = 0; w < kEngTile / 32; w++) sum += s_red[threadIdx.x][w];
                P.partials[((size_t)s_act[threadIdx.x] * 2) * max_tiles + lt] = sum;
                __threadfence();  // visible before the lattice's ticket is taken
            }
        }
        __syncthreads();  // s_act and the staged links are rewritten by the next item
        if constexpr (NRED > 0)
            arrive_and_finish<PHASE, NRED, FERM_STAGGERED_LOW, kStagLowBlock>(P, La, l, smem, last,
                                                                             TP.items(La.ntiles));
    }
}

// P5 of those slots: p = r + beta p (p = r in a slot's first iteration), the slots of a tile
// four at a time so that their loads are in flight together
constexpr int kStagP5Src = 4;
__global__ void __launch_bounds__(kEngTile) k_stag_low_p5(EngPtrs P) {
    const EngTables *T = P.T;
    for (int tile = blockIdx.x; tile < T->ntiles; tile += gridDim.x) {
        const int l = find_lattice(T, tile);
        const EngLattice &La = T->lat[l];
        if (La.fermion != FERM_STAGGERED) continue;
        const int i = (tile - La.tile0) * kEngTile + threadIdx.x;
        if (i >= La.g.Vh) continue;
        for (int q0 = 0; q0 < La.nprob; q0 += kStagP5Src) {
            Cx<float> r[kStagP5Src][3], p[kStagP5Src][3];
            bool on[kStagP5Src];
#pragma unroll
            for (int k = 0; k < kStagP5Src; k++) {
                on[k] = q0 + k < La.nprob && active<PH_P5, FERM_STAGGERED_LOW>(P.S[La.prob[q0 + k]]);
                if (on[k]) {
                    const EngProblem &pr = T->prob[La.prob[q0 + k]];
                    HalfStag16{static_cast<uint4 *>(pr.r), pr.rn}.ld(i, r[k]);
                    HalfStag16{static_cast<uint4 *>(pr.p), pr.pn}.ldp(i, p[k]);
                }
            }
#pragma unroll
            for (int k = 0; k < kStagP5Src; k++)
                if (on[k]) {
                    const int j = La.prob[q0 + k];
                    const EngProblem &pr = T->prob[j];
                    const EngState &st = P.S[j];
                    const float beta = (float)st.beta;
                    if (!st.init)
#pragma unroll
                        for (int c = 0; c < 3; c++) r[k][c] = r[k][c] + beta * p[k][c];
                    HalfStag16{static_cast<uint4 *>(pr.p), pr.pn}.st(i, r[k]);
                }
        }
    }
}

template <int PHASE>
__global__ void __launch_bounds__(kEngTile, 3) k_stag_eng(EngPtrs P) {
    constexpr int SIGN = (PHASE == PH_P1 || PHASE == PH_P2 || PHASE == PH_R2 || PHASE == PH_R3) ? 1 : -1;
    constexpr int OUTPAR =
        (PHASE == PH_P1 || PHASE == PH_P3 || PHASE == PH_R2 || PHASE == PH_R4 || PHASE == PH_R4L) ? 1 : 0;
    constexpr int NRED = (PHASE == PH_P2 || PHASE == PH_P4 || PHASE == PH_R5L) ? 1
                         : (PHASE == PH_R3 || PHASE == PH_R5)                   ? 2
                                                                                : 0;
    constexpr bool HOP = PHASE != PH_R1 && PHASE != PH_P5;
    __shared__ double smem[kEngTile / 32];
    __shared__ bool last;
    __shared__ ActiveTable act;
    if (eng_ru_phase(PHASE) && *(volatile int *)(P.ctl + 2) == 0) return;  // no reliable update pending
    const EngTables *T = P.T;
    const int nitems = T->ntiles * kEngMaxRhs;
    const int max_tiles = T->max_tiles;
    build_active<PHASE, FERM_STAGGERED>(P, act);
    for (int item = blockIdx.x; item < nitems; item += gridDim.x) {
        const int tile = item / kEngMaxRhs, a = item % kEngMaxRhs;
        const int l = find_lattice(T, tile);
        const EngLattice &La = T->lat[l];
        const int na = act.n[l];
        if (La.fermion != FERM_STAGGERED || a >= na) continue;
        const int j = act.slot[l][a];
        const Geom g = La.g;
        const int stride = La.stride;
        const int lt = tile - La.tile0;
        const int i = lt * kEngTile + threadIdx.x;
        const EngProblem &pr = T->prob[j];
        const EngState &st = P.S[j];
        const double m = pr.kappa;  // the mass of a staggered solve
        const bool low = pr.stag_low != 0;
        const HalfStag x{pr.x, stride}, b{pr.b, stride}, sv{pr.s, stride};
        const HalfStag p{static_cast<double2 *>(pr.p), stride}, r{static_cast<double2 *>(pr.r), stride};
        const HalfStag Dp{static_cast<double2 *>(pr.Dp), stride};
        // the odd FP64 half of the reliable update: t itself, or t64 beside the FP16 t
        const HalfStag t{low ? pr.t64 : static_cast<double2 *>(pr.t), stride};
        double red[2] = {0.0, 0.0};
        if (i < g.Vh) {
            if constexpr (PHASE == PH_R1) {
                // first update: record whether the initial x is nonzero anywhere (read by R2, R3)
                bool nz = false;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const Cx<double> v = x.ld(c, i);
                    nz |= v.re != 0.0 || v.im != 0.0;
                }
                const unsigned am = __activemask();
                if (st.init && __any_sync(am, nz) && (threadIdx.x & 31) == __ffs(am) - 1 &&
                    !*(volatile int *)&P.S[j].xnz)
                    atomicOr(&P.S[j].xnz, 1);
                if (low) {  // x += y, y = 0
                    const HalfStagY y{reinterpret_cast<float2 *>(pr.y), stride};
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const Cx<float> yv = y.ld(c, i);
                        const Cx<double> xv = x.ldp(c, i);
                        x.st(c, i, {xv.re + (double)yv.re, xv.im + (double)yv.im});
                        y.st(c, i, {0.f, 0.f});
                    }
                }
            } else if constexpr (PHASE == PH_P5) {
                const double beta = st.beta;
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const Cx<double> rv = r.ld(c, i);
                    p.st(c, i, st.init ? rv : rv + beta * p.ldp(c, i));
                }
            } else {
                static_assert(HOP, "hop phases");
                const HalfStag in = PHASE == PH_P1 ? p : PHASE == PH_P3 ? Dp : PHASE == PH_R2 ? x
                                                     : (PHASE == PH_R4 || PHASE == PH_R4L) ? sv
                                                                                          : t;
                // R3 of a first update from x = 0: R2 did not run and the hop of zeros is zero
                const bool zero_in = PHASE == PH_R3 && st.init && !st.xnz;
                Cx<double> acc[3] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
                if (!zero_in) {
                    if (La.l64_planes == 9)
                        stag_hop_site(g, LinksF64x18{La.l64, stride}, OUTPAR, i, in, acc);
                    else
                        stag_hop_site(g, LinksF64x12{La.l64, stride}, OUTPAR, i, in, acc);
                }
                Cx<double> h[3];
#pragma unroll
                for (int c = 0; c < 3; c++) h[c] = (0.5 * SIGN) * acc[c];
                if constexpr (OUTPAR == 1) {  // P1, P3, R2, R4, R4L: t = (1/m) D in
                    const double im = 1.0 / m;
#pragma unroll
                    for (int c = 0; c < 3; c++) t.st(c, i, im * h[c]);
                } else if constexpr (PHASE == PH_P2) {  // Dp = m p + D t
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const Cx<double> v = m * p.ld(c, i) + h[c];
                        Dp.st(c, i, v);
                        red[0] += norm2(v);
                    }
                } else if constexpr (PHASE == PH_P4) {  // r -= alpha (m Dp + D t), x += alpha p
                    const double alpha = st.alpha;
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const Cx<double> ddp = m * Dp.ld(c, i) + h[c];
                        const Cx<double> rv = r.ldp(c, i) - alpha * ddp;
                        r.st(c, i, rv);
                        x.st(c, i, x.ldp(c, i) + alpha * p.ld(c, i));
                        red[0] += norm2(rv);
                    }
                } else if constexpr (PHASE == PH_R3) {  // s = b - M x (solve) or s = M x (normal)
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        const Cx<double> mx = m * x.ld(c, i) + h[c];
                        if (pr.mode == ENG_MODE_SOLVE) {
                            const Cx<double> bv = b.ld(c, i);
                            const Cx<double> v = bv - mx;
                            sv.st(c, i, v);
                            red[0] += norm2(v);
                            red[1] += norm2(bv);
                        } else {
                            sv.st(c, i, mx);
                        }
                    }
                } else if constexpr (PHASE == PH_R5L || PHASE == PH_R5) {
                    // R5L: r = M^dag s; R5: r = b - M^dag M x (normal system); FP16 r for a
                    // low-precision slot
                    Cx<float> rl[3];
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        Cx<double> v = m * sv.ld(c, i) + h[c];
                        if (PHASE == PH_R5) {
                            const Cx<double> bv = b.ld(c, i);
                            v = bv - v;
                            red[1] += norm2(bv);
                        }
                        red[0] += norm2(v);
                        if (low)
                            rl[c] = {(float)v.re, (float)v.im};
                        else
                            r.st(c, i, v);
                    }
                    if (low) HalfStag16{static_cast<uint4 *>(pr.r), pr.rn}.st(i, rl);
                }
            }
        }
        if constexpr (NRED > 0) {
            // the item's sums with one barrier: warp sums in shared memory, added by thread 0
            // in warp order (block_sum's order, the same bits)
            __shared__ double s_w[NRED][kEngTile / 32];
#pragma unroll
            for (int k = 0; k < NRED; k++) {
                const double v = warp_sum(red[k]);
                if ((threadIdx.x & 31) == 0) s_w[k][threadIdx.x >> 5] = v;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
#pragma unroll
                for (int k = 0; k < NRED; k++) {
                    double sum = 0;
#pragma unroll
                    for (int w = 0; w < kEngTile / 32; w++) sum += s_w[k][w];
                    P.partials[((size_t)j * 2 + k) * max_tiles + lt] = sum;
                }
            }
            arrive_and_finish<PHASE, NRED, FERM_STAGGERED>(P, La, l, smem, last, La.ntiles * na);
        }
    }
}

// one iteration of the staggered slots: the phases of the slot kinds present (FP64 and FP16
// slots of a phase are disjoint; each kernel finishes its own); the reliable-update phases,
// which serve both kinds, return at once unless some slot asked for one
void enqueue_stag_iteration(const EngPtrs &P, const EngGrid &G, cudaStream_t s, int parts) {
    const bool f64 = G.kinds & 2, low = G.kinds & 4;
    if (parts & ENG_PART_INNER) {
        if (f64) k_stag_eng<PH_P1><<<G.f64, kEngTile, 0, s>>>(P);
        if (low) k_stag_low<PH_P1><<<G.stag, kStagLowBlock, 0, s>>>(P);
        if (f64) k_stag_eng<PH_P2><<<G.f64, kEngTile, 0, s>>>(P);
        if (low) k_stag_low<PH_P2><<<G.stag, kStagLowBlock, 0, s>>>(P);
        if (f64) k_stag_eng<PH_P3><<<G.f64, kEngTile, 0, s>>>(P);
        if (low) k_stag_low<PH_P3><<<G.stag, kStagLowBlock, 0, s>>>(P);
        if (f64) k_stag_eng<PH_P4><<<G.f64, kEngTile, 0, s>>>(P);
        if (low) k_stag_low<PH_P4><<<G.stag, kStagLowBlock, 0, s>>>(P);
    }
    if (parts & ENG_PART_RU) {
        k_stag_eng<PH_R1><<<G.f64, kEngTile, 0, s>>>(P);
        k_stag_eng<PH_R2><<<G.f64, kEngTile, 0, s>>>(P);
        k_stag_eng<PH_R3><<<G.f64, kEngTile, 0, s>>>(P);
        k_stag_eng<PH_R4><<<G.f64, kEngTile, 0, s>>>(P);
        k_stag_eng<PH_R4L><<<G.f64, kEngTile, 0, s>>>(P);
        k_stag_eng<PH_R5><<<G.f64, kEngTile, 0, s>>>(P);
        k_stag_eng<PH_R5L><<<G.f64, kEngTile, 0, s>>>(P);
    }
    if (parts & ENG_PART_P5) {
        if (f64) k_stag_eng<PH_P5><<<G.f64, kEngTile, 0, s>>>(P);
        if (low) k_stag_low_p5<<<4 * G.stag, kEngTile, 0, s>>>(P);
    }
}
