"""Workloads of the Wilson and staggered solve path, as a lattice program calls it.

Every case is one call (or the short chain of calls a program makes together) on the
public Python entry points of ``hila_b200``.  Inputs are SU(3) links near the identity
(the ``exp(i eps H)`` ensemble of the generator, built here with torch) and Gaussian
sources.  Results live in device fields; a program reads them into page-locked host
memory with ``download_eo``, and so does ``run``, unless the call itself already
delivers host arrays or torch tensors.

Sizes run from 4^4 to 32^3 x 64 with every extent even, cubic or not, as the lattices
of the tests, of ``bench.py`` and of the serving workload do.
"""
import math

import numpy as np
import torch

import hila_b200 as hb

# ------------------------------------------------------------------ cases


def listed():
    return [
        # The operator on memory another framework owns, the smallest call there is: one
        # application on a test-size lattice, bound by launches and latency.
        dict(name="op_noalloc_8", kind="noalloc", x=8, y=8, z=8, t=8, fmt=18, sign=1, reps=1),
        # Repeated M^dag M on one field (power iteration for the largest eigenvalue, the
        # operator benchmark): the FP64 hop at the usual 32^4, then the vector is read back.
        dict(name="op_chain_32", kind="chain", x=32, y=32, z=32, t=32, fmt=18, reps=20),
        # Plain FP64 CG on the smallest lattice used in earnest (tests, tuning runs).
        dict(name="cg_f64_8", kind="solve", x=8, y=8, z=8, t=8, fmt=18, prec="f64", nrhs=1),
        # Plain FP64 CG at 32^4: one propagator component, the reference's own use.
        dict(name="cg_f64_32", kind="solve", x=32, y=32, z=32, t=32, fmt=12, prec="f64", nrhs=1),
        # A whole point-source propagator: 12 sources on one gauge field in FP16 mixed
        # precision, the batched solve that the framework is used for most.
        dict(name="batch12_f16_32", kind="solve", x=32, y=32, z=32, t=32, fmt=12, prec="f16", nrhs=12),
        # The solve server with gauge fields of several sizes, requests of 1 to 12 sources
        # from page-locked host arrays, all in flight together.
        dict(name="serve_uneven", kind="serve", x=16, y=16, z=16, t=32, fmt=12, prec="f16", nrhs=12),
        # One source on a large lattice in FP16 mixed precision (links dominate the traffic).
        dict(name="single_f16_large", kind="solve", x=32, y=32, z=32, t=64, fmt=12, prec="f16", nrhs=1),
        # FP32 mixed precision, a few sources, a lattice that no tile divides.
        dict(name="batch3_f32_ragged", kind="solve", x=20, y=12, z=28, t=36, fmt=18, prec="f32", nrhs=3),
        # The fermion part of one molecular-dynamics step: initial guess from the last
        # solutions, CG on the normal equations, M psi, and the force of both signs.
        dict(name="hmc_step", kind="hmc", x=16, y=12, z=12, t=24, fmt=18, nrhs=4),
        # CG on the unpreconditioned operator over all sites.
        dict(name="cg_full_16", kind="full", x=16, y=16, z=16, t=16, fmt=18),
        # Staggered fermions, a batch of sources with FP16 inner iterations.
        dict(name="stag_batch8_f16_24", kind="stagbatch", x=24, y=24, z=24, t=24, fmt=18, prec="f16", nrhs=8),
        # Staggered CG of one source in FP64, on a ragged lattice.
        dict(name="stag_cg_ragged", kind="stagcg", x=14, y=18, z=12, t=26, fmt=18),
    ]


# smallest and largest volume of each kind's draws (a draw costs no more than op_chain_32,
# batch12_f16_32 or single_f16_large)
_RANGE = {"noalloc": (256, 65536), "chain": (256, 32 ** 4), "solve": (256, 32 ** 4), "serve": (4096, 16 ** 3 * 32),
          "hmc": (256, 16 ** 3 * 24), "full": (256, 24 ** 4), "stagbatch": (256, 24 ** 3 * 32),
          "stagcg": (256, 24 ** 4)}


def draw(rng):
    kind = rng.choice(["noalloc", "chain", "solve", "solve", "solve", "solve", "serve", "hmc", "full", "stagbatch",
                       "stagcg"])
    lo, hi = _RANGE[kind]
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    side = want ** 0.25
    while True:
        d = [2 * max(1, round(side * math.exp(rng.uniform(-0.5, 0.5)) / 2)) for _ in range(3)]
        t = 2 * round(want / (d[0] * d[1] * d[2]) / 2)
        vol = d[0] * d[1] * d[2] * t
        if 2 <= t <= 96 and min(d) >= 4 and t >= 4 and lo <= vol <= hi:
            break
    case = dict(kind=kind, x=d[0], y=d[1], z=d[2], t=t, fmt=rng.choice([12, 18]))
    if kind == "noalloc":
        case.update(sign=rng.choice([1, -1]), reps=rng.choice([1, 2, 4]))
    elif kind == "chain":
        case.update(reps=rng.randint(4, 20))
    elif kind == "solve":
        prec = rng.choice(["f64", "f32", "f16", "f16"])
        case.update(prec=prec, nrhs=1 if prec == "f64" else rng.randint(1, 12 if prec == "f16" else 6))
    elif kind == "serve":
        case.update(prec="f16", nrhs=rng.randint(2, 12))
    elif kind == "hmc":
        case.update(nrhs=rng.randint(1, 6))
    elif kind == "stagbatch":
        case.update(prec=rng.choice(["f64", "f16"]), nrhs=rng.randint(1, 12))
    return case


KAPPA = 0.124   # Wilson hopping parameter of the benchmark workloads (about 70 CG iterations)
EPS = 0.3       # width of the links around the identity
MASS = 2.3      # staggered mass just above the hop's spectral radius
ACC = 1e-10     # |b - M x| / |b| asked of every solve

# iteration counts that the work model takes (measured on the listed lattices)
_ITERS = 73
_ITERS_HMC = 46
_ITERS_STAG = 150


def _dims(case):
    return (case["x"], case["y"], case["z"], case["t"])


def _serve_dims(case):
    """Lattices of the serving case: the largest, and smaller ones as a mixed stream has them."""
    x, y, z, t = _dims(case)
    half = lambda n: max(4, 2 * (n // 4))  # noqa: E731
    return [(x, y, z, t), (half(x), half(y), half(z), half(t)), (x, half(y), z, half(t)), (half(x), y, z, half(t))]


def _serve_requests(case):
    """(lattice, sources) of the requests in flight together."""
    n = case["nrhs"]
    return [(0, n), (1, 1), (2, max(1, n // 2)), (3, max(1, n // 3)), (1, n), (2, 1)]


# ------------------------------------------------------------------ inputs


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _links(dims, seed):
    """SU(3) links (4, V, 3, 3) complex128 on the GPU: rows of 1 + i eps H, H a Gaussian
    traceless Hermitian matrix, made orthonormal, the third the conjugate cross product."""
    V = math.prod(dims)
    g = _gen(seed)
    a = torch.randn(8, 4, V, generator=g, device="cuda", dtype=torch.float64) * (EPS * math.sqrt(2.0) / 2)
    one = torch.ones_like(a[0])
    r0 = torch.stack([torch.complex(one, a[2] + a[7] / math.sqrt(3.0)), torch.complex(a[1], a[0]),
                      torch.complex(a[4], a[3])], -1)
    r1 = torch.stack([torch.complex(-a[1], a[0]), torch.complex(one, -a[2] + a[7] / math.sqrt(3.0)),
                      torch.complex(a[6], a[5])], -1)
    del a, one
    r0 /= r0.abs().square().sum(-1, keepdim=True).sqrt()
    r1 -= (r0.conj() * r1).sum(-1, keepdim=True) * r0
    r1 /= r1.abs().square().sum(-1, keepdim=True).sqrt()
    r2 = torch.stack([r0[..., 1] * r1[..., 2] - r0[..., 2] * r1[..., 1],
                      r0[..., 2] * r1[..., 0] - r0[..., 0] * r1[..., 2],
                      r0[..., 0] * r1[..., 1] - r0[..., 1] * r1[..., 0]], -1).conj()
    return torch.stack([r0, r1, r2], -2).resolve_conj().contiguous()


def _source(sites, comps, seed):
    """Gaussian colour(-spin) vectors (sites, comps...) complex128 on the GPU."""
    return torch.randn(sites, *comps, 2, generator=_gen(seed), device="cuda", dtype=torch.float64)


def _host(t):
    t = torch.view_as_real(t) if t.is_complex() else t
    return t.cpu().numpy()


def _order(dims):
    """Lexicographic site index of each even-first position (EVEN sites, then ODD), on the GPU."""
    X, Y, Z, T = dims
    lex = torch.arange(X * Y * Z * T, device="cuda")
    par = (lex % X + (lex // X) % Y + (lex // (X * Y)) % Z + lex // (X * Y * Z)) % 2
    return torch.cat([lex[par == 0], lex[par == 1]])


def _pinned(*shape):
    """A page-locked host array (the array keeps its memory alive)."""
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


_kept = {}


def _context():
    """The program's one context (it owns the stream and the engines)."""
    if "ctx" not in _kept:
        _kept["ctx"] = hb.Context(0)
    return _kept["ctx"]


class State:
    """What a program holds for one case; handles go in the order the library asks for."""

    server = None
    handles = ()

    def __del__(self):
        try:
            if self.server is not None:
                self.server.close()
            for h in self.handles:
                h.close()
        except Exception:
            pass


def _gauge(dims, seed, fmt, s):
    lat = hb.Lattice(_context(), dims)
    s.handles = (*s.handles, lat)  # closes the fields made on it
    return hb.GaugeField(lat, _host(_links(dims, seed)), link_format=fmt)


def _full_source(dims, comps, seed):
    """A source on EVEN in lexicographic order (ODD zero), as (V, comps..., 2)."""
    V = math.prod(dims)
    f = torch.zeros(V, *comps, 2, device="cuda", dtype=torch.float64)
    f[_order(dims)[:V // 2]] = _source(V // 2, comps, seed)
    return f


def prepare(case, seed):
    s = State()
    s.case, s.dims, kind = case, _dims(case), case["kind"]
    V = math.prod(s.dims)
    if kind == "noalloc":
        s.stride = (V // 2 + 63) // 64 * 64
        planes = case["fmt"] // 2
        U = _links(s.dims, seed).reshape(4, V, 9)[:, _order(s.dims), :planes].reshape(4, 2, V // 2, planes)
        s.links = torch.zeros(2, 4, planes, s.stride, device="cuda", dtype=torch.complex128)
        s.links[..., :V // 2] = U.permute(1, 0, 3, 2)
        s.a = torch.zeros(12, s.stride, device="cuda", dtype=torch.complex128)
        s.a[:, :V // 2] = torch.view_as_complex(_source(V // 2, (12,), seed + 1000)).T
        s.b, s.c = torch.zeros_like(s.a), torch.zeros_like(s.a)
        return s
    if kind == "serve":
        s.server = hb.Server(_context(), precision=case["prec"], hbm_budget_bytes=16 << 30)
        s.requests = []
        gauges = [_gauge(d, seed + 100 * k, case["fmt"], s) for k, d in enumerate(_serve_dims(case))]
        s.ids = [s.server.add_gauge(g) for g in gauges]
        s.gauges = gauges
        for r, (k, n) in enumerate(_serve_requests(case)):
            half = math.prod(_serve_dims(case)[k]) // 2
            src, sol = _pinned(n, half, 4, 3, 2), _pinned(n, half, 4, 3, 2)
            for j in range(n):
                src[j] = _host(_source(half, (4, 3), seed + 1000 + 100 * r + j))
            s.requests.append((k, src, sol))
        return s
    s.gauge = _gauge(s.dims, seed, case["fmt"], s)
    lat = s.gauge.lattice
    if kind in ("stagbatch", "stagcg"):
        n = case.get("nrhs", 1)
        s.op = hb.dirac_staggered_evenodd(MASS, s.gauge)
        s.b = [hb.StaggeredField(lat, _host(_full_source(s.dims, (3,), seed + 1000 + j))) for j in range(n)]
        s.x = [hb.StaggeredField(lat) for _ in range(n)]
        return s
    half = V // 2
    n = case.get("nrhs", 1)
    s.out = _pinned(n if kind == "solve" else 1, V if kind == "full" else half, 4, 3, 2)
    s.op = hb.Dirac_Wilson(KAPPA, s.gauge) if kind == "full" else hb.Dirac_Wilson_evenodd(KAPPA, s.gauge)
    if kind == "full":
        s.b, s.x = hb.Field(lat), hb.Field(lat)
        s.b.upload_eo(_host(_source(V, (4, 3), seed + 1000)), hb.ALL)
        return s

    def even(j):
        f = hb.Field(lat)
        f.upload_eo(_host(_source(half, (4, 3), seed + 1000 + j)), hb.EVEN)
        return f

    if kind == "hmc":
        s.chi, s.psi, s.y = even(0), hb.Field(lat), hb.Field(lat)
        s.cg = hb.CG(s.op, accuracy=ACC, true_residual=True)
        # earlier solutions of nearby systems: this one's to about a percent each
        x, s.old = hb.Field(lat), []
        hb.CG(s.op, accuracy=1e-6).apply(s.chi, x)
        base = x.download_eo(hb.EVEN)[:half]
        scale = 0.01 * math.sqrt(float(np.mean(base * base)))
        for j in range(n):
            f = hb.Field(lat)
            f.upload_eo(base + scale * _host(_source(half, (4, 3), seed + 2000 + j)), hb.EVEN)
            s.old.append(f)
        return s
    s.b = [even(j) for j in range(n)]
    s.x = [hb.Field(lat) for _ in range(n)]
    if kind == "chain":
        s.tmp = hb.Field(lat)
    return s


# ------------------------------------------------------------------ one pass


def run(s):
    case, kind = s.case, s.case["kind"]
    if kind == "noalloc":
        src = s.a
        for r in range(case["reps"]):
            dst = s.b if r % 2 == 0 else s.c
            hb.wilson_evenodd_apply_noalloc(s.dims, KAPPA, case["sign"], s.links.data_ptr(), src.data_ptr(),
                                            dst.data_ptr(), s.stride, case["fmt"],
                                            stream=torch.cuda.current_stream().cuda_stream)
            src = dst
        return src
    if kind == "chain":
        src, a, b = s.b[0], s.x[0], s.tmp
        for _ in range(case["reps"]):
            s.op.apply(src, b)
            s.op.dagger(b, a)
            src = a
        a.download_eo(hb.EVEN, s.out[0])
        return s.out[0]
    if kind == "serve":
        ids = []
        for k, src, sol in s.requests:
            ids.append(s.server.submit_eo(s.ids[k], KAPPA, list(src), list(sol), accuracy=ACC))
        for rid, (k, src, _) in zip(ids, s.requests):
            s.server.wait(rid, len(src), s.gauges[k].lattice.volume, copy=False)
        return [sol for _, _, sol in s.requests]
    if kind == "full":
        s.x.zero(hb.ALL)
        s.op.cg(s.b, s.x, accuracy=ACC)
        s.x.download_eo(hb.ALL, s.out[0])
        return s.out[0]
    if kind == "hmc":
        hb.mre_guess(s.op, s.old, s.chi, s.psi)
        s.cg.apply(s.chi, s.psi)
        s.op.apply(s.psi, s.y)
        f1 = s.op.force(s.y, s.psi, 1)
        f2 = s.op.force(s.psi, s.y, -1)
        s.psi.download_eo(hb.EVEN, s.out[0])
        return {"psi": s.out[0], "force": f1, "force_dagger": f2}
    for x in s.x:
        x.zero(hb.EVEN)
    if kind == "stagcg":
        s.op.cg(s.b[0], s.x[0], accuracy=ACC)
        return s.x[0].download(hb.EVEN)
    if kind == "stagbatch":
        hb.staggered_batch_solve(_context(), [(s.op, b, x, ACC) for b, x in zip(s.b, s.x)], precision=case["prec"])
        return [x.download(hb.EVEN) for x in s.x]
    if case["prec"] == "f64":
        s.op.solve(s.b[0], s.x[0], accuracy=ACC)
    else:
        delta = 0.005 if case["prec"] == "f16" else 1e-5
        hb.batch_solve(_context(), [(s.op, b, x, ACC) for b, x in zip(s.b, s.x)], precision=case["prec"], delta=delta)
    for j, x in enumerate(s.x):
        x.download_eo(hb.EVEN, s.out[j])
    return s.out


# ------------------------------------------------------------------ work


def _solve_bytes(prec, fmt, half, nrhs, iters):
    """CG on the normal equations: per iteration M^dag M reads the links of both parities once
    (its two halves may share one read of M's) and reads p, r, x (or the increment), writes them."""
    if prec == "f64":
        spin, acc, link = 192, 192, 16 * (fmt // 2)
    elif prec == "f32":
        spin, acc, link = 96, 96, 48
    else:
        spin, acc, link = 52, 96, 24
    return iters * half * (8 * link + nrhs * (4 * spin + 2 * acc))


def work(case):
    kind, dims = case["kind"], _dims(case)
    V = math.prod(dims)
    half, n = V // 2, case.get("nrhs", 1)
    flink = 16 * (case["fmt"] // 2)  # bytes of an FP64 link
    hop = 1320 * V                   # flops of an even-odd application (two hops of V/2 sites)
    apply_bytes = 4 * V * flink + 2 * half * 192
    if kind == "noalloc":
        return {"bytes": case["reps"] * apply_bytes, "flops": case["reps"] * hop}
    if kind == "chain":
        return {"bytes": 2 * case["reps"] * apply_bytes, "flops": 2 * case["reps"] * hop}
    if kind == "solve":
        return {"bytes": _solve_bytes(case["prec"], case["fmt"], half, n, _ITERS),
                "flops": n * _ITERS * (2 * hop + 48 * 6 * half)}
    if kind == "serve":
        b = f = 0
        for k, m in _serve_requests(case):
            h = math.prod(_serve_dims(case)[k]) // 2
            b += _solve_bytes("f16", 12, h, m, _ITERS)
            f += m * _ITERS * (2 * 2640 * h + 48 * 6 * h)
        return {"bytes": b, "flops": f}
    if kind == "hmc":
        b = _solve_bytes("f64", case["fmt"], half, 1, _ITERS_HMC) + n * (2 * apply_bytes + half * 192)
        b += 2 * (4 * V * 144 + 2 * half * 192)
        return {"bytes": b, "flops": (_ITERS_HMC + n) * 2 * hop}
    if kind == "full":
        iters = 190
        return {"bytes": iters * (4 * V * flink + 6 * V * 192), "flops": iters * 2 * 1320 * V}
    iters = _ITERS_STAG
    if kind == "stagbatch" and case["prec"] == "f16":
        return {"bytes": iters * half * (8 * 24 + n * (4 * 16 + 2 * 24)), "flops": n * iters * 2 * 570 * V}
    return {"bytes": iters * half * (8 * flink + n * 6 * 48), "flops": n * iters * 2 * 570 * V}


def tolerance(case):
    kind = case["kind"]
    if kind == "noalloc":
        return {"rel": 1e-15}  # M is near the identity: 1e-16 measured against 64 bits
    if kind == "chain":
        return {"rel": 4e-15}  # 3e-16 measured after 20 M^dag M
    # a solve ends anywhere below the accuracy asked for: two correct ones differ by its error
    # (1e-10 to 1e-9 measured against 64 bits, most in the normal-equation solve of the hmc case)
    return {"rel": 4e-9}


# ------------------------------------------------------------------ 64-bit reference
#
# The operators written out on whole lattices (T, Z, Y, X, ...) in complex128.


_GAMMA = {  # (1 + s gamma_mu) w = w + s (rows below): (phase, source spin) of each spin
    0: [(1j, 3), (1j, 2), (-1j, 1), (-1j, 0)],
    1: [(-1, 3), (1, 2), (1, 1), (-1, 0)],
    2: [(1j, 2), (-1j, 3), (-1j, 0), (1j, 1)],
    3: [(1, 2), (1, 3), (1, 0), (1, 1)],
}


def _gamma(mu, w):
    return torch.stack([ph * w[..., sp, :] for ph, sp in _GAMMA[mu]], -2)


def _shift(f, mu, step):
    """f(x + step mu) with the antiperiodic t boundary."""
    g = torch.roll(f, -step, dims=3 - mu)
    if mu == 3:
        g = g.clone()
        g[-1 if step > 0 else 0] *= -1
    return g


def _mul(U, v):
    """U v on the last (colour) axis; a spin axis before it is broadcast."""
    if v.dim() > U.dim() - 1:
        U = U.unsqueeze(-3)
    return (U * v.unsqueeze(-2)).sum(-1)


class _Exact:
    def __init__(self, dims, seed):
        X, Y, Z, T = dims
        self.dims, self.shape = dims, (T, Z, Y, X)
        self.V = math.prod(dims)
        U = _links(dims, seed)
        self.U = [U[d].reshape(T, Z, Y, X, 3, 3) for d in range(4)]
        # U(x - mu) on the links' periodic boundary, conjugate transposed
        self.Ub = [torch.roll(u, 1, dims=3 - d).mH.resolve_conj().contiguous() for d, u in enumerate(self.U)]
        self.order = _order(dims)
        c = [torch.arange(n, device="cuda") for n in (T, Z, Y, X)]
        t, z, y, x = torch.meshgrid(*c, indexing="ij")
        self.even = ((x + y + z + t) % 2 == 0)
        self.eta = [((s % 2) * 2 - 1).double() for s in (0 * x, x, x + y, x + y + z)]

    def field(self, even_first, comps):
        f = torch.zeros(self.V, *comps, device="cuda", dtype=torch.complex128)
        e = torch.view_as_complex(even_first)
        f[self.order[:len(e)]] = e
        return f.reshape(*self.shape, *comps)

    def mask(self, f, even=True):
        m = self.even if even else ~self.even
        return f * m.reshape(*self.shape, *([1] * (f.dim() - 4)))

    def hop(self, v, s):
        out = torch.zeros_like(v)
        for mu in range(4):
            f = _mul(self.U[mu], _shift(v, mu, 1))
            out += f + s * _gamma(mu, f)
            b = _shift(v, mu, -1)
            b = _mul(self.Ub[mu], b)
            out += b - s * _gamma(mu, b)
        return out

    def M(self, v, s):
        return v - KAPPA ** 2 * self.mask(self.hop(self.mask(self.hop(v, s), False), s))

    def D(self, v, s):
        return v - KAPPA * self.hop(v, s)

    def stag_hop(self, v, s):
        out = torch.zeros_like(v)
        for mu in range(4):
            b = _mul(self.Ub[mu], _shift(v, mu, -1))
            out += (0.5 * s) * self.eta[mu].unsqueeze(-1) * (_mul(self.U[mu], _shift(v, mu, 1)) - b)
        return out

    def S(self, v, s):
        return MASS * v + self.mask(self.stag_hop(self.mask(self.stag_hop(v, s), False) / MASS, s))

    def cg(self, op, b, tol=1e-13):
        """op(op(x, 1), -1) = b"""
        x = torch.zeros_like(b)
        r, p = b.clone(), b.clone()
        rr = bb = float(torch.linalg.vector_norm(r) ** 2)
        for _ in range(3000):
            q = op(p, 1)
            a = rr / float(torch.linalg.vector_norm(q) ** 2)
            x += a * p
            r -= a * op(q, -1)
            new = float(torch.linalg.vector_norm(r) ** 2)
            if new <= tol * tol * bb:
                break
            p = r + (new / rr) * p
            rr = new
        return x

    def outer(self, a, b):
        return torch.einsum("...si,...sj->...ij", a, b.conj())

    def force(self, chi, psi, s):
        t1 = -KAPPA * self.mask(self.hop(chi, -s), False)
        t2 = -KAPPA * self.mask(self.hop(psi, s), False)
        F = torch.zeros(4, *self.shape, 3, 3, device="cuda", dtype=torch.complex128)
        for mu in range(4):
            def pr(v, sign):
                w = _shift(v, mu, 1)
                return w + sign * _gamma(mu, w)
            F[mu] = KAPPA * (self.outer(pr(t1, -s), psi) + self.outer(pr(t2, s), chi)
                             + self.outer(pr(psi, s), t1) + self.outer(pr(chi, -s), t2))
        return F.reshape(4, self.V, 3, 3)

    def eo(self, f, sites=None):
        f = f.reshape(self.V, *f.shape[4:])[self.order[:sites or self.V // 2]]
        return _host(f.contiguous())

    def lex(self, f):
        return _host(f.reshape(self.V, *f.shape[4:]).contiguous())


def _exact_solutions(dims, seed, sources, comps, count):
    """x of M x = b for the first `count` sources, None for the others."""
    E = _Exact(dims, seed)
    op = E.M if len(comps) == 2 else E.S
    out = []
    for j, sd in enumerate(sources):
        if j >= count:
            out.append(None)
            continue
        b = E.field(_source(E.V // 2, comps, sd), comps)
        x = E.cg(op, op(b, -1))
        out.append(E.eo(x) if len(comps) == 2 else E.lex(x))
    return out


def exact(case, seed):
    kind, dims = case["kind"], _dims(case)
    V = math.prod(dims)
    if kind == "serve":
        out = []
        for r, (k, n) in enumerate(_serve_requests(case)):
            sources = [seed + 1000 + 100 * r + j for j in range(n)]
            if math.prod(_serve_dims(case)[k]) * n > 65536 * 8:
                out.append(None)
                continue
            out.append(np.stack(_exact_solutions(_serve_dims(case)[k], seed + 100 * k, sources, (4, 3), n)))
        return out
    if kind == "solve":
        n = case["nrhs"]
        if V * n > 32 ** 4 * 3:
            return None
        return np.stack(_exact_solutions(dims, seed, [seed + 1000 + j for j in range(n)], (4, 3), n))
    if kind == "stagbatch":
        n = case["nrhs"]
        count = max(1, min(n, 24 ** 4 // V))
        return _exact_solutions(dims, seed, [seed + 1000 + j for j in range(n)], (3,), count)
    E = _Exact(dims, seed)
    if kind == "noalloc":
        src = torch.view_as_real(torch.view_as_complex(_source(V // 2, (12,), seed + 1000)).reshape(V // 2, 4, 3))
        v = E.field(src.contiguous(), (4, 3))
        for _ in range(case["reps"]):
            v = E.M(v, case["sign"])
        out = np.zeros((12, (V // 2 + 63) // 64 * 64), np.complex128)
        out[:, :V // 2] = E.eo(v).reshape(V // 2, 12, 2).view(np.complex128)[..., 0].T
        return torch.from_numpy(out)
    if kind == "chain":
        v = E.field(_source(V // 2, (4, 3), seed + 1000), (4, 3))
        for _ in range(case["reps"]):
            v = E.M(E.M(v, 1), -1)
        return E.eo(v)
    if kind == "full":
        b = E.field(_source(V, (4, 3), seed + 1000), (4, 3))
        return E.eo(E.cg(E.D, b), V)
    if kind == "stagcg":
        b = E.field(_source(V // 2, (3,), seed + 1000), (3,))
        return E.lex(E.cg(E.S, b))
    chi = E.field(_source(V // 2, (4, 3), seed + 1000), (4, 3))
    psi = E.cg(E.M, chi)
    y = E.M(psi, 1)
    return {"psi": E.eo(psi), "force": _host(E.force(y, psi, 1)), "force_dagger": _host(E.force(psi, y, -1))}
