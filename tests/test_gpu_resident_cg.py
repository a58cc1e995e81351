"""The FP64 hop of small lattices (eight warps per 32 sites) against the one-thread-per-site
kernel, and the loop graphs of the unpreconditioned and staggered CG on consecutive sources, at
the edges of their groups of 32 sites and blocks of 128.

Two solves that stop at |b - A x| / |b| <= acc differ by at most 2 acc |A^-1| |A| |x|; the
condition numbers here are below 20 for M (kappa 0.12) and 400 for its normal system, so
1e-8 bounds the solutions at acc = 1e-11.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ACC = 1e-11
SOL_TOL = 1e-8


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# sites per parity: 8 (a quarter of a group), 24, 96, 240, 2048, 9240 (near the limit of the rule)
@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 2, 2, 6), (4, 2, 6, 4), (6, 4, 2, 10), (8, 8, 8, 8),
                                  (6, 10, 14, 22)])
@pytest.mark.parametrize("link_format", [18, 12])
def test_split_hop(hw, ctx, oracle, monkeypatch, dims, link_format):
    """Every epilogue of the small lattices' hop: the same bits as the one-thread-per-site kernel
    for operators, and the same solutions (the sums of |.|^2 are formed in another order)."""
    U = oracle.gen_links(dims, 0.3, 5)
    src, guess = oracle.gen_spinor(dims, 6, oracle.ALL), 0.1 * oracle.gen_spinor(dims, 7, oracle.EVEN)

    def run(variant):
        if variant is None:
            monkeypatch.delenv("HW_HOP_VARIANT", raising=False)
        else:
            monkeypatch.setenv("HW_HOP_VARIANT", variant)
        lat = hw.Lattice(ctx, dims)  # the launch shape is chosen per lattice
        G = hw.GaugeField(lat, U, link_format)
        D, F = hw.Dirac_Wilson_evenodd(0.12, G), hw.Dirac_Wilson(0.12, G)
        b, bits, sols = hw.Field(lat, src), [], []
        for op in (D.apply, D.dagger, F.apply, F.dagger, hw.Hasenbusch_operator(D, 0.3).dagger):
            o = hw.Field(lat, guess, oracle.ALL)
            op(b, o)
            bits.append(o.download())
        for parity in (hw.EVEN, hw.ODD):
            for sign in (1, -1):
                for set_ in (True, False):
                    o = hw.Field(lat, src)
                    D.hop(b, o, parity, sign, set_)
                    bits.append(o.download())
        for solve in (lambda x: hw.CG(D, accuracy=ACC, true_residual=True).apply(b, x),
                      lambda x: hw.Hasenbusch_operator(D, 0.05).solve(b, x, accuracy=ACC),
                      lambda x: D.solve(b, x, accuracy=ACC, use_graph=False)):
            x = hw.Field(lat, guess)
            r = solve(x)
            assert r.converged and r.true_residual <= ACC
            sols.append((r.iterations, x.download()))
        return bits, sols

    split, one = run(None), run("0")
    for a, b in zip(split[0], one[0]):
        assert np.array_equal(a, b)
    for (ia, a), (ib, b) in zip(split[1], one[1]):
        assert abs(ia - ib) <= 2 and rel(a, b) <= SOL_TOL


def test_cg_limits(hw, ctx, oracle):
    """A zero source, an iteration limit, and the same bits on a repeated solve."""
    dims = (4, 4, 4, 4)
    lat = hw.Lattice(ctx, dims)
    D = hw.Dirac_Wilson_evenodd(0.12, hw.GaugeField(lat, oracle.gen_links(dims, 0.3, 5)))
    zero, x = hw.Field(lat), hw.Field(lat)
    r = hw.CG(D).apply(zero, x)
    assert r.converged and r.iterations == 0 and not x.download().any()
    b = hw.Field(lat, oracle.gen_spinor(dims, 6, oracle.EVEN))
    r = D.solve(b, x, accuracy=1e-10, maxiters=3)
    assert r.status == hw.HW_ERR_NOT_CONVERGED and r.iterations == 3
    runs = []
    for _ in range(2):
        x.zero()
        r = D.solve(b, x, accuracy=1e-10)
        runs.append((r.iterations, x.download().tobytes()))
    assert runs[0] == runs[1]


@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (6, 2, 4, 10), (8, 8, 8, 8), (18, 14, 10, 22), (24, 24, 24, 20)])
@pytest.mark.parametrize("link_format", [18, 12])
def test_loop_graph_solvers(hw, ctx, oracle, dims, link_format):
    """Several sources, solutions, couplings and gauge fields on one lattice share a workspace and
    rebuild its loop graph; the operator of the solution gives the source back."""
    lat = hw.Lattice(ctx, dims)
    for seed, kappa, mass in ((5, 0.11, 4.0), (6, 0.11, 4.0), (6, 0.12, 5.0)):
        G = hw.GaugeField(lat, oracle.gen_links(dims, 0.3, seed), link_format)
        D, S = hw.Dirac_Wilson(kappa, G), hw.dirac_staggered_evenodd(mass, G)
        for k in range(2):
            b, x, y, z = (hw.Field(lat, oracle.gen_spinor(dims, 10 + k, oracle.ALL)), hw.Field(lat), hw.Field(lat),
                          hw.Field(lat))
            r = D.cg(b, x, accuracy=ACC)
            assert r.converged
            D.apply(x, y)
            D.dagger(y, z)
            assert rel(z.download(), b.download()) <= 10 * ACC
            rng = np.random.default_rng(20 + k)
            sb = hw.StaggeredField(lat, rng.standard_normal((lat.volume, 3, 2)), hw.EVEN)
            sx, sy, sz = (hw.StaggeredField(lat) for _ in range(3))
            r = S.cg(sb, sx, accuracy=ACC)
            assert r.converged
            S.apply(sx, sy)
            S.dagger(sy, sz)
            assert rel(sz.download(hw.EVEN), sb.download(hw.EVEN)) <= 10 * ACC


@pytest.mark.parametrize("variant", ["0", "1", "2", "3"])
def test_every_hop_shape(hw, ctx, oracle, monkeypatch, variant):
    """Each launch shape on a lattice above the limit of the small lattices' rule (10368 sites per
    parity): the sums of an explicit residual fit the buffer reserved for that shape."""
    dims = (12, 12, 12, 12)
    monkeypatch.setenv("HW_HOP_VARIANT", variant)
    lat = hw.Lattice(ctx, dims)
    D = hw.Dirac_Wilson_evenodd(0.12, hw.GaugeField(lat, oracle.gen_links(dims, 0.3, 5)))
    b, x, y = hw.Field(lat, oracle.gen_spinor(dims, 6, oracle.EVEN)), hw.Field(lat), hw.Field(lat)
    r = D.solve(b, x, accuracy=ACC)
    assert r.converged and r.true_residual <= ACC
    D.apply(x, y)
    assert rel(y.download(), b.download()) <= 2 * ACC


@pytest.mark.parametrize("kind", ["wilson", "staggered"])
def test_loop_graph_limits(hw, ctx, oracle, kind):
    """The loop-graph solvers on a source or guess that is not finite (a breakdown, as in the
    even-odd CG), at an iteration limit, on a zero source, and on a good source afterwards."""
    dims = (4, 6, 2, 8)
    lat = hw.Lattice(ctx, dims)
    G = hw.GaugeField(lat, oracle.gen_links(dims, 0.3, 5))
    op = hw.Dirac_Wilson(0.11, G) if kind == "wilson" else hw.dirac_staggered_evenodd(4.0, G)
    comps = (4, 3, 2) if kind == "wilson" else (3, 2)
    good = np.random.default_rng(3).standard_normal((lat.volume, *comps))

    def field(host):
        return hw.Field(lat, host) if kind == "wilson" else hw.StaggeredField(lat, host, hw.EVEN)

    def solve(b, x, **kw):
        fb, fx = field(b), field(x)
        r = op.cg(fb, fx, accuracy=1e-10, **kw)
        return r, fx.download(hw.ALL if kind == "wilson" else hw.EVEN)

    zero = np.zeros_like(good)
    for value in (np.nan, np.inf, 1e200):  # the square of the last overflows
        for site in ((0, lat.volume - 1) if kind == "wilson" else (0,)):
            bad = good.copy()
            bad[(site,) + (0,) * len(comps)] = value
            for true_residual in (False, True):
                r, _ = solve(bad, zero, true_residual=true_residual)
                assert r.status == hw.HW_ERR_BREAKDOWN and r.iterations == 0
                r, _ = solve(good, bad, true_residual=true_residual)
                assert r.status == hw.HW_ERR_BREAKDOWN and r.iterations == 0
    r, _ = solve(good, zero, maxiters=3)
    assert r.status == hw.HW_ERR_NOT_CONVERGED and r.iterations == 3
    r, x = solve(zero, zero)
    assert r.converged and r.iterations == 0 and not x.any()
    r, _ = solve(good, zero, true_residual=True)
    assert r.converged and r.true_residual <= 1e-10


def test_launch_counts(hw, ctx, oracle, monkeypatch):
    """kernel_launches against the kernels that the loops are made of: start + bodies + check."""
    dims = (4, 4, 4, 4)
    U = oracle.gen_links(dims, 0.3, 5)

    def system(c):
        lat = hw.Lattice(c, dims)
        G = hw.GaugeField(lat, U)
        return lat, G, hw.Field(lat, oracle.gen_spinor(dims, 6, oracle.EVEN)), hw.Field(lat)

    lat, G, b, x = system(ctx)
    D, F, S = hw.Dirac_Wilson_evenodd(0.12, G), hw.Dirac_Wilson(0.12, G), hw.dirac_staggered_evenodd(4.0, G)
    r = D.solve(b, x, accuracy=1e-10, maxiters=3)
    assert r.iterations == 3 and r.kernel_launches == 7 + 5 * 3 + 2
    x.zero()
    r = D.solve(b, x, accuracy=1e-10, maxiters=3, use_graph=False)  # 16 bodies before the host looks
    assert r.iterations == 3 and r.kernel_launches == 7 + 6 * 16 + 2
    x.zero()
    r = hw.CG(D, accuracy=1e-10).apply(b, x)
    assert r.kernel_launches == 5 + 5 * r.iterations + 4
    x.zero()
    r = F.cg(b, x, accuracy=1e-10)
    assert r.kernel_launches == 4 + 3 * r.iterations
    sb, sx = hw.StaggeredField(lat, np.ones((lat.volume, 3, 2)), hw.EVEN), hw.StaggeredField(lat)
    r = S.cg(sb, sx, accuracy=1e-10)
    assert r.kernel_launches == 8 + 5 * r.iterations
    # engine: per chunk 1, per body P1..P4, gate, P5, control, per update R1..R5L
    for prec in ("f16", "f32"):
        x.zero()
        r = D.solve(b, x, accuracy=1e-10, precision=prec)
        chunks = -(-(r.iterations + 1) // 64)
        assert r.converged and r.kernel_launches == chunks + 7 * (r.iterations + 1) + 7 * r.reliable_updates
    # a host loop launches every phase in all 64 iterations of a chunk, and no gate
    monkeypatch.setenv("HW_USE_GRAPH", "0")
    c = hw.Context(0)
    lat, G, b, x = system(c)
    r = hw.Dirac_Wilson_evenodd(0.12, G).solve(b, x, accuracy=1e-10, precision="f16")
    chunks = -(-(r.iterations + 1) // 64)
    assert r.converged and r.kernel_launches == chunks * (1 + 64 * 13)
    lat.close()
    c.close()


def test_workspaces_are_given_back(hw, ctx):
    """The workspaces that the loop-graph solvers keep with their lattices stay within 1 GiB
    together (ten lattices of 123 MB each here), and go with the lattices."""
    import torch
    dims = (20, 20, 20, 20)
    U = np.zeros((4, 20 ** 4, 3, 3, 2))
    U[:, :, range(3), range(3), 0] = 1.0
    b = np.ones((20 ** 4, 4, 3, 2))
    c = hw.Context(0)
    lats, before = [], None
    for k in range(11):
        lat = hw.Lattice(c, dims)
        G, fb, fx = hw.GaugeField(lat, U), hw.Field(lat, b), hw.Field(lat)
        lats.append((lat, hw.Dirac_Wilson(0.1, G), fb, fx))
        if k == 0:  # what a first solve makes besides its workspace
            lats[0][1].cg(fb, fx, maxiters=1)
            lats[0][0].close()
    before = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        for lat, D, fb, fx in lats[1:]:
            assert D.cg(fb, fx, maxiters=1).status in (hw.HW_OK, hw.HW_ERR_NOT_CONVERGED)
    kept = before - torch.cuda.mem_get_info()[0]
    assert 0.5 * 2 ** 30 <= kept <= 2 ** 30 + 64 * 2 ** 20
    for lat, *_ in lats[1:]:
        lat.close()
    assert torch.cuda.mem_get_info()[0] >= before
    c.close()


def test_out_of_memory_is_reported_once(hw, ctx, oracle):
    """A field that no device holds (204 GB a half) fails by itself; calls after it do not."""
    lat = hw.Lattice(ctx, (4, 4, 4, 4))
    D = hw.Dirac_Wilson_evenodd(0.12, hw.GaugeField(lat, oracle.gen_links((4, 4, 4, 4), 0.3, 5)))
    a, b = hw.Field(lat, oracle.gen_spinor((4, 4, 4, 4), 6, oracle.EVEN)), hw.Field(lat)
    D.apply(a, b)
    huge = hw.Lattice(ctx, (208, 200, 200, 256))
    with pytest.raises(hw.HilaError) as e:
        hw.Field(huge)
    assert e.value.code == hw.HW_ERR_OOM
    D.apply(a, b)
    huge.close()
