"""Work items of the engine that divide a tile's solves, pairs of sources in the staggered FP16
phases, and copies into pageable memory by several threads.

A solve gives the same bits however its tile's solves are divided and whichever solve shares
its thread; sizes sit at the edges of tiles (128 sites), of pairs and of the division (one tile
to more than two per block)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-10


# tiles of 128 sites: 1 (8 sites), 2 (one partly filled), 81, 162 and 1800 (no division in the
# phases with the fewest blocks)
@pytest.mark.parametrize("dims,counts", [((2, 2, 2, 2), (1, 5)), ((6, 4, 2, 6), (2, 3, 16)), ((12, 12, 12, 12), (13,)),
                                         ((12, 24, 12, 12), (1, 7)), ((24, 20, 24, 40), (3,))])
@pytest.mark.parametrize("precision", ["f16", "f32"])
def test_divided_tiles(hw, ctx, dims, counts, precision):
    lat = hw.Lattice(ctx, dims)
    D = hw.Dirac_Wilson_evenodd(0.12, hw.GaugeField(lat, hw.generate_links(dims, 0.3, 3)))
    delta = 0.005 if precision == "f16" else 1e-5
    bs = [hw.Field(lat, hw.generate_spinor(dims, 30 + k, hw.EVEN)) for k in range(max(counts))]

    def solve(idx):
        xs = [hw.Field(lat) for _ in idx]
        res = hw.batch_solve(ctx, [(D, bs[k], x, TOL) for k, x in zip(idx, xs)], precision=precision, delta=delta)
        assert all(r.converged and r.true_residual <= TOL for r in res)
        return [(r.iterations, x.download().tobytes()) for r, x in zip(res, xs)]

    alone = {}
    for n in counts:
        batch = solve(range(n))
        for k in {0, n // 2, n - 1}:
            if k not in alone:
                alone[k] = solve([k])[0]
            assert batch[k] == alone[k], (n, k)


@pytest.mark.parametrize("precision", ["f16", "f32"])
def test_divided_lattices(hw, ctx, precision):
    """Lattices with 1, 3 and 13 solves in one launch, divided by one rule (their solves leave at
    different iterations): the bits of the solves alone."""
    delta = 0.005 if precision == "f16" else 1e-5
    reqs, alone = [], []
    for dims, n, kappa in (((8, 8, 8, 12), 13, 0.12), ((2, 4, 6, 2), 1, 0.1), ((12, 12, 12, 12), 3, 0.11)):
        lat = hw.Lattice(ctx, dims)
        D = hw.Dirac_Wilson_evenodd(kappa, hw.GaugeField(lat, hw.generate_links(dims, 0.3, 3), 18 if n == 3 else 12))
        for k in range(n):
            tol = TOL * 10 ** (k % 4)
            reqs.append((D, hw.Field(lat, hw.generate_spinor(dims, 50 + k, hw.EVEN)), hw.Field(lat), tol))
    for D, b, x, tol in reqs:
        r = hw.batch_solve(ctx, [(D, b, x, tol)], precision=precision, delta=delta)[0]
        assert r.converged
        alone.append((r.iterations, x.download().tobytes()))
        x.zero()
    res = hw.batch_solve(ctx, reqs, precision=precision, delta=delta)
    for r, (_, _, x, _), a in zip(res, reqs, alone):
        assert (r.iterations, x.download().tobytes()) == a


@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (6, 4, 2, 6), (8, 8, 8, 8), (12, 12, 12, 14)])
@pytest.mark.parametrize("normal", [False, True])
def test_staggered_pairs(hw, ctx, dims, normal):
    """1 to 16 sources, odd counts among them, beside FP64 slots of the same engine."""
    lat = hw.Lattice(ctx, dims)
    S = hw.dirac_staggered_evenodd(4.0, hw.GaugeField(lat, hw.generate_links(dims, 0.3, 4)))
    rng = np.random.default_rng(5)
    bs = [hw.StaggeredField(lat, rng.standard_normal((lat.volume, 3, 2)), hw.EVEN) for _ in range(16)]

    def solve(idx, precision="f16"):
        xs = [hw.StaggeredField(lat) for _ in idx]
        res = hw.staggered_batch_solve(ctx, [(S, bs[k], x, TOL, 10000, normal) for k, x in zip(idx, xs)],
                                       precision=precision)
        assert all(r.converged and r.true_residual <= TOL for r in res)
        return [x.download(hw.EVEN) for x in xs]

    whole = solve(range(16))
    for n in (1, 2, 3, 5):
        for a, b in zip(solve(range(n)), whole):
            assert np.array_equal(a, b)
    for a, b in zip(solve(range(3), "f64"), whole):  # the same solution: both residuals are <= TOL
        assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)
    for a, b in zip(solve(range(3)), whole):  # the FP16 phases again, after the FP64 ones ran
        assert np.array_equal(a, b)


# field bytes below, at and above the 2 MiB where the threads begin, whole and broken chunks
@pytest.mark.parametrize("dims", [(8, 8, 8, 10), (16, 8, 8, 16), (10, 10, 12, 14), (16, 16, 16, 16)])
def test_pageable_copies(hw, ctx, dims):
    V = int(np.prod(dims))
    lat = hw.Lattice(ctx, dims)
    data = np.random.default_rng(6).standard_normal((V, 4, 3, 2))
    f = hw.Field(lat)
    f.upload_eo(data, hw.ALL)
    assert np.array_equal(f.download_eo(hw.ALL), data)
    pinned = hw.PinnedArray((V, 4, 3, 2))
    f.download_eo(hw.ALL, pinned.array)
    assert np.array_equal(pinned.array, data)
    f.upload(data)
    assert np.array_equal(f.download(), data)
    s = hw.StaggeredField(lat, data[:, 0])
    assert np.array_equal(s.download(), data[:, 0])
    D = hw.Dirac_Wilson_evenodd(0.12, hw.GaugeField(lat, hw.generate_links(dims, 0.3, 4)))
    a, b = D.force(f, f, 1), D.force(f, f, 1)
    assert np.isfinite(a).all() and np.array_equal(a, b)
