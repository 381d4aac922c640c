"""The ray kernel's search of the ray map and the grouping of the importance walks, at the sizes where they can go
wrong: entries per ray below and above one, weights that leave lanes beyond the searched interval, ray counts around
a warp and a work item; line counts around the teams' sizes, several levels of a point in one team."""

from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from conftest import legacy_mesh, legacy_spectrum

pytestmark = pytest.mark.gpu


def _weights(kind, n, rng):
    if kind == "uniform":
        return np.ones(n)
    if kind == "one_heavy":  # almost every ray in one entry, the rest of the entries share a few
        w = np.full(n, 1e-7)
        w[n // 3] = 1.0
        return w
    if kind == "clusters":  # runs of empty entries between dense ones
        w = np.zeros(n)
        w[:: max(1, n // 37)] = 1.0
        w[5:9] = 1e-3
        return w
    return rng.random(n) ** 12  # "spiky"


@pytest.mark.parametrize("kind", ["uniform", "one_heavy", "clusters", "spiky"])
@pytest.mark.parametrize("rays", [1, 31, 33, 1000, 70_000])
def test_rays_follow_the_map(oracle, native, kind, rays):
    """Every ray starts in its map entry: the estimate from the caller's weights equals the oracle's replay of the same
    rays (the parity level of the replays, 1e-4)."""
    import torch

    from haseongpu_b200 import DeviceMesh

    mesh = legacy_mesh("cylindrical")
    sa, se = legacy_spectrum("cylindrical")
    w = np.where(mesh.betaVolume > 0, _weights(kind, mesh.numberOfPrisms, np.random.default_rng(1)), 0.0).astype(np.float32)
    sample = 2050
    with DeviceMesh(mesh, sa, se) as ctx:
        d_w, d_out = torch.from_numpy(w).cuda(), torch.zeros(4, dtype=torch.float64, device="cuda")
        native.check(native.lib().hase_estimate_sample_noalloc(ctx.handle, sample, C.c_void_p(d_w.data_ptr()), rays, 9,
                                                               0, 1, C.c_void_p(d_out.data_ptr())))
        got = d_out.cpu().numpy()
    ref = oracle.phi_ase(mesh, (sa, se), minRays=rays, seed=9, minSample=sample, maxSample=sample, weights=w[None])
    assert got[2] == rays and got[3] == 0
    np.testing.assert_allclose(got[0], float(ref["phiAse"][0]), rtol=1e-4)


@pytest.mark.parametrize("levels,reflections,cladding", [
    (2, False, False), (4, False, False), (6, False, False), (9, True, False), (3, True, False), (14, True, False),
    (5, False, True), (8, False, True), (4, True, True), (9, True, True)])
def test_grouped_levels_give_the_single_rows(oracle, levels, reflections, cladding):
    """A range over every level of every point walks a point's levels together (1 to 13 layers, 2 to 14 levels, 1 or 5
    slices: 2 to 910 lines, every team width with every number of lines per lane); the same rows one by one (1 to 65
    lines) give the same bits, and the oracle's weights to the replays' 1e-5 for 99.9 % (5e-4 for all: a line that
    grazes an edge), with and without cladding triangles on the way."""
    from haseongpu_b200 import DeviceMesh, PrismMesh
    from haseongpu_b200.mesh import delaunay_triangles, disc_points, gaussian_pump_beta

    rng = np.random.default_rng(levels)
    pts = disc_points(0.8, 4, rng)
    tri = delaunay_triangles(pts)
    T = tri.shape[0]
    mesh = PrismMesh(points=pts, triangles=tri, numberOfLevels=levels, thickness=0.5 / levels,
                     betaVolume=gaussian_pump_beta(pts, tri, levels, 0.5 / levels), nTot=1.38e20, crystalTFluo=1e-3,
                     reflectivities=np.tile([0.3, 0.9], (T, 1)), refractiveIndices=[1.83, 1.0, 1.5, 1.0])
    if cladding:
        mesh.claddingCellTypes = (np.arange(T) % 4 == 1).astype(np.uint32)
        mesh.claddingNumber, mesh.claddingAbsorption = 1, 5.5
    spectrum = ([1.1e-21], [2.2e-20])
    S = mesh.numberOfSamples
    with DeviceMesh(mesh, *spectrum) as ctx:
        every = ctx.importance_weights(0, S, reflections)
        picks = [0, pts.shape[0] - 1, S // 2, S - 1]
        for s in picks:
            np.testing.assert_array_equal(ctx.importance_weights(s, 1, reflections)[0], every[s])
        part = ctx.importance_weights(3, S - 7, reflections)
        np.testing.assert_array_equal(part, every[3:S - 4])
    for s in picks:
        ref = np.asarray(oracle.importance(mesh, spectrum, s, slices=5 if reflections else 1), float).ravel()
        ref = ref / ref.max()
        big = ref > 1e-6
        rel = np.abs(every[s][big] / ref[big] - 1.0)
        # lines that graze the border of the cladding, at 20 times the contrast in g, are more than one in a thousand
        assert np.quantile(rel, 0.9 if cladding else 0.999) < 1e-5 and rel.max() < 5e-4


def _square(n, rng=None):
    """n x n points on a square, two triangles per cell, one layer."""
    from haseongpu_b200 import PrismMesh

    x = np.linspace(-1.0, 1.0, n)
    pts = np.column_stack([np.tile(x, n), np.repeat(x, n)])
    i = (np.arange(n - 1)[:, None] * n + np.arange(n - 1)[None]).ravel()
    tri = np.concatenate([np.column_stack([i, i + 1, i + n]), np.column_stack([i + 1, i + n + 1, i + n])]).astype(np.uint32)
    beta = 0.1 + 0.2 * np.cos(np.arange(tri.shape[0]))**2
    return PrismMesh(points=pts, triangles=tri, numberOfLevels=2, thickness=0.1, betaVolume=beta, nTot=1.38e20,
                     crystalTFluo=1e-3)


def test_more_rows_than_a_grid_has_in_y():
    """66,049 points in one workspace: a grid has 65,535 blocks in y, so the rows past them are another launch; the same
    weights and estimates as in two ranges of fewer rows."""
    from haseongpu_b200 import DeviceMesh

    mesh = _square(257)
    Np, half = mesh.numberOfPoints, 40_000
    assert Np > 65_535
    kw = dict(minRays=32, rngSeed=3, workspaceBytes=64 << 30)
    with DeviceMesh(mesh, [1.1e-21], [2.2e-20]) as ctx:
        ctx.set_local_proposal(2)
        every = ctx.importance_weights(0, 2 * Np, False)
        np.testing.assert_array_equal(every[:half], ctx.importance_weights(0, half, False))
        np.testing.assert_array_equal(every[2 * Np - half:], ctx.importance_weights(2 * Np - half, half, False))
        whole = ctx.calc_phi_ase(maxSample=Np - 1, **kw)
        parts = [ctx.calc_phi_ase(minSample=a, maxSample=b, **kw) for a, b in ((0, half - 1), (half, Np - 1))]
    assert np.all(np.isfinite(every)) and np.all(every.max(axis=1) == 1.0)
    for k in ("phiAse", "relativeStandardError", "totalRays", "droppedRays"):
        np.testing.assert_array_equal(getattr(whole, k), np.concatenate([getattr(p, k) for p in parts]))


@pytest.mark.parametrize("reflections", [False, True])
def test_lines_of_no_length_and_no_place(oracle, reflections):
    """A triangle smaller than an FP32 spacing has its centroid on its own vertices: its prisms are straight above and
    below those samples, and their weights are the oracle's (3e-4: positions rounded by up to 4e-6, 0.1 apart, squared).  A
    point that no triangle uses and that is nowhere (NaN, inf) has no weights and leaves the other samples' alone."""
    from haseongpu_b200 import DeviceMesh

    mesh = _square(5)
    mesh.points = mesh.points + 100.0
    a, b, c = mesh.triangles[7].astype(int)
    A, B, C = mesh.points[a], mesh.points[b], mesh.points[c]
    p1, p2 = (A + 1e-6 * (x * (B - A) + y * (C - A)) for x, y in ((0.6, 0.2), (0.2, 0.6)))
    i, j = len(mesh.points), len(mesh.points) + 1
    mesh.points = np.vstack([mesh.points, p1, p2])
    more = np.array([[a, i, j], [a, b, i], [b, c, i], [i, c, j], [a, j, c]], np.uint32)
    mesh.triangles = np.vstack([mesh.triangles[:7], mesh.triangles[8:], more])
    T = mesh.triangles.shape[0]
    layers = 4
    mesh.numberOfLevels = layers + 1
    mesh.betaVolume = np.random.default_rng(3).uniform(0.05, 0.3, T * layers)
    mesh.reflectivities = np.tile([0.3, 0.9], (T, 1))
    mesh.refractiveIndices = np.array([1.83, 1.0, 1.83, 1.0])
    tiny = T - 5
    cen = mesh.points[mesh.triangles[tiny]].astype(np.float32)
    assert np.all(cen == np.float32(mesh.points[a]))
    spectrum, slices = ([1.1e-21], [2.2e-20]), 5 if reflections else 1
    Np = mesh.numberOfPoints
    with DeviceMesh(mesh, *spectrum) as ctx:
        for pt in (a, i, j):
            for level in (0, 2, layers):
                w = ctx.importance_weights(level * Np + pt, 1, reflections)[0].astype(np.float64)
                ref = np.asarray(oracle.importance(mesh, spectrum, level * Np + pt, slices=slices), float).ravel()
                at = (np.arange(slices * layers) * T + tiny)
                assert np.all(np.isfinite(w))
                np.testing.assert_allclose(w[at] / w.max(), ref[at] / ref.max(), rtol=3e-4)
        plain = ctx.importance_weights(0, layers + 1, reflections)
    for nowhere in (np.nan, np.inf):
        mesh.points = np.vstack([mesh.points[:Np], [[nowhere, 0.0]]])
        with DeviceMesh(mesh, *spectrum) as ctx:
            w = ctx.importance_weights(Np, 1, reflections)[0]
            assert not np.any(np.isfinite(w) & (w > 0))
            if np.isnan(nowhere):
                np.testing.assert_array_equal(ctx.importance_weights(0, layers + 1, reflections), plain)


@pytest.mark.parametrize("field", ["uniform", "pumped"])
def test_gain_of_few_levels_beside_much_gain_in_height(oracle, field):
    """Lines across one to four of 60 levels, in a medium whose gain over its height is e^50: their integral is a
    difference of table entries that must not carry the rounding of the whole height's (2e-6 of ln w rms with entries of
    that size).  Of ln w, up to 20, an FP32 sum over the path keeps 4e-7 rms."""
    from haseongpu_b200 import DeviceMesh, PrismMesh
    from haseongpu_b200.mesh import delaunay_triangles, disc_points

    rng = np.random.default_rng(5)
    pts = disc_points(0.3, 6, rng)
    tri = delaunay_triangles(pts)
    T, Np, layers, h = tri.shape[0], pts.shape[0], 60, 0.02
    z = (np.arange(layers) + 0.5) / layers
    beta = 0.3 * (np.ones(layers) if field == "uniform" else 0.4 + np.exp(-2.0 * z))
    mesh = PrismMesh(points=pts, triangles=tri, numberOfLevels=layers + 1, thickness=h,
                     betaVolume=np.repeat(beta, T) * rng.uniform(0.95, 1.05, T * layers if field == "pumped" else 1),
                     nTot=6e21, crystalTFluo=1e-3)
    spectrum = ([1.1e-21], [2.2e-20])
    err = []
    with DeviceMesh(mesh, *spectrum) as ctx:
        for s in (5 * Np + 3, 30 * Np + 60, 59 * Np + 100):
            w = ctx.importance_weights(s, 1, False)[0].astype(np.float64).reshape(layers, T)
            ref = np.asarray(oracle.importance(mesh, spectrum, s, slices=1), float).reshape(layers, T)
            ls = s // Np
            near = np.abs(np.arange(layers) + 0.5 - ls) < 4
            ok = (w[near] > 1e-36) & (ref[near] > 0)
            d = np.log(w[near][ok]) - np.log(ref[near][ok])
            err.append(d - np.median(d))  # the normalisation is another line's
    err = np.concatenate(err)
    err = err[np.abs(err) < np.quantile(np.abs(err), 0.99)]  # lines that graze an edge
    assert err.size > 1500
    rms = np.sqrt((err * err).mean())
    print("rms", field, rms)
    assert rms < 1.8e-6, rms
