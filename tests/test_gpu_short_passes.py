"""Tables and passes whose launches were merged or moved to the device, at the sizes where they can go wrong: the
forward method's source table with empty cells at its ends, the end of a reflection chain, the training step's images
and group statistics."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ball(pattern):
    from haseongpu_b200 import TetMesh

    mesh = TetMesh.ball(1.0, 4, 0.1, 1e20, 1e-3)
    beta = np.random.default_rng(2).uniform(0.05, 0.3, mesh.numberOfCells)
    if pattern == "empty_ends":
        beta[:40] = 0.0
        beta[-40:] = 0.0
    elif pattern == "one_source":
        beta[:] = 0.0
        beta[77] = 0.2
    elif pattern == "cladding":
        mesh.claddingCellTypes = (np.arange(mesh.numberOfCells) % 5 == 0).astype(np.uint32)
        mesh.claddingNumber, mesh.claddingAbsorption = 1, 5.5
    elif pattern == "last_cell":
        beta[:] = 0.0
        beta[-1] = 0.2
    return mesh.withBeta(beta)


@pytest.mark.parametrize("pattern", ["dense", "empty_ends", "one_source", "last_cell", "cladding"])
def test_source_table_draws_the_oracle_cells(oracle, pattern):
    """The guide table built on the device starts the oracle's rays: visits equal, phi to a few float ulps (the replay
    level); beta handed over after the context was made with another one."""
    from haseongpu_b200 import TetDeviceMesh

    mesh = _ball(pattern)
    spectrum = ([1e-21], [2e-20])
    ref = oracle.forward_phi_ase(mesh, spectrum, minRays=20_000, seed=3)
    with TetDeviceMesh(mesh.withBeta(np.full(mesh.numberOfCells, 0.1)), *spectrum) as ctx:
        ctx.update_beta(mesh.betaVolume)
        dev = ctx.calc_phi_ase(forwardRayCount=20_000, rngSeed=3)
        for bad, text in ((np.nan, "betaVolume[5] is not finite"), (np.inf, "betaVolume[5] is not finite"),
                          (-0.1, "betaVolume[5] is negative")):
            beta = mesh.betaVolume.copy()
            beta[5:9] = bad
            with pytest.raises(RuntimeError, match=text.replace("[", r"\[").replace("]", r"\]")):
                ctx.update_beta(beta)
        again = ctx.calc_phi_ase(forwardRayCount=20_000, rngSeed=3)
    assert (dev.totalRays != ref["rayVisits"]).mean() < 2e-3
    live = ref["phiAse"] > 0
    rel = np.abs(dev.phiAse[live] / ref["phiAse"][live] - 1.0)
    assert np.quantile(rel, 0.999) < 1e-5
    np.testing.assert_array_equal(again.totalRays, dev.totalRays)  # a refused beta changes nothing


@pytest.mark.parametrize("limit", [1, 2, 3, 40])
@pytest.mark.parametrize("reflectivity", [0.0, 0.05, 0.6])
def test_reflection_chains_end_where_the_oracle_ends_them(oracle, limit, reflectivity):
    from haseongpu_b200 import TetDeviceMesh

    mesh = _ball("dense").withReflectingBoundary(reflectivity)
    spectrum = ([1e-21], [2e-20])
    kw = dict(useReflections=True, reflectionMaxIterations=limit, surfaceReservoirSize=64)
    ref = oracle.forward_phi_ase(mesh, spectrum, minRays=4_000, seed=7, **kw)
    with TetDeviceMesh(mesh, *spectrum) as ctx:
        dev = ctx.calc_phi_ase(forwardRayCount=4_000, rngSeed=7, **kw)
        two = ctx.calc_phi_ase(forwardRayCount=4_000, rngSeed=7, **kw)
    assert (dev.srmStatus, dev.srmPasses) == (ref["srmStatus"], ref["srmPasses"])
    assert (two.srmStatus, two.srmPasses) == (dev.srmStatus, dev.srmPasses)


@pytest.mark.parametrize("steps", [1, 2, 5])
def test_training_leaves_the_images_of_its_parameters(steps):
    """The network a training call leaves behind computes what a network given the same parameters computes."""
    from haseongpu_b200.proposal import ProposalNet

    rng = np.random.default_rng(4)
    off = np.array([0, 300, 700, 1000], np.uint32)
    f = rng.normal(size=(1000, 12)).astype(np.float32)
    t = rng.random(1000).astype(np.float32)
    with ProposalNet(seed=2) as a, ProposalNet(seed=5) as b:
        a.train(off, f, t, steps=steps, groups_per_step=2, learning_rate=1e-2)
        b.params = a.params
        np.testing.assert_array_equal(a.forward(f), b.forward(f))
        la, ga = a.loss_grad(off, f, t)
        lb, gb = b.loss_grad(off, f, t)
    assert la == pytest.approx(lb, rel=1e-6)  # FP32 sums of 1,000 terms in another order
    np.testing.assert_allclose(ga, gb, atol=1e-5 * np.abs(gb).max())


@pytest.mark.parametrize("sizes", [[1], [31, 33], [1023, 1024, 1025], [2048, 0, 3], [5000]])
def test_group_statistics_at_block_edges(sizes):
    """The loss of groups around the statistics kernel's block and warp sizes, from the device's own logits in FP64:
    FP32 sums of up to 5,000 terms and exponentials of 2 ulp, 1e-5."""
    from haseongpu_b200.proposal import ProposalNet

    rng = np.random.default_rng(sum(sizes))
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    f = rng.normal(size=(off[-1], 12)).astype(np.float32)
    t = (rng.random(off[-1]) ** 3).astype(np.float32)
    with ProposalNet(seed=8) as net:
        logits = net.forward(f).astype(np.float64)
        loss, _ = net.loss_grad(off, f, t)
    ref = 0.0
    for a, b in zip(off[:-1], off[1:]):
        if b > a and t[a:b].sum() > 0:
            l, y = logits[a:b], t[a:b].astype(np.float64)
            lse = np.log(np.exp(l - l.max()).sum()) + l.max()
            ref += (lse - (y * l).sum() / y.sum()) / len(sizes)
    assert loss == pytest.approx(ref, rel=1e-5, abs=1e-5)


@pytest.mark.parametrize("rings,levels,streamed", [(3, 2, False), (9, 9, False), (9, 10, True)])
@pytest.mark.parametrize("tally", ["global", "shared"])
def test_cell_records_read_either_way(oracle, rings, levels, streamed, tally):
    """Meshes below and above the 12,000 cells from which the records are read without allocating L1 lines start and walk
    the oracle's rays: visits equal, phi to a few float ulps (the replay level)."""
    from haseongpu_b200 import PrismMesh, TetDeviceMesh, TetMesh
    from haseongpu_b200.mesh import delaunay_triangles, disc_points

    rng = np.random.default_rng(rings)
    pts = disc_points(1.0, rings, rng)
    tri = delaunay_triangles(pts)
    T = tri.shape[0]
    mesh = TetMesh.fromPrismMesh(PrismMesh(points=pts, triangles=tri, numberOfLevels=levels, thickness=0.7 / (levels - 1),
                                           betaVolume=rng.uniform(0.05, 0.3, T * (levels - 1)), nTot=1e20,
                                           crystalTFluo=1e-3))
    assert (mesh.numberOfCells > 12_000) == streamed
    spectrum = ([1e-21], [2e-20])
    ref = oracle.forward_phi_ase(mesh, spectrum, minRays=20_000, seed=3)
    with TetDeviceMesh(mesh, *spectrum) as ctx:
        dev = ctx.calc_phi_ase(forwardRayCount=20_000, rngSeed=3, tallyMode=tally)
    assert (dev.totalRays != ref["rayVisits"]).mean() < 2e-3
    live = ref["phiAse"] > 0
    rel = np.abs(dev.phiAse[live] / ref["phiAse"][live] - 1.0)
    assert np.quantile(rel, 0.999) < 1e-5
