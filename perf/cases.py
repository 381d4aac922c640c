"""What the framework is timed on: the phi-ASE work its users have it do, through the public entry points.

The media are the seeded discs of this repository's own configurations (concentric rings, Delaunay, extruded to
levels; pump-shaped beta with noise), from a few hundred prisms to half a million.  A case's geometry follows from
its numbers, its beta (or training rows) from the seed.  ``exact`` restates the estimators in 64 bits: the prism walk,
the ray map and Philox4x32-10 for the backward method, the Tet4 walk for the forward method, autograd and Adam for
the proposal network.
"""

from __future__ import annotations

import math
from functools import lru_cache

import numpy as np
import torch

from haseongpu_b200 import DeviceMesh, MediaBatch, PrismMesh, TetDeviceMesh, TetMesh
from haseongpu_b200.learned import pump_field
from haseongpu_b200.mesh import delaunay_triangles, disc_points, point_beta
from haseongpu_b200.proposal import ProposalNet
from haseongpu_b200.spectra import CrossSectionData, two_lorentzian_spectrum

N_TOT, TAU = 1.38e20, 9.41e-4
RNG_SEED = 5489  # the entry points' default Philox key


# ------------------------------------------------------------------ cases ----
def listed() -> list:
    return [
        # one query of a few sample points on a small cladded crystal: an interactive caller; launches and host work count
        dict(name="query", kind="solve", proposal="walks", rings=6, levels=5, lambdas=1, reflect=False, cladding=True,
             samples=5, rays=10_000, max_rays=10_000),
        # the whole small disc, one wavelength, adaptive to 0.5 % error: the everyday monochromatic solve
        dict(name="disc_mono", kind="solve", proposal="walks", rings=13, levels=10, lambdas=1, reflect=False,
             cladding=False, samples=0, rays=100_000, max_rays=1_000_000),
        # a block of the large disc's samples, full spectrum, reflecting surfaces: the expensive exact weights
        dict(name="disc_poly", kind="solve", proposal="walks", rings=29, levels=20, lambdas=16, reflect=True,
             cladding=False, samples=256, rays=100_000, max_rays=100_000),
        # the same physics with the walk-free weights, a larger block per call
        dict(name="disc_poly_grid", kind="solve", proposal="grid", rings=29, levels=20, lambdas=16, reflect=True,
             cladding=False, samples=512, rays=100_000, max_rays=100_000),
        # a new pump field solved with a trained proposal network (a fit or a design loop calls this per field)
        dict(name="disc_learned", kind="solve", proposal="learned", rings=13, levels=10, lambdas=1, reflect=False,
             cladding=False, samples=2735, rays=100_000, max_rays=100_000),
        # one step's ASE on the finest mesh: few rays for many samples, local proposal
        dict(name="pulse_local", kind="solve", proposal="local", rings=40, levels=30, lambdas=8, reflect=True,
             cladding=False, samples=8192, rays=2_000, max_rays=2_000),
        # a design sweep: media of different sizes in one batched, adaptive solve
        dict(name="media_batch", kind="batch", media=12, rings=8, levels=7, lambdas=4, reflect=False, cladding=True,
             samples=48, rays=10_000, max_rays=100_000),
        # the forward Tet4 method on the large disc's twin (the reference's current method): the largest tables
        dict(name="tet_poly", kind="forward", rings=29, levels=20, lambdas=16, reflect=False, cladding=False,
             rays=4_000_000),
        # the forward method with surface reflections on a small mesh: many short passes
        dict(name="tet_reflect", kind="forward", rings=18, levels=10, lambdas=4, reflect=True, cladding=True,
             rays=5_000),
        # fine-tuning the proposal network between two solves
        dict(name="train", kind="train", groups=24, rows=9126, groups_per_step=8, steps=20),
        # one medium's training rows: contributions logged per prism, and the features of the same pairs
        dict(name="log_rows", kind="log", rings=13, levels=10, lambdas=4, reflect=False, cladding=False, samples=32,
             rays=100_000),
        # a pump pulse, a few steps of the rate equations with the backward method at every sample point
        dict(name="time_steps", kind="time", rings=11, levels=8, lambdas=8, reflect=True, cladding=False, rays=4_000,
             steps=3),
    ]


def _log_int(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["solve"] * 5 + ["batch", "forward", "forward", "train", "log", "time"])
    lambdas = rng.choice([1, 1, 2, 4, 8, 16])
    reflect, cladding = rng.random() < 0.5, rng.random() < 0.35
    if kind == "solve":
        proposal = rng.choice(["walks", "walks", "grid", "learned", "local"])
        rings = rng.randint(5, 13) if proposal == "learned" else rng.randint(20, 40) if proposal == "local" else rng.randint(5, 29)
        levels = rng.randint(4, 30 if proposal == "local" else 20)
        rays = _log_int(rng, 2_000, 100_000)
        entries = 6 * rings * rings * (levels - 1) * (5 if reflect else 1)
        # lines to weigh and rays to walk of one call stay within the listed cases'
        most = int(min(1.2e8 / entries if proposal != "local" else 8192, 5e7 / rays, (3 * rings * rings) * levels))
        return dict(kind=kind, proposal=proposal, rings=rings, levels=levels, lambdas=lambdas, reflect=reflect,
                    cladding=cladding, samples=_log_int(rng, 1, max(1, most)), rays=rays, max_rays=rays)
    if kind == "batch":
        return dict(kind=kind, media=rng.randint(2, 12), rings=rng.randint(5, 9), levels=rng.randint(4, 10),
                    lambdas=lambdas, reflect=reflect, cladding=cladding, samples=_log_int(rng, 4, 48),
                    rays=_log_int(rng, 2_000, 10_000), max_rays=100_000)
    if kind == "forward":
        # with reflections: few enough rays that no face's reservoir overflows (an overflow's survivors are not reproducible)
        rings = rng.randint(14, 18) if reflect else rng.randint(6, 29)
        return dict(kind=kind, rings=rings, levels=rng.randint(4, 14), lambdas=lambdas, reflect=reflect, cladding=cladding,
                    rays=_log_int(rng, 500, 12 * rings * rings) if reflect else _log_int(rng, 100_000, 4_000_000))
    if kind == "train":
        groups = rng.randint(4, 24)
        return dict(kind=kind, groups=groups, rows=_log_int(rng, 300, 9_126), groups_per_step=rng.randint(1, min(8, groups)),
                    steps=rng.randint(5, 20))
    if kind == "log":
        return dict(kind=kind, rings=rng.randint(5, 13), levels=rng.randint(4, 12), lambdas=lambdas, reflect=False,
                    cladding=cladding, samples=_log_int(rng, 4, 32), rays=_log_int(rng, 10_000, 100_000))
    return dict(kind=kind, rings=rng.randint(5, 11), levels=rng.randint(4, 8), lambdas=lambdas, reflect=reflect,
                cladding=cladding, rays=_log_int(rng, 1_000, 4_000), steps=rng.randint(2, 3))


# ----------------------------------------------------------------- inputs ----
@lru_cache(maxsize=32)
def _geometry(rings: int, levels: int, radius: float):
    rng = np.random.default_rng([20261203, rings, levels])
    pts = disc_points(radius, rings, rng)
    return pts, delaunay_triangles(pts)


def _spectra(lambdas: int) -> CrossSectionData:
    if lambdas == 1:
        return CrossSectionData.monochromatic(wavelength=1030e-9, crossSectionAbsorption=1.1e-21,
                                              crossSectionEmission=2.2e-20)
    return two_lorentzian_spectrum(lambdas)


def _mesh(case: dict, rng: np.random.Generator, radius: float = 1.0) -> PrismMesh:
    """The case's disc, 0.7 cm high, with a seeded pump field; the outer ring is cladding if the case has one."""
    rings, levels = case["rings"], case["levels"]
    pts, tri = _geometry(rings, levels, radius)
    h = 0.7 / (levels - 1)
    T = tri.shape[0]
    mesh = PrismMesh(points=pts, triangles=tri, numberOfLevels=levels, thickness=h,
                     betaVolume=np.zeros(T * (levels - 1)), nTot=N_TOT, crystalTFluo=TAU,
                     betaCells=point_beta(pts, levels, h), name=f"disc{rings}x{levels}")
    if case.get("cladding"):
        r = np.linalg.norm(pts[tri].mean(axis=1), axis=1)
        mesh.claddingCellTypes = (r > 0.85 * radius).astype(np.uint32)
        mesh.claddingNumber, mesh.claddingAbsorption = 1, 5.5
    if case.get("reflect"):
        mesh.reflectivities = np.tile([0.3, 0.9], (T, 1))
        mesh.refractiveIndices = np.array([1.83, 1.0, 1.83, 1.0])
    mesh.betaVolume = pump_field(mesh, rng)
    return mesh


def _block(mesh, samples: int):
    """A block of consecutive sample points from the middle of the mesh (0: every one)."""
    S = mesh.numberOfSamples
    if samples == 0 or samples >= S:
        return 0, S - 1
    first = (S - samples) // 2
    return first, first + samples - 1


def _network(rng) -> np.ndarray:
    """Parameters of a proposal network that carries ln(beta V / d^2) + ln gain (features 9 and 8) to the logit through
    its three SiLU layers (silu(x) - silu(-x) = x), plus small seeded weights everywhere else, as training leaves them."""
    w1, w2, w3, w4 = (rng.normal(0, 0.02, s) for s in ((12, 64), (64, 64), (64, 64), (64,)))
    w1[:, :2] *= 0.1
    w1[8:10, 0] += 1.0
    w1[8:10, 1] -= 1.0
    for w in (w2, w3):
        w[0, 0], w[1, 0], w[0, 1], w[1, 1] = 1.0, -1.0, -1.0, 1.0
    w4[0], w4[1] = 1.0, -1.0
    z = np.zeros(64)
    return np.concatenate([w1.ravel(), z, w2.ravel(), z, w3.ravel(), z, w4, [0.0]]).astype(np.float32)


def _training_rows(case, rng):
    """Feature rows and logged contributions of `groups` sample points, in the ranges the feature kernel gives."""
    n, G = case["rows"], case["groups"]
    sizes = [n - int(rng.integers(0, max(1, n // 8))) for _ in range(G)]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint32)
    R = int(off[-1])
    f = rng.uniform(-1.0, 1.0, (R, 12)).astype(np.float32)
    f[:, 2] = rng.uniform(0, 1, R)
    f[:, 6] = np.log(rng.uniform(0.02, 2.0, R))
    f[:, 7] = rng.uniform(0.02, 0.4, R)
    f[:, 8] = rng.uniform(-0.5, 1.5, R)
    f[:, 9] = np.log(f[:, 7]) - 2.0 * f[:, 6]
    f[:, 10] = 0.0
    f[:, 11] = 3.0
    t = np.exp(f[:, 8] + f[:, 9] + 0.3 * rng.standard_normal(R)).astype(np.float32)
    t[rng.random(R) < 0.2] = 0.0  # prisms that no logged ray started in
    return off, f, t


_PUMP = dict(peakIntensity=16e3, radius=0.6, exponent=40.0, centerX=0.0, centerY=0.0, wavelength=940e-9,
             sigmaA=0.8e-20, sigmaE=0.16e-20, retroreflect=True)


def prepare(case: dict, seed: int):
    """The contexts, weights and fields a user's program holds before the call."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "train":
        s["off"], s["features"], s["targets"] = _training_rows(case, rng)
        s["net"] = ProposalNet(seed=1)
        s["net"].params = _network(rng)
        return s
    sa, se = _spectra(case["lambdas"]).resampled()
    if kind == "batch":
        s["media"] = []
        for i in range(case["media"]):  # sizes and radii spread over the family
            sub = dict(case, rings=case["rings"] + i % 4, levels=case["levels"] + i % 3)
            mesh = _mesh(sub, rng, radius=0.6 + 0.2 * (i % 5))
            first, last = _block(mesh, case["samples"])
            s["media"].append((DeviceMesh(mesh, sa, se), first, last))
        s["batch"] = MediaBatch()
        return s
    mesh = _mesh(case, rng)
    s["mono"] = case["lambdas"] == 1
    if kind == "forward":
        twin = TetMesh.fromPrismMesh(mesh)
        s["ctx"], s["beta"] = TetDeviceMesh(twin, sa, se), twin.betaVolume
        return s
    ctx = s["ctx"] = DeviceMesh(mesh, sa, se)
    s["beta"] = mesh.betaVolume
    if kind == "time":
        return s
    s["first"], s["last"] = _block(mesh, case["samples"])
    proposal = case.get("proposal")
    if proposal == "grid":
        ctx.set_grid_proposal(True)
    elif proposal == "local":
        ctx.set_local_proposal(16, 0.9)
        ctx.calc_phi_ase(minRays=64, useReflections=case["reflect"], minSample=0, maxSample=0)  # the candidate tables
    elif proposal == "learned":
        s["net"] = ProposalNet(seed=1)
        s["net"].params = _network(rng)
    return s


# ------------------------------------------------------------------- run ----
def _fields(r) -> dict:
    return {k: getattr(r, k) for k in ("phiAse", "relativeStandardError", "dndtAse", "totalRays", "droppedRays")}


def _threshold(case) -> float:
    return 0.005 if case["max_rays"] > case["rays"] else 0.0


def run(s: dict):
    """One call as a user's program makes it; a program with a new field hands it over first."""
    case = s["case"]
    kind = case["kind"]
    if kind == "train":
        loss = s["net"].train(s["off"], s["features"], s["targets"], steps=case["steps"],
                              groups_per_step=case["groups_per_step"], learning_rate=1e-3)
        return {"loss": loss, "params": s["net"].params}
    if kind == "batch":
        outs, _ = s["batch"].solve(s["media"], minRays=case["rays"], maxRays=case["max_rays"], mseThreshold=0.005,
                                   useReflections=case["reflect"], adaptiveSteps=3, rngSeed=RNG_SEED)
        keys = _fields(outs[0])
        return {k: np.concatenate([_fields(o)[k] for o in outs]) for k in keys}
    ctx = s["ctx"]
    if kind == "forward":
        ctx.update_beta(s["beta"])
        return _fields(ctx.calc_phi_ase(forwardRayCount=case["rays"], monochromatic=s["mono"], rngSeed=RNG_SEED,
                                        useReflections=case["reflect"]))
    if kind == "time":
        ctx.update_beta(s["beta"])
        n = case["steps"]
        out = ctx.simulate(pump=_PUMP, time=dict(timeStep=20e-6, steps=n, pumpSteps=n, aseSteps=n, integrator=0),
                           minRays=case["rays"], useReflections=case["reflect"], monochromatic=s["mono"],
                           rngSeed=RNG_SEED)
        return {k: out[k] for k in ("betaVolume", "meanBeta", "meanPhi", "pumpAbsorbed")}
    opts = dict(useReflections=case["reflect"], monochromatic=s["mono"], rngSeed=RNG_SEED, minSample=s["first"],
                maxSample=s["last"])
    if kind == "log":
        ctx.update_beta(s["beta"])
        r, contributions = ctx.log_contributions(minRays=case["rays"], **opts)
        features = ctx.proposal_features(s["first"], s["last"] - s["first"] + 1, useReflections=case["reflect"],
                                         monochromatic=s["mono"])
        return dict(_fields(r), contributions=contributions, features=features)
    adaptive = dict(minRays=case["rays"], maxRays=case["max_rays"], mseThreshold=_threshold(case),
                    adaptiveSteps=4 if case["max_rays"] > case["rays"] else 0)
    if case["proposal"] == "learned":
        ctx.update_beta(s["beta"])
        return _fields(ctx.calc_phi_ase_learned(s["net"], **adaptive, **opts))
    if case["proposal"] != "walks":
        ctx.update_beta(s["beta"])
    return _fields(ctx.calc_phi_ase(**adaptive, **opts))


# ------------------------------------------------------------------ work ----
def _crossings(rings: int, levels: int, reflect: bool) -> float:
    """Prisms on the way of a ray: 2.2 triangle edges per edge length over a mean path of 0.6 radii, and its levels."""
    return 2.2 * rings * 0.6 + levels / 3.0 * (2.0 if reflect else 1.0)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "train":
        rows = case["rows"] * case["groups_per_step"]
        macs = 12 * 64 + 2 * 64 * 64 + 64
        return {"bytes": case["steps"] * rows * 13 * 4.0 + 2 * 9_100 * 4.0, "flops": case["steps"] * rows * 6.0 * macs}
    if kind == "batch":
        sub = [work(dict(case, kind="solve", proposal="walks", rings=case["rings"] + i % 4, levels=case["levels"] + i % 3))
               for i in range(case["media"])]
        return {k: sum(w[k] for w in sub) for k in ("bytes", "flops")}
    T, layers = 6 * case["rings"] ** 2, case["levels"] - 1
    points = 3 * case["rings"] ** 2 + 3 * case["rings"] + 1
    P, S = T * layers, points * case["levels"]
    cross = _crossings(case["rings"], case["levels"], case["reflect"])
    slices = 5 if case["reflect"] else 1
    if kind == "forward":
        passes = 8 if case["reflect"] else 1  # reflected passes of as many rays until the chain has decayed
        # per cell: three of four face coordinates and their rates, the exit, an exponential, four weights
        crossings = case["rays"] * passes * cross * 2.0
        return {"bytes": 3 * P * (128.0 + 8 + 28), "flops": crossings * 60.0}
    samples = S if kind == "time" or case["samples"] == 0 else min(case["samples"], S)
    solves = case["steps"] if kind == "time" else 1
    # per ray: its start (random words, point, direction) and 12 per crossing (exit edge, level plane, gain)
    flops = samples * case["rays"] * (60.0 + 12.0 * cross + 4.0 * (case["lambdas"] if case["lambdas"] > 1 else 0))
    entries = samples * (slices * layers * 16 if case.get("proposal") == "local" else slices * P)
    if case.get("proposal") == "learned":
        flops += entries * 2.0 * (12 * 64 + 2 * 64 * 64 + 64)
    elif case.get("proposal") == "grid":
        flops += entries * 30.0
    else:  # every line's gain: 3 per crossed prism
        flops += entries * 3.0 * cross
    data = T * 60.0 + P * 8.0 + samples * 32.0
    if kind == "log":
        data += entries * 13 * 4.0
    return {"bytes": data * solves, "flops": flops * solves}


def tolerance(case: dict):
    """Rounding of a weight in 32 bits moves a few of a sample's rays to the next prism, and the path of a ray that
    grazes an edge to its other side: a share of the sample's own statistical error, which grows as the rays get
    fewer, and the relative error's estimate, which hangs on the largest contributions, most of all (against 64 bits:
    phi 2e-6 to 6e-4, its error's estimate 4e-6 at 1e5 rays without reflections, 1.2e-3 with, 1.7e-2 at 7e3)."""
    kind = case["kind"]
    if kind == "train":  # 16-bit operands; Adam's steps have the learning rate's size whatever the gradient's: 1e-3 twice
        return {"rel": 5e-3, "max": 0.4}
    if kind == "forward":  # 64-bit walk, phi rounded to 32 bits; a moved ray's reflections all move with it
        return {"rel": 1e-4, "max": 0.05, "differ": 0.01} if case["reflect"] else {"rel": 2e-7, "max": 1e-5, "differ": 1e-3}
    if kind == "time":  # beta after a few steps: the mean over many samples
        return {"rel": 1e-3, "max": 0.05}
    scale = math.sqrt(1e5 / case["rays"])
    if kind == "log":  # a moved ray's contribution is logged for the other prism: 7e-4 of the contributions at 1e5 rays
        return {"rel": min(0.03, 3e-3 * scale), "max": 0.9, "differ": 1e-3}
    rel = min(0.03, 5e-3 * scale)
    # batch: samples near the threshold may stop a pass earlier or later
    return {"rel": rel, "max": min(0.9, 10 * rel), "differ": 0.01 if case["max_rays"] > case["rays"] else 0.0}


# ----------------------------------------------------------------- exact ----
_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_F = dict(dtype=torch.float64, device=_DEV)
_I = dict(dtype=torch.int64, device=_DEV)
_M32 = 0xFFFFFFFF


def _mul32(a, b: int):
    """(high, low) words of a * b, a an int64 tensor of 32-bit words."""
    al, ah = a & 0xFFFF, a >> 16
    lo, hi = al * b, ah * b
    mid = hi + (lo >> 16)
    return mid >> 16, ((mid & 0xFFFF) << 16) | (lo & 0xFFFF)


def _philox(c0, c1, c2, c3, k0: int, k1: int):
    """Philox4x32-10 (Salmon et al., SC'11) on broadcast int64 tensors of 32-bit words."""
    c = list(torch.broadcast_tensors(*(torch.as_tensor(x, **_I) for x in (c0, c1, c2, c3))))
    for _ in range(10):
        h0, l0 = _mul32(c[0], 0xD2511F53)
        h1, l1 = _mul32(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return c


def _unit(x):
    return ((x >> 8).double() + 0.5) / 16777216.0


class _Prisms:
    """The prism mesh in 64 bits: outward edge lines, neighbours, centroids, areas."""

    def __init__(self, mesh: PrismMesh, sa, se):
        p, tri = mesh.points, mesh.triangles.astype(np.int64)
        T = tri.shape[0]
        v = p[tri]
        e = np.roll(v, -1, axis=1) - v
        cross = e[:, 0, 0] * -e[:, 2, 1] + e[:, 0, 1] * e[:, 2, 0]
        n = np.stack([e[..., 1], -e[..., 0]], -1) / np.linalg.norm(e, axis=-1, keepdims=True) * np.sign(cross)[:, None, None]
        a, b = tri, np.roll(tri, -1, axis=1)
        key = (np.minimum(a, b) * p.shape[0] + np.maximum(a, b)).ravel()
        order = np.argsort(key, kind="stable")
        same = key[order][1:] == key[order][:-1]
        nbr = np.full(3 * T, -1, np.int64)
        i, j = order[:-1][same], order[1:][same]
        nbr[i], nbr[j] = j, i
        self.n, self.c = torch.tensor(n, **_F), torch.tensor((n * v).sum(-1), **_F)
        self.nbr = torch.tensor(nbr.reshape(T, 3), **_I)
        self.v, self.tri = torch.tensor(v, **_F), torch.tensor(tri, **_I)
        self.cen, self.area = torch.tensor(v.mean(1), **_F), torch.tensor(0.5 * np.abs(cross), **_F)
        self.points = torch.tensor(p, **_F)
        self.T, self.layers, self.h, self.Np = T, mesh.numberOfLevels - 1, mesh.thickness, p.shape[0]
        self.beta = torch.tensor(mesh.betaVolume, **_F)
        clad = np.zeros(T, bool) if mesh.claddingCellTypes is None else mesh.claddingCellTypes == mesh.claddingNumber
        self.clad, self.abs = torch.tensor(np.tile(clad, self.layers), device=_DEV), mesh.claddingAbsorption
        self.A, self.B = N_TOT * (np.asarray(se) + np.asarray(sa)), N_TOT * np.asarray(sa)
        self.sa, self.se = np.max(sa), np.max(se)
        self.betaCells = mesh.betaCells
        self.R = None if mesh.reflectivities is None else torch.tensor(mesh.reflectivities, **_F)
        r = (1.0, 1.0) if mesh.refractiveIndices is None else (mesh.refractiveIndices[1] / mesh.refractiveIndices[0],
                                                               mesh.refractiveIndices[3] / mesh.refractiveIndices[2])
        self.tir = torch.tensor([1.0 - x * x if x < 1.0 else -1.0 for x in r], **_F)

    def image(self, ls, j):
        L = self.layers
        return torch.where(j == 1, -ls, torch.where(j == 2, 2 * L - ls, torch.where(j == 3, ls - 2 * L,
                           torch.where(j == 4, ls + 2 * L, ls))))

    def walk(self, S, kimg, j, t, layer, d, A: float, B: float):
        """From the start points (offset d from the image points) to the sample points: the integral of g = beta A - B
        plus the logarithm of the bounces' factors, of beta, and of the cladding's length along the way."""
        N = t.numel()
        D = d.norm(dim=1)
        u = d / D[:, None]
        G, Jb, Lc = torch.zeros(N, **_F), torch.zeros(N, **_F), torch.zeros(N, **_F)
        step = torch.where(u[:, 2] > 0, -1, 1)
        at = dict(i=torch.arange(N, device=_DEV), S=S, k=kimg, t=t, l=layer, s=D.clone(), u=u, step=step,
                  plane=torch.where(u[:, 2] > 0, layer, layer + 1) - kimg,
                  left=torch.where(j == 0, 0, torch.where(j <= 2, 1, 2)), entry=torch.full((N,), -1, **_I))
        done = torch.zeros(N, dtype=torch.bool, device=_DEV)
        for _ in range(10000):
            if not at["i"].numel():
                break
            t, s, u = at["t"], at["s"], at["u"]
            n = self.n[t]
            den = -(n[..., 0] * u[:, 0:1] + n[..., 1] * u[:, 1:2])
            num = n[..., 0] * at["S"][:, 0:1] + n[..., 1] * at["S"][:, 1:2] - self.c[t]
            ok = (den > 0) & (self.nbr[t] >= 0) & (torch.arange(3, device=_DEV) != at["entry"][:, None])
            cut = torch.where(ok, num / torch.where(ok, den, torch.ones_like(den)), torch.full_like(den, -1.0))
            se, e = cut.max(dim=1)
            sz = at["plane"].double() * self.h / u[:, 2]
            nxt = torch.minimum(torch.maximum(torch.maximum(se, sz), torch.zeros_like(s)), s)
            end = nxt <= 1e-12
            nxt = torch.where(end, torch.zeros_like(nxt), nxt)
            p = at["l"] * self.T + t
            cl = self.clad[p]
            seg = s - nxt
            g = torch.where(cl, torch.full_like(s, -self.abs), self.beta[p] * A - B)
            G.index_add_(0, at["i"], g * seg)
            Jb.index_add_(0, at["i"], torch.where(cl, torch.zeros_like(s), self.beta[p] * seg))
            Lc.index_add_(0, at["i"], torch.where(cl, seg, torch.zeros_like(s)))
            onplane = ~end & (sz >= se)
            l2 = at["l"] + at["step"]
            surf = onplane & ((l2 < 0) | (l2 >= self.layers))
            late = end & (at["left"] > 0)  # a bounce at the sample point itself
            f = surf & (at["left"] > 0) | late
            if bool(f.any()):
                which = (l2[f] >= 0).long()
                fac = self.R[t[f], which] if self.R is not None else torch.zeros(int(f.sum()), **_F)
                fac = torch.where(u[f, 2] ** 2 <= self.tir[which], torch.ones_like(fac), fac)
                G.index_add_(0, at["i"][f], torch.log(fac))
            lost = surf & (at["left"] <= 0)
            done[at["i"][end]] = True
            at["left"] = at["left"] - surf.long()
            at["step"] = torch.where(surf, -at["step"], at["step"])
            at["l"] = torch.where(onplane & ~surf, l2, at["l"])
            at["plane"] = at["plane"] + torch.where(onplane, torch.where(u[:, 2] > 0, -1, 1), 0)
            code = self.nbr[t, e]
            over = ~end & ~onplane
            at["t"] = torch.where(over, code // 3, t)
            at["entry"] = torch.where(over, code % 3, at["entry"])
            at["s"] = nxt
            keep = ~end & ~lost
            at = {k: v[keep] for k, v in at.items()}
        return D, G, Jb, Lc, done

    def weights(self, samples, slices: int):
        """ln w of every (slice, prism) of the samples: the straight line from the prism's centre."""
        P = self.T * self.layers
        x = torch.arange(slices * P, **_I)
        j, p = x // P, x % P
        l, t = p // self.T, p % self.T
        out = []
        for s in samples.tolist():
            S, ls = self.points[s % self.Np], s // self.Np
            k = self.image(torch.full_like(j, ls), j)
            d = torch.cat([self.cen[t] - S, ((l - k).double() + 0.5)[:, None] * self.h], dim=1)
            D, G, _, _, done = self.walk(S.expand(x.numel(), 2), k, j, t, l, d, float(self.A.mean()), float(self.B.mean()))
            w = torch.log(self.beta[p] * self.area[t] * self.h) - 2 * torch.log(D) + G
            out.append(torch.where(done & (self.beta[p] > 0), w, torch.full_like(w, -math.inf)))
        return torch.stack(out)

    def start(self, S, pS, k, t, l, rnd):
        """Start points: uniform in the prism, or by direction and distance in a prism that touches the image point.
        Returns the offsets from the image point and the ray's weight without q."""
        w0, w1 = rnd[0] >> 8, rnd[1] >> 8
        flip = w0 + w1 + 1 > (1 << 24)
        u1 = (torch.where(flip, (1 << 24) - 1 - w0, w0).double() + 0.5) / 16777216.0
        u2 = (torch.where(flip, (1 << 24) - 1 - w1, w1).double() + 0.5) / 16777216.0
        v = self.v[t]
        xy = v[:, 0] + u1[:, None] * (v[:, 1] - v[:, 0]) + u2[:, None] * (v[:, 2] - v[:, 0])
        d = torch.cat([xy - S, (((l - k).double() + _unit(rnd[2])) * self.h)[:, None]], dim=1)
        wf = self.area[t] * self.h / (d * d).sum(1)
        corner = self.tri[t] == pS[:, None]
        near = ((l == k) | (l + 1 == k)) & corner.any(1)
        if bool(near.any()):
            q = torch.nonzero(near)[:, 0]
            iv = corner[q].long().argmax(1)
            vv, Sq = v[q], S[q]
            r = torch.arange(q.numel(), device=_DEV)
            e1, e2 = vv[r, (iv + 1) % 3] - Sq, vv[r, (iv + 2) % 3] - Sq
            e1, e2 = e1 / e1.norm(dim=1, keepdim=True), e2 / e2.norm(dim=1, keepdim=True)
            ca = (e1 * e2).sum(1).clamp(-1, 1)
            alpha = torch.acos(ca)
            az = _unit(rnd[0][q]) * alpha
            b2 = torch.sin(az) / torch.sin(alpha)
            c = (torch.cos(az) - ca * b2)[:, None] * e1 + b2[:, None] * e2
            el = _unit(rnd[2][q])
            ce = torch.sqrt(1 - el * el)
            eo = (iv + 1) % 3
            n = self.n[t[q], eo]
            lxy = (self.c[t[q], eo] - (n * Sq).sum(1)) / (n * c).sum(1)
            L = torch.minimum(lxy / ce, self.h / el)
            rr = _unit(rnd[3][q]) * L
            up = torch.where(l[q] == k[q], 1.0, -1.0)
            d[q] = torch.cat([(rr * ce)[:, None] * c, (up * rr * el)[:, None]], dim=1)
            wf[q] = alpha * L
        return d, wf

    def solve(self, first: int, last: int, rays: int, max_rays: int, steps: int, threshold: float, reflect: bool,
              mono: bool, key: int, logged: bool = False):
        slices = 5 if reflect else 1
        P = self.T * self.layers
        A, B = (self.A[:1], self.B[:1]) if mono else (self.A, self.B)
        At, Bt = torch.tensor(A, **_F), torch.tensor(B, **_F)
        n = last - first + 1
        phi, rse, log = np.zeros(n), np.zeros(n), []
        C = N_TOT / (4 * math.pi * TAU)
        for i in range(n):
            s = first + i
            lnw = self.weights(torch.tensor([s]), slices)[0]
            w = torch.exp(lnw - lnw.max())
            q = torch.ceil(w * 16777216.0).long()
            Q = int(q.sum())
            cum = torch.cumsum(q, 0) - q
            S, ls, pS = self.points[s % self.Np], s // self.Np, s % self.Np
            s1 = s2 = 0.0
            total = 0
            con = torch.zeros(slices * P, **_F)
            for k in range(steps + 1):
                target = rays if max_rays <= rays or not steps else (max_rays if k >= steps else min(max_rays, max(rays, int(
                    math.ceil(rays * ((max_rays / rays) ** (1.0 / steps)) ** k)))))
                M = target - total
                phase = int(_philox(0, s, k, 1, key, 0)[0])
                off = torch.div(cum * M + ((phase * Q) >> 32), Q, rounding_mode="floor")
                r = torch.arange(M, **_I)
                b = torch.searchsorted(off, r, right=True) - 1
                j, p = b // P, b % P
                l, t = p // self.T, p % self.T
                kk = self.image(torch.full_like(j, ls), j)
                SS = S.expand(M, 2)
                d, wf = self.start(SS, torch.full_like(t, pS), kk, t, l, _philox(r, s, k, 0, key, 0))
                D, G, Jb, Lc, done = self.walk(SS, kk, j, t, l, d, float(A[0]), float(B[0]))
                gain = torch.exp(G[:, None] + (At - A[0]) * Jb[:, None] - (Bt - B[0]) * (D - Lc)[:, None]).mean(1)
                X = torch.where(done, C * Q * self.beta[p] * wf * gain / q[b].double(), torch.zeros_like(gain))
                con.index_add_(0, b, X)
                s1, s2, total = s1 + float(X.sum()), s2 + float((X * X).sum()), target
                m = s1 / total
                phi[i], rse[i] = m, math.sqrt(abs(s2 / total - m * m) / total) / m
                if rse[i] <= threshold or target >= max_rays:
                    break
            log.append(con)
        sa, se = (float(self.B[0] / N_TOT), float((self.A - self.B)[0] / N_TOT)) if mono else (self.sa, self.se)
        bc = self.betaCells[first:last + 1]
        out = {"phiAse": phi, "relativeStandardError": rse, "dndtAse": (bc * (se + sa) - sa) * phi, "totalRays": None,
               "droppedRays": None}
        return (out, torch.stack(log).cpu().numpy()) if logged else out


def _exact_forward(case, twin: TetMesh, sa, se):
    """The forward method without reflections in 64 bits: 8 batches, stratified sources, track-length tallies."""
    C, Np, B, M = twin.numberOfCells, twin.numberOfPoints, 8, case["rays"]
    cells = np.sort(twin.cells.astype(np.int64), axis=1)
    v = twin.points[cells]
    inv = np.linalg.inv(np.swapaxes(v[:, 1:] - v[:, :1], 1, 2))
    a = np.concatenate([-inv.sum(1, keepdims=True), inv], 1)
    dd = -np.einsum("cfk,ck->cf", a, v[:, 0])
    dd[:, 0] += 1.0
    faces = np.stack([np.delete(cells, f, axis=1) for f in range(4)], 1).reshape(-1, 3)
    key = (faces[:, 0] * Np + faces[:, 1]) * Np + faces[:, 2]
    order = np.argsort(key, kind="stable")
    same = key[order][1:] == key[order][:-1]
    nbr = np.full(4 * C, -1, np.int64)
    i, j = order[:-1][same], order[1:][same]
    nbr[i], nbr[j] = j, i
    vol = twin.cellVolumes()
    clad = twin.claddingMask()
    matv = cells + Np * clad[:, None]
    lumped = np.bincount(matv.ravel(), np.repeat(vol / 4.0, 4), 2 * Np)
    beta = twin.betaVolume
    prefix = torch.tensor(np.cumsum(beta * vol), **_F)
    Bt = float(prefix[-1])
    a, dd, nbr, mv, ct = (torch.tensor(x, device=_DEV) for x in (a, dd, nbr.reshape(C, 4), matv, cells))
    pts, bt, cl = torch.tensor(twin.points, **_F), torch.tensor(beta, **_F), torch.tensor(clad, device=_DEV)
    mono = case["lambdas"] == 1
    sA, sE = torch.tensor(sa, **_F), torch.tensor(se, **_F)
    score = torch.zeros(B, 2 * Np, **_F)
    nb = [(M - b + B - 1) // B for b in range(B)]
    for b in range(B):
        o = _philox(b, 0, 0, 2, RNG_SEED, 1)
        shift, phase = int(o[0]) / 4294967296.0, int(o[1])
        i = torch.arange(nb[b], **_I)
        c = torch.searchsorted(prefix, (i.double() + shift) / nb[b] * Bt, right=True).clamp(max=C - 1)
        ray = i * B + b
        r1, r2 = _philox(ray, 0, 0, 3, RNG_SEED, 1), _philox(ray, 0, 1, 3, RNG_SEED, 1)
        ex = torch.stack([-torch.log(_unit(x)) for x in r1], 1)
        x = ((ex / ex.sum(1, keepdim=True))[..., None] * pts[ct[c]]).sum(1)
        z, ph = 2 * _unit(r2[0]) - 1, 2 * math.pi * _unit(r2[1])
        rr = torch.sqrt(1 - z * z)
        u = torch.stack([rr * torch.cos(ph), rr * torch.sin(ph), z], 1)
        lam = ((((i * 0x9E3779B9 + phase) & _M32) * (1 if mono else len(sa))) >> 32)
        st = dict(c=c, x=x, u=u, G=torch.ones(nb[b], **_F), ff=torch.full((nb[b],), -1, **_I), A=sA[lam], E=sE[lam])
        for _ in range(10000):
            if not st["c"].numel():
                break
            c = st["c"]
            L0 = (a[c] * st["x"][:, None]).sum(-1) + dd[c]
            dl = (a[c] * st["u"][:, None]).sum(-1)
            ok = (dl < 0) & (torch.arange(4, device=_DEV) != st["ff"][:, None])
            tt = torch.where(ok, L0.clamp(min=0) / torch.where(ok, -dl, torch.ones_like(dl)), torch.full_like(dl, math.inf))
            ln, f = tt.min(1)
            g = torch.where(cl[c], torch.full_like(ln, -twin.claddingAbsorption), N_TOT * (bt[c] * (st["E"] + st["A"]) - st["A"]))
            E = torch.expm1(g * ln)
            w = (L0 + 0.5 * ln[:, None] * dl).clamp(min=0)
            con = st["G"] * torch.where((g * ln).abs() < 1e-8, ln, E / g)
            score[b].index_add_(0, mv[c].reshape(-1), (w / w.sum(1, keepdim=True) * con[:, None]).reshape(-1))
            code = nbr[c, f]
            st["G"], st["x"] = st["G"] * (1 + E), st["x"] + ln[:, None] * st["u"]
            st["c"], st["ff"] = code // 4, code % 4
            keep = code >= 0
            st = {k: y[keep] for k, y in st.items()}
    score = score.cpu().numpy()
    dens = np.where(lumped > 0, score / np.where(lumped > 0, lumped, 1.0), 0.0)[:, matv].mean(-1) * vol
    phi = dens.sum(0) * Bt / (M * vol) * N_TOT / TAU
    per = dens / np.array(nb, np.float64)[:, None]
    with np.errstate(divide="ignore", invalid="ignore"):
        rse = per.std(0, ddof=1) / math.sqrt(B) / np.abs(per.mean(0))
    k = 1 if mono else len(sa)
    return {"phiAse": phi, "relativeStandardError": rse, "totalRays": None, "droppedRays": None,
            "dndtAse": (beta * (max(se[:k]) + max(sa[:k])) - max(sa[:k])) * phi}


def _exact_train(case, off, f, t, params):
    """The network, the groups' softmax cross entropy and Adam, in 64 bits."""
    shapes = [(12, 64), (64,), (64, 64), (64,), (64, 64), (64,), (64,), ()]
    p, at = [], 0
    for s in shapes:
        n = int(np.prod(s))
        p.append(torch.tensor(params[at:at + n].reshape(s), **_F).requires_grad_())
        at += n
    opt = torch.optim.Adam(p, lr=1e-3)
    f, t = torch.tensor(f, **_F), torch.tensor(t, **_F)
    per = case["groups_per_step"]
    hist = []
    for step in range(case["steps"]):
        g0 = (step % (case["groups"] // per)) * per
        loss = 0.0
        for g in range(g0, g0 + per):
            x, y = f[off[g]:off[g + 1]], t[off[g]:off[g + 1]]
            h = x
            for k in (0, 2, 4):
                h = torch.nn.functional.silu(h @ p[k] + p[k + 1])
            lg = h @ p[6] + p[7]
            loss = loss + (torch.logsumexp(lg, 0) - (y * lg).sum() / y.sum()) / per
        opt.zero_grad()
        loss.backward()
        opt.step()
        hist.append(float(loss.detach()))
    return {"loss": np.array(hist), "params": torch.cat([x.detach().reshape(-1) for x in p]).cpu().numpy()}


def exact(case: dict, seed: int):
    """Weights from 16-bit networks and coarse grids draw other rays than 64-bit ones would, reservoirs fill in arrival
    order, and whole discs or time steps take too long: no value there."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "train":
        off, f, t = _training_rows(case, rng)
        return _exact_train(case, off, f, t, _network(rng))
    sa, se = _spectra(case.get("lambdas", 1)).resampled()
    if kind == "forward" and not case["reflect"]:
        return _exact_forward(case, TetMesh.fromPrismMesh(_mesh(case, rng)), sa, se)
    plain = kind == "solve" and case["proposal"] == "walks" or kind == "log"
    if not plain or case["samples"] == 0 or case["samples"] > 64:
        return None
    mesh = _mesh(case, rng)
    first, last = _block(mesh, case["samples"])
    m = _Prisms(mesh, sa, se)
    args = (case["rays"], case.get("max_rays", case["rays"]), 0, 0.0, case["reflect"], case["lambdas"] == 1, RNG_SEED)
    if kind == "log":
        out, con = m.solve(first, last, *args, logged=True)
        return dict(out, contributions=con, features=None)
    return m.solve(first, last, *args)
