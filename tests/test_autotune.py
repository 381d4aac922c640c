"""The autotuner's sweep on a stand-in for the device context (CPU): what it may choose and what it hands on."""

from __future__ import annotations

from types import SimpleNamespace

import pytest


class _Context:
    """Solves take `cost(variant, rays per lane)` milliseconds."""

    numberOfWavelengths = 1

    def __init__(self, triangles, cost):
        self.mesh = SimpleNamespace(numberOfTriangles=triangles, numberOfLevels=5)
        self.cost, self.seen = cost, []

    def calc_phi_ase(self, *, rayKernelVariant=0, raysPerThread=0, **kw):
        self.seen.append((rayKernelVariant, raysPerThread))
        return SimpleNamespace(rayMilliseconds=self.cost(rayKernelVariant, raysPerThread), importanceMilliseconds=2.5)


@pytest.mark.parametrize("best", [(0, 0), (3, 0), (2, 64)])
def test_every_item_size_is_a_candidate(native, best):
    """The library's own item size (0: chosen from each pass's rays) is swept with every launch shape, so a tuned solve
    is never slower than an untuned one for want of it."""
    from haseongpu_b200.autotune import RAYS_PER_LANE, autotune, variant_names

    ctx = _Context(1000 + 10 * best[0] + best[1], lambda v, r: 1.0 if (v, r) == best else 2.0)
    tuned = autotune(ctx, firstSample=0, samples=8, rays=1000, useReflections=False, monochromatic=True)
    names = variant_names()
    assert {(v, r) for v in range(len(names)) for r in RAYS_PER_LANE} <= set(ctx.seen)
    assert (tuned.rayKernelVariant, tuned.raysPerThread, tuned.name) == (*best, names[best[0]])
    assert tuned.kwargs() == {"rayKernelVariant": best[0], "raysPerThread": best[1], "importanceLayers": 0}
    assert tuned.importanceMilliseconds == 2.5


@pytest.mark.parametrize("best", [(1, 0), (2, 128)])
def test_batches_sweep_the_same_candidates(native, best):
    from haseongpu_b200.autotune import autotune_batch

    def solve(media, *, rayKernelVariant, raysPerThread, **kw):
        return None, SimpleNamespace(rayMilliseconds=1.0 if (rayKernelVariant, raysPerThread) == best else 2.0)

    tuned = autotune_batch(SimpleNamespace(solve=solve), [], rays=1000)
    assert (tuned.rayKernelVariant, tuned.raysPerThread) == best
