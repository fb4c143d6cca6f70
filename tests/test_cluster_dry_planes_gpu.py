"""k_cluster's exchange where the planes between its CTAs are dry or half wet: bodies of water with air
between them, water in the first CTA's planes alone, planes with cells of one colour. Bit for bit against
the per-level launches (MPP_CMG=0), over several projections of one context."""
import dataclasses
import os

import numpy as np
import pytest

from mpp import scene

pytestmark = pytest.mark.gpu

# the fine grid, and the planes a CTA holds of the level that is spread (half the fine extents)
# (in Float64 only the last one's levels fit the cluster; the others' largest stays a launch a pass there)
GRIDS = {"32_of_2": ((64, 64, 64), 2), "48x24x24_of_2": ((96, 48, 48), 2), "32x32x64_of_4": ((64, 64, 128), 4),
         "32x16x32_of_2": ((64, 32, 64), 2)}


def _wet(case, n, per, rng):
    """Wet cells of the spread level, [plane, row, column]."""
    m3, m2, m1 = n[2] // 2, n[1] // 2, n[0] // 2
    k, j, i = np.meshgrid(np.arange(m3), np.arange(m2), np.arange(m1), indexing="ij")
    wet = k < (7 * m3) // 8
    if case == "gap_above":      # a CTA's highest plane dry, water in the next one's lowest
        return wet & (k != 3 * per - 1)
    if case == "gap_below":      # a CTA's lowest plane dry, water in the highest of the one before
        return wet & (k != 5 * per)
    if case == "unequal":        # dry planes on both sides of a boundary, a small body above a large one
        return wet & ((k < 4 * per - 1) | ((k > 4 * per) & (i < m1 // 2) & (j >= m2 // 4) & (j < m2 // 2)))
    if case == "first_only":     # water in CTA 0's planes and nowhere else
        return k < per
    if case == "first_plane":    # and in its lowest alone
        return k < 1
    if case == "one_colour":     # boundary planes with cells of one colour, the other colour next
        odd = (i + j + k) % 2 == 1
        return wet & ((k != 2 * per - 1) | odd) & ((k != 4 * per) | odd) & ((k != 6 * per - 1) | ~odd)
    if case == "drops":          # anywhere
        return rng.random(k.shape) < 0.35
    raise KeyError(case)


def _basins(case, grid, count):
    n, per = GRIDS[grid]
    out = []
    for s in range(count):
        b = scene.box_basin(n, seed=90 + s, wall=0.48)
        rng = np.random.default_rng(700 + s)
        wet = np.repeat(np.repeat(np.repeat(_wet(case, n, per, rng), 2, 0), 2, 1), 2, 2)
        d = (0.2 + 0.8 * rng.random(wet.shape)) * b.grid.dx
        phi = np.where(wet, -d, d).astype(np.float32)
        solid = (b.types == scene.SOLID).reshape(wet.shape)
        types = np.where(solid, scene.SOLID, np.where(wet, scene.LIQUID, scene.AIR)).astype(np.uint8)
        out.append(dataclasses.replace(b, types=types.reshape(-1), phi=phi.reshape(-1)))
    return out


def _solve(basins, precision, cluster, sweeps):
    import torch

    import mpp

    saved = {k: os.environ.get(k) for k in ("MPP_CMG", "MPP_BOTTOM_CELLS")}
    os.environ["MPP_BOTTOM_CELLS"] = "512"
    if cluster:
        os.environ.pop("MPP_CMG", None)
    else:
        os.environ["MPP_CMG"] = "0"
    try:  # the context reads both when it is created
        s = mpp.FlipBasin.from_scene(basins[0], tol=1e-6 if precision != "fp64" else 1e-10, maxiter=60,
                                     precision=precision, graph=True, sweeps=sweeps)
    finally:
        for k, v in saved.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v
    out = []
    for b in basins:
        for name in ("u", "v", "w", "types", "phi"):
            getattr(s, name).copy_(torch.from_numpy(getattr(b, name)).cuda())
        s.P.zero_()
        s.volume0 = s.projector.volume(s.phi)
        mpp.project(s, 1 / 48)
        out.append((s.P.cpu().numpy(), s.u.cpu().numpy(), s.last.iterations))
    return out


@pytest.mark.parametrize("case", ["gap_above", "gap_below", "unequal", "first_only", "first_plane", "one_colour", "drops"])
@pytest.mark.parametrize("grid", sorted(GRIDS))
@pytest.mark.parametrize("precision,sweeps", [("fp32", 1), ("fp32", 2), ("fp16", 6), ("bf16", 4), ("fp64", 3)])
def test_dry_planes(cuda, case, grid, precision, sweeps):
    basins = _basins(case, grid, 3)
    want, got = (_solve(basins, precision, cluster, sweeps) for cluster in (False, True))
    for (P0, u0, it0), (P1, u1, it1) in zip(want, got):
        assert it1 == it0 and it0 > 0
        assert np.array_equal(P1, P0)
        assert np.array_equal(u1, u0)
