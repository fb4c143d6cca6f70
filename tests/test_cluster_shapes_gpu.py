"""k_cluster (the small levels in one launch) against the per-level launches and the one-CTA bottom
solve, bit for bit, over the shapes at which its layout changes: levels in one CTA alone, one
level spread over the cluster, planes that do not divide by the cluster, an odd coarsest level, more
cells of a colour than a CTA's threads hold at once, and bottom levels above the coarsest."""
import dataclasses
import os

import numpy as np
import pytest

from mpp import scene

pytestmark = pytest.mark.gpu

CASES = {
    "one_cta": dict(n=(32, 32, 32)),                              # 16^3, 8^3
    "one_cta_small": dict(n=(16, 16, 32)),                        # 8 x 8 x 16 coarsest straight below the fine level
    "spread_one": dict(n=(64, 64, 64)),                           # 32^3 spread, 16^3, 8^3
    "spread_uneven": dict(n=(88, 72, 56)),                        # 28 planes over 16 CTAs; 11 x 9 x 7 coarsest
    "spread_24": dict(n=(96, 48, 48)),                            # 48 x 24 x 24, 24 x 12 x 12, 12 x 6 x 6
    "many_cells": dict(n=(80, 40, 20), wall=0.9, height=0.95),    # 40 x 20 x 10 all water: 3600 cells a colour
    "two_spread": dict(n=(128, 64, 128), wall=0.9, height=0.9),   # 64 x 32 x 64 too large, 32 x 16 x 32 spread
    "bottom_levels": dict(n=(64, 64, 64), levels=6),              # 8^3, 4^3 and 2^3 below the 16^3 level
}


def _solve(basin, precision, cluster, sweeps):
    import mpp

    saved = {k: os.environ.get(k) for k in ("MPP_CMG", "MPP_BOTTOM_CELLS")}
    os.environ["MPP_BOTTOM_CELLS"] = "512"
    if cluster:
        os.environ.pop("MPP_CMG", None)
    else:
        os.environ["MPP_CMG"] = "0"
    try:  # the context reads both when it is created
        s = mpp.FlipBasin.from_scene(basin, tol=1e-6 if precision != "fp64" else 1e-10, maxiter=100, precision=precision,
                                     graph=True, sweeps=sweeps)
    finally:
        for k, v in saved.items():
            if v is None:
                os.environ.pop(k, None)
            else:
                os.environ[k] = v
    mpp.project(s, 1 / 48)
    return s.P.cpu().numpy(), s.u.cpu().numpy(), s.last.iterations


@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("precision,sweeps", [("fp32", 2), ("fp16", 3), ("bf16", 1), ("fp64", 2)])
def test_cluster_shapes(cuda, case, precision, sweeps):
    c = dict(CASES[case])
    levels = c.pop("levels", None)
    b = scene.box_basin(c.pop("n"), seed=77, **c)
    if levels:
        b = dataclasses.replace(b, grid=dataclasses.replace(b.grid, levels=levels))
    P0, u0, it0 = _solve(b, precision, False, sweeps)
    P1, u1, it1 = _solve(b, precision, True, sweeps)
    assert it1 == it0 and it0 > 0
    assert np.array_equal(P1, P0)
    assert np.array_equal(u1, u0)
