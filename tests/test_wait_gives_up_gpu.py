"""A wait of the cluster's halo exchange that gives up (MPP_CMG_TRIES=0: each does, at once, having waited
for nothing) is an error of every call that runs V-cycles, which names the exchange; the next call on a
context that waits is right again."""
import os

import numpy as np
import pytest

from mpp import scene

pytestmark = pytest.mark.gpu

MATCH = "halo exchange"


def _without_waits(make):
    saved = os.environ.get("MPP_CMG_TRIES")
    os.environ["MPP_CMG_TRIES"] = "0"
    try:  # the context reads it when it is created
        return make()
    finally:
        if saved is None:
            os.environ.pop("MPP_CMG_TRIES")
        else:
            os.environ["MPP_CMG_TRIES"] = saved


def _dev(a):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_project(cuda, precision, graph):
    import mpp

    b = scene.box_basin(64, seed=31)
    s = _without_waits(lambda: mpp.FlipBasin.from_scene(b, tol=1e-5, maxiter=3, precision=precision, graph=graph))
    with pytest.raises(mpp.MppError, match=MATCH):
        mpp.project(s, 1 / 48)
    ok = mpp.FlipBasin.from_scene(b, tol=1e-5, maxiter=60, precision=precision, graph=graph)
    mpp.project(ok, 1 / 48)
    assert ok.last.status == 0


def test_vcycle(cuda):
    import mpp

    b = scene.box_basin(64, seed=32)
    r = np.where(b.types == scene.LIQUID, scene.uniform(3, 7, b.grid.ncells), 0).astype(np.float32)
    p = _without_waits(lambda: mpp.Projector(b.grid))
    with pytest.raises(mpp.MppError, match=MATCH):
        p.vcycle(_dev(r), _dev(b.types), _dev(b.phi))


@pytest.mark.parametrize("precision", ["fp32", "fp16", "fp64"])
def test_fallback(cuda, precision):
    """CG ends before its first V-cycle (the warm start is NaN), so the V-cycles are FGMRES's."""
    import mpp

    b = scene.box_basin((64, 32, 64), seed=33)  # (a size whose spread level fits the cluster in Float64 too)
    rhs = np.where(b.types == scene.LIQUID, scene.uniform(4, 7, b.grid.ncells), 0).astype(np.float32)
    P0 = np.where(b.types == scene.LIQUID, np.nan, 0).astype(np.float32)
    run = lambda p: p.pressure(_dev(P0), _dev(rhs), _dev(b.types), _dev(b.phi))
    kw = dict(tol=1e-5, fallback=True, precision=precision, fallback_maxiter=60)
    res = run(mpp.Projector(b.grid, **kw))
    assert res.iterations == 0 and res.fallback_used == 1 and res.fallback_iterations > 0
    with pytest.raises(mpp.MppError, match=MATCH):
        run(_without_waits(lambda: mpp.Projector(b.grid, **kw)))


@pytest.mark.parametrize("grouped", [True, False])
def test_batch(cuda, grouped):
    import mpp
    from mpp.batch import Batch

    basins = [scene.box_basin(64, seed=34 + i) for i in range(3)]
    bt = _without_waits(lambda: Batch(basins, tol=1e-5, maxiter=3))
    bt.set_grouped(grouped)
    with pytest.raises(mpp.MppError, match="basin 0.*" + MATCH):
        bt.project(1 / 48)
