"""A context that projects one state after another, the water elsewhere each time: every projection
equals a fresh context's, bit for bit (no value that an earlier state left off the water enters)."""
import numpy as np
import pytest

from mpp import scene

pytestmark = pytest.mark.gpu

STATES = [dict(height=0.62, seed=11), dict(height=0.41, seed=12), dict(height=0.55, seed=13)]


def _load(s, b):
    import torch

    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    for name in ("u", "v", "w", "types", "phi"):
        getattr(s, name).copy_(t(getattr(b, name)))
    s.P.zero_()
    s.volume0 = s.projector.volume(s.phi)


@pytest.mark.parametrize("precision", ["fp32", "fp16", "fp64"])
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("n", [(64, 64, 64), (48, 40, 24)])
def test_reused_context_equals_fresh(cuda, precision, graph, n):
    import mpp

    kw = dict(tol=1e-6 if precision != "fp64" else 1e-10, maxiter=100, precision=precision, graph=graph)
    basins = [scene.box_basin(n, **c) for c in STATES]
    reused = mpp.FlipBasin.from_scene(basins[0], **kw)
    for b in basins:
        _load(reused, b)
        mpp.project(reused, 1 / 48)
        fresh = mpp.FlipBasin.from_scene(b, **kw)
        mpp.project(fresh, 1 / 48)
        assert reused.last.iterations == fresh.last.iterations
        for name in ("P", "u", "v", "w", "fu", "fv", "fw"):
            assert np.array_equal(getattr(reused, name).cpu().numpy(), getattr(fresh, name).cpu().numpy()), name
