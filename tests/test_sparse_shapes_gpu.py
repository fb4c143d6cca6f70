"""The sparse composite passes over basins whose coarse unknowns meet fine blocks in every way (blocks on
several sides of a coarse cell, at the box's edge, free slots between used ones), bit for bit against
the oracle: the operator, one V-cycle and a whole projection."""
import numpy as np
import pytest

from oracle import sparse as osp
from mpp import sparse_scene as ss
from test_sparse_gpu import _dev, _host, _unknowns, _used

pytestmark = pytest.mark.gpu

BASINS = {
    "narrow": dict(nb=(3, 5, 4), seed=41, rings=0, funnel=0.6),
    "ringed": dict(nb=(5, 4, 3), seed=42, rings=1, funnel=0.3, wall=0.48),
    "tall": dict(nb=(3, 3, 9), seed=43, rings=0, height=0.3, free_every=2),
    "full": dict(nb=(4, 4, 3), seed=44, rings=2),
}


@pytest.mark.parametrize("name", sorted(BASINS))
def test_shapes_match_oracle(cuda, name):
    import torch

    from mpp import sparse as msp

    sc = ss.sparse_basin(warm=True, **BASINS[name])
    fine_u, coarse_u = _unknowns(sc)
    s = msp.SparseBasin.from_scene(sc, tol=1e-5, maxiter=200)
    rng = np.random.default_rng(5)
    xf = np.where(fine_u, rng.standard_normal(fine_u.size), 0).astype(np.float32)
    xc = np.where(coarse_u, rng.standard_normal(coarse_u.size), 0).astype(np.float32)
    s.operator()
    for op in ("apply", "vcycle"):
        qf, qc = torch.zeros(xf.size, device="cuda"), torch.zeros(xc.size, device="cuda")
        getattr(s, op)(_dev(xf), _dev(xc), qf, qc)
        of, oc = getattr(osp, op)(sc, xf, xc)
        assert np.array_equal(_used(sc, _host(qf), 4096), _used(sc, of, 4096)), op
        assert np.array_equal(_host(qc), oc), op
    ref = sc.copy()
    info = osp.project(ref, s.volume0, tol=1e-5, maxiter=200)
    for _ in range(2):  # the second projection finds the first one's values in its workspace
        for k in ("uf", "uc", "vf", "vc", "wf", "wc", "Pf", "Pc"):
            getattr(s, k).copy_(_dev(getattr(sc, k)))
        msp.project(s, 1 / 48)
        assert abs(s.last.iterations - info["iterations"]) <= 1
        P, Q = _used(sc, _host(s.Pf), 4096), _used(sc, ref.Pf, 4096)
        assert np.linalg.norm(P - Q) <= 1e-3 * np.linalg.norm(Q)  # both stop at 1e-5 of the right-hand side
        assert np.array_equal(_used(sc, _host(s.fuf), 4352), _used(sc, ref.fuf, 4352))
