"""pressure! of the sparse basin for a right-hand side that is not zero in the air: the V-cycle's residual
carries it to the coarser levels from every cell that is not SOLID, in whatever row pieces it lies."""
import numpy as np
import pytest

from mpp import sparse_scene as ss
from oracle import sparse as osp
from test_sparse_gpu import _dev, _host, _used

pytestmark = pytest.mark.gpu

BASINS = {"4x4x4": dict(nb=(4, 4, 4), seed=2201), "8x8x8_rings": dict(nb=(8, 8, 8), seed=2203, rings=1),
          "tall": dict(nb=(3, 3, 9), seed=43, rings=0, height=0.3, free_every=2)}


@pytest.mark.parametrize("name", sorted(BASINS))
@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("sweeps", [1, 2])
def test_noise_in_the_air(cuda, name, graph, sweeps):
    from mpp import sparse as msp

    sc = ss.sparse_basin(warm=False, **BASINS[name])
    bf, bc = osp.rhs(sc, np.float32(0.01))
    water, air = sc.tf == 1, sc.tf == 2
    rng = np.random.default_rng(3)
    rms = float(np.sqrt(np.mean(bf[water].astype(np.float64) ** 2)))
    bf[air] = (0.02 * rms * rng.standard_normal(np.count_nonzero(air))).astype(np.float32)
    want = sc.copy()
    info = osp.pressure(want, bf, bc, tol=1e-6, maxiter=4, sweeps=sweeps)
    s = msp.SparseBasin.from_scene(sc, graph=graph, tol=1e-6, maxiter=4, sweeps=sweeps)
    with pytest.warns(RuntimeWarning, match="did not converge"):
        its = msp.pressure(s, _dev(bf), _dev(bc))
    assert its == info["iterations"] == 4
    P, Q = _used(sc, _host(s.Pf), 4096).astype(np.float64), _used(sc, want.Pf, 4096)
    # the same four iterations but for the dot products' sums (Float32 trees in the oracle, about 1e-6); the noise
    # left out of the pieces without water moves the pressure by 2e-4 and more
    assert np.linalg.norm(P - Q) <= 1e-5 * np.linalg.norm(Q)
