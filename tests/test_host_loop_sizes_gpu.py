"""The host-driven loop against the graph's, bit for bit, on either side of the size from which one colour pass
instead of three is launched before the host knows whether the loop goes on, and with fewer passes than that."""
import numpy as np
import pytest

from mpp import scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(32, 32, 32), (256, 128, 112), (256, 128, 128)])
@pytest.mark.parametrize("precision,sweeps", [("fp32", 1), ("fp32", 2), ("fp16", 4)])
def test_host_loop_equals_graph(cuda, n, precision, sweeps):
    import mpp

    b = scene.box_basin(n, seed=58, wall=0.24 if n[0] > n[1] else 0.45)
    out = []
    for graph in (False, True):
        s = mpp.FlipBasin.from_scene(b, tol=1e-5, maxiter=60, precision=precision, sweeps=sweeps, graph=graph)
        for _ in range(2):  # the second projection starts from the first one's pressure and velocities
            mpp.project(s, 1 / 48)
        out.append((s.P.cpu().numpy(), s.w.cpu().numpy(), list(s.iterations)))
    assert out[0][2] == out[1][2] and out[0][2][0] > 0
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
