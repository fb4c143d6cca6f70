"""The level-set sweeps and the extrapolation at the shapes and alignments where their kernels change
form, bit for bit against the oracle: rows of whole quads and not, walls that touch the box's edge or
leave no open cell, a floor inside the grid, NaN, infinities and signed zeros, flags of any nonzero
value, arrays that are not 16-byte aligned."""
import dataclasses

import numpy as np
import pytest

import oracle
from mpp import scene
from test_levelset_gpu import _noisy_phi

pytestmark = pytest.mark.gpu

GRIDS = {
    "quads": dict(n=(36, 20, 12)),
    "one_quad": dict(n=(4, 6, 8), wall=0.8),
    "no_quads": dict(n=(18, 10, 14)),
    "all_open": dict(n=(24, 16, 16), wall=2.0),
    "narrow": dict(n=(40, 24, 16), wall=0.03),
    "floor": dict(n=(32, 32, 24), floor=0.31),
}


def _basin(name):
    c = dict(GRIDS[name])
    floor = c.pop("floor", None)
    b = scene.box_basin(c.pop("n"), seed=91, **c)
    if floor is not None:
        b = dataclasses.replace(b, grid=dataclasses.replace(b.grid, floor=floor))
    return b


def _shifted(a, by):
    """A device copy of `a` that starts `by` elements into its allocation."""
    import torch

    t = torch.zeros(a.size + by, dtype=torch.from_numpy(a).dtype, device="cuda")
    t[by:] = torch.from_numpy(a).cuda()
    return t[by:]


@pytest.mark.parametrize("name", sorted(GRIDS))
@pytest.mark.parametrize("odd_values", [False, True])
@pytest.mark.parametrize("shift", [0, 1])
def test_redistance_shapes(cuda, name, odd_values, shift):
    import mpp

    b = _basin(name)
    phi = _noisy_phi(b, 17)
    if odd_values:
        rng = np.random.default_rng(3)
        for v in (np.nan, np.inf, -np.inf, 0.0, -0.0, 1e-40):
            phi[rng.integers(0, phi.size, max(2, phi.size // 200))] = v
    p = mpp.Projector(b.grid)
    a, a0 = _shifted(phi, shift), _shifted(phi, shift)
    types = _shifted(np.zeros(phi.size, np.uint8), shift)
    out = p.redistance(a, a0, 5, types=types)
    want = oracle.redistance(b.grid, phi, 5)
    assert np.array_equal(out.cpu().numpy(), want, equal_nan=True)
    classes = oracle.classify(b.grid, want)
    assert np.array_equal(types.cpu().numpy(), classes)
    types.zero_()
    p.classify(types, out)
    assert np.array_equal(types.cpu().numpy(), classes)


@pytest.mark.parametrize("name", sorted(GRIDS))
@pytest.mark.parametrize("layers", [0, 1, 4])
@pytest.mark.parametrize("shift", [0, 1])
def test_extrapolate_shapes(cuda, name, layers, shift):
    import mpp

    b = _basin(name)
    g = b.grid
    rng = np.random.default_rng(29)
    vel = [rng.uniform(-1, 1, int(np.prod(g.face_shape(a)))).astype(np.float32) for a in range(3)]
    fl = [rng.choice(np.array([0, 0, 0, 0, 1, 7, 255], np.uint8), v.size) for v in vel]
    p = mpp.Projector(g)
    tv, tf = [_shifted(v, shift) for v in vel], [_shifted(f, shift) for f in fl]
    p.extrapolate(*tv, *tf, layers=layers)
    want = oracle.extrapolate(g, *vel, *fl, layers=layers)
    for t, w in zip(tv + tf, want):
        assert np.array_equal(t.cpu().numpy(), np.asarray(w))
