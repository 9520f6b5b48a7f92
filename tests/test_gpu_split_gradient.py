"""The FP64 gradient of long quartet lists (far and near quartets apart)
against finite differences of the energy along a random direction, closed and
open shell, and its translational invariance."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("open_shell,n,basis", [(False, 24, "sto-3g"), (True, 24, "sto-2g")])
def test_split_gradient_vs_finite_difference(engine, open_shell, n, basis):
    from pyfacc import geometry as G
    sp, xyz = (G.radical if open_shell else G.alkane)(n, seed=n)
    d = np.random.default_rng(5).standard_normal(xyz.shape)
    d /= np.linalg.norm(d)
    opt = dict(eps_diis=1e-9)
    g = engine.run(engine.Molecule(sp, xyz, basis), gradient=True, **opt).gradient
    h = 2e-4
    # central difference, error h^2 E''' / 6 (|E'''| of a unit displacement of
    # the whole chain < 1 Ha/bohr^3) plus the energies' 1e-10 Ha over 2 h
    e = [engine.run(engine.Molecule(sp, xyz + s * h * d, basis), **opt).energy for s in (1, -1)]
    assert abs((g * d).sum() - (e[0] - e[1]) / (2 * h)) < h * h / 6 + 1e-10 / h
    assert np.abs(g.sum(0)).max() < 1e-9
