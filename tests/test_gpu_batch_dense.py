"""The batch's dense step at the edges of its 16 x 16 tiles: one function,
ragged and whole tiles, a triangle of more tiles than warps, the
largest molecule a batch takes.  H2 chains in STO-3G have as many functions as
atoms; the single-molecule engine, whose products and DIIS are other code, is
the reference, with the tolerances of the other batch tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain(n):
    """n / 2 H2 molecules in a row (bohr), shifted off the axis by turns."""
    x = np.zeros((n, 3))
    x[:, 2] = 4.2 * (np.arange(n) // 2) + 1.4 * (np.arange(n) % 2)
    x[:, 0] = 0.5 * ((np.arange(n) // 2) % 3)
    return ["H"] * n, x


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_dense_step_sizes(engine, precision):
    specs = [(["He"], np.zeros((1, 3)))] + [chain(n) for n in (2, 4, 14, 16, 18, 30, 32, 34, 66, 112, 160)]
    mols = [engine.Molecule(s, x) for s, x in specs]
    rb = engine.run_batch(mols, gradient=True, precision=precision)
    tol = 1e-8 if precision == "fp64" else 1e-6
    for m, r in zip(mols, rb):
        rs = engine.System(m, precision=precision).scf(gradient=True)
        assert r.converged and rs.converged
        assert r.energy == pytest.approx(rs.energy, abs=tol)
        assert np.abs(r.gradient - rs.gradient).max() < 10 * tol


def test_batch_core_guess_sizes(engine):
    mols = [engine.Molecule(*chain(n)) for n in (2, 18, 48)]
    for m, r in zip(mols, engine.run_batch(mols, guess="core")):
        assert r.energy == pytest.approx(engine.System(m, guess="core").scf().energy, abs=1e-8)
