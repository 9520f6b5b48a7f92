"""Pair lists written on the device: shells of s and p in every order within a
molecule, molecules of one type only and of one shell, in both orders within
the batch; the energies of the molecules one by one are the reference (with the
tolerance of the other batch tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

Z = np.array([[0.0, 0.0, 0.0], [0.0, 0.0, 2.1], [0.0, 2.3, -0.9], [2.4, 0.0, -0.7], [-2.2, -0.4, -1.0]])
SPECIES = [["He"], ["O", "H", "H"], ["H", "O", "H"], ["H", "C", "H", "H", "H"], ["C", "O"], ["H", "F"], ["Li", "H"]]


@pytest.mark.parametrize("basis", ["sto-3g", "sto-6g"])
@pytest.mark.parametrize("order", [1, -1])
def test_shell_orders(engine, basis, order):
    mols = []
    for sp in SPECIES[::order]:
        x = Z[:len(sp)].copy()
        if sp == ["H", "O", "H"]:
            x = x[[1, 0, 2]]
        if len(sp) == 5:
            x = x[[1, 0, 2, 3, 4]]
        mols.append(engine.Molecule(sp, x, basis))
    for m, r in zip(mols, engine.run_batch(mols)):
        assert r.energy == pytest.approx(engine.run(m).energy, abs=1e-8)
