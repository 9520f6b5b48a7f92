"""FP64 and FP32 gradients in Hermite Gaussians against the oracle's: shells on
one axis (whole Hermite components vanish), on one atom, in deep contractions,
closed and open shells; the lists are short enough for the undivided kernels.
The tolerances are those of the other gradient tests against the oracle for
FP64; in mixed precision single integrals are good to 2^-20 of their bound and
the densities converge to 1e-8, which leaves 1e-5."""
import numpy as np
import pytest

from conftest import basis_file

pytestmark = pytest.mark.gpu

MOLS = {
    "CO on z": (["C", "O"], [[0, 0, 0], [0, 0, 2.13]], "sto-3g"),
    "CO on x": (["C", "O"], [[-1.0, 0, 0], [1.13, 0, 0]], "sto-6g"),
    "NH2": (["N", "H", "H"], [[0.1, 0, 0.2], [1.5, 0.3, 1.2], [-1.4, -0.2, 1.3]], "sto-3g"),
    "2 HF apart": (["F", "H", "F", "H"], [[0, 0, 0], [0, 0, 1.8], [3.0, 12.0, 1.0], [3.0, 13.0, 2.5]], "sto-3g"),
    "HCN": (["H", "C", "N"], [[0, 0.1, -2.0], [0, 0, 0], [0.2, 0, 2.2]], "sto-4g"),
}


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-7), ("mixed", 1e-5)])
@pytest.mark.parametrize("name", list(MOLS))
def test_gradient_vs_oracle(engine, oracle, name, precision, tol):
    sp, xyz, basis = MOLS[name]
    xyz = np.array(xyz, dtype=float)
    m = oracle.molecule(sp, xyz, basis_file(basis))
    r = engine.run(engine.Molecule(sp, xyz, basis), gradient=True, matrices=True, precision=precision)
    # at the engine's density: an open shell has more than one SCF solution
    Ca = r.matrices["C_alpha"][:, :m.nalpha]
    Cb = (r.matrices["C_beta"] if r.uhf else r.matrices["C_alpha"])[:, :m.nbeta]
    ref = oracle.gradient_at_density(m, [Ca @ Ca.T, Cb @ Cb.T], uhf=r.uhf)
    assert np.abs(r.gradient - ref).max() < tol
