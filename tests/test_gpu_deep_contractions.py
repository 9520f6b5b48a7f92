"""Pairs of more primitive pairs than STO-6G has: the loops over a pair's
primitives stop at a cut, so the records have to be in falling order of their
prefactors whatever the basis file's order and however many there are (64 on
either side: the sort changes there)."""
import numpy as np
import pytest

from conftest import basis_file

pytestmark = pytest.mark.gpu


def _deep_basis(folder, depth, rising):
    """STO-3G with a helium of `depth` primitives in rising or falling order."""
    a = np.geomspace(0.1, 2000.0, depth)
    c = np.exp(-0.5 * ((np.log(a) - 0.5) / 1.5) ** 2)
    rows = [f"  {x:.10E}  {y:.10E}\n" for x, y in zip(a, c / c.sum())]
    text = open(basis_file("sto-3g")).read()
    lo = text.index("He     0")
    hi = text.index("****", lo)
    (folder / "basis_set").mkdir()
    path = folder / "basis_set" / "deep.txt"
    path.write_text(text[:lo] + f"He     0\nS   {depth}   1.00\n" + "".join(rows if rising else rows[::-1]) + text[hi:])
    return str(path)


@pytest.mark.parametrize("depth", [8, 9, 16])
@pytest.mark.parametrize("rising", [True, False])
def test_primitives_in_any_order(engine, oracle, tmp_path, depth, rising):
    import torch
    path = _deep_basis(tmp_path, depth, rising)
    sp = ["O", "H", "H", "He", "C", "He"]
    xyz = np.array([[0, 0, 0], [0, 1.43, 1.1], [0, -1.43, 1.1], [2.5, 0.3, 0.2], [0.4, 0.2, 5.1], [1.0, 3.0, 4.0]])
    om = oracle.molecule(sp, xyz, path)
    rng = np.random.default_rng(depth)
    n = om.shells.nbf
    D = 0.3 * rng.standard_normal((n, n))
    D = D + D.T
    Jo, Ko = oracle.jk(om, D, thresh=0)
    with engine.System(engine.Molecule(sp, xyz, "deep"), data_dir=str(tmp_path)) as s:
        J, K = s.jk(torch.tensor(D))
    assert np.abs(J.cpu().numpy() - Jo).max() < 1e-10  # the J/K tolerance of the FP64 parity tests
    assert np.abs(K.cpu().numpy() - Ko).max() < 1e-10
