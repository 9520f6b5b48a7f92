"""J and K of a converged density from the split kernels against the undivided
ones for the same quartets, to the rounding of the sums: far quartets that only
J needs are not digested for K, and what that leaves out has to stay below it.

A neon of nine primitives per shell, whose functions the density does not
touch, makes every class too deep for the split kernels; its functions come
last, so the chain's block is J and K of the chain alone."""
import numpy as np
import pytest

from conftest import basis_file

pytestmark = pytest.mark.gpu


def _basis_with_deep_neon(folder):
    a = np.geomspace(0.15, 400.0, 9)
    c = 0.1 * np.exp(-0.5 * ((np.log(a) - 0.5) / 1.5) ** 2)
    rows = "".join(f"  {x:.10E}  {y:.10E}  {y:.10E}\n" for x, y in zip(a, c))
    text = open(basis_file("sto-3g")).read()
    lo = text.index("Ne     0")
    hi = text.index("****", lo)
    (folder / "basis_set").mkdir()
    (folder / "basis_set" / "deep.txt").write_text(text[:lo] + "Ne     0\nSP   9   1.00\n" + rows + text[hi:])


@pytest.mark.parametrize("n", [30, 40])
def test_scf_density(engine, tmp_path, n):
    import torch
    from pyfacc import _native as N
    from pyfacc import geometry as G
    _basis_with_deep_neon(tmp_path)
    sp, xyz = G.alkane(n, seed=n)
    with engine.System(engine.Molecule(sp, xyz)) as s:
        D = torch.tensor(s.scf(matrices=True).matrices["P"], device="cuda")
        before = N.lib().pyfacc_split_launch_count(1)
        J, K = s.jk(D)
        assert N.lib().pyfacc_split_launch_count(1) > before
    m = len(D)
    with engine.System(engine.Molecule(sp + ["Ne"], np.vstack([xyz, xyz.max(0) + 20.0]), "deep"),
                       data_dir=str(tmp_path)) as s:
        De = torch.zeros(s.nbf, s.nbf, dtype=torch.float64, device="cuda")
        De[:m, :m] = D
        before = N.lib().pyfacc_split_launch_count(0)
        Jr, Kr = (x[:m, :m] for x in s.jk(De))
        assert N.lib().pyfacc_split_launch_count(0) == before
    # an element sums some 1e4 contributions in any order, a contribution up to
    # 81 primitive quartets of 1e-15: 1e2 * 1.1e-16 + 9 * 1e-15 = 2e-14
    assert ((K - Kr).norm() / Kr.norm()).item() < 2e-14
    assert ((J - Jr).norm() / Jr.norm()).item() < 2e-14
