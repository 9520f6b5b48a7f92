"""The FP32 derivative quartets of long lists (far and near kernels, two bra
primitives at a time: 9 primitive pairs leave one over) against the FP64
gradient at the same density: single molecules on either side of the line and
more atoms than the undivided kernels sum in shared memory, open shells, deep
contractions, a batch.  Mixed-precision gradients are good to 1e-5 Ha/bohr of
the FP64 ones in the other tests; with the density held equal, a fifth."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-6


@pytest.mark.parametrize("open_shell,n,basis", [(False, 18, "sto-3g"), (False, 32, "sto-3g"), (False, 86, "sto-2g"),
                                                (True, 26, "sto-3g"), (True, 22, "sto-6g")])
def test_fp32_lists(engine, open_shell, n, basis):
    from pyfacc import geometry as G
    m = engine.Molecule(*(G.radical if open_shell else G.alkane)(n, seed=n), basis)
    g64 = engine.run(m, gradient=True).gradient
    g = engine.run(m, gradient=True, gradient_precision="mixed").gradient
    assert np.abs(g - g64).max() < TOL
    assert np.abs(g.sum(0)).max() < 1e-8


@pytest.mark.parametrize("basis", ["sto-3g", "sto-4g"])
def test_fp32_lists_of_a_batch(engine, basis):
    from pyfacc import geometry as G
    mols = [engine.Molecule(*x, basis) for x in G.water_clusters(40, 5, 6, 16)]
    a = engine.run_batch(mols, gradient=True)
    b = engine.run_batch(mols, gradient=True, gradient_precision="mixed")
    for x, y in zip(a, b):
        assert np.abs(x.gradient - y.gradient).max() < TOL
