"""Gradients of batches whose atoms' sums in shared memory come up to the
allowances of the one-electron kernel: 48 KB (2048 atoms) less its own static
arrays, and 96 KB (4096 atoms), where it goes over to global atomics."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [500, 600, 640, 682, 683, 1365, 1366])
def test_gradients(engine, count):
    from pyfacc import geometry as G
    waters = G.water_clusters(4, 3, 1, 1)
    mols = [engine.Molecule(*waters[i % 4]) for i in range(count)]  # three atoms each
    res = engine.run_batch(mols, gradient=True)
    ref = engine.run_batch(mols[:4], gradient=True)
    for i, r in enumerate(res):
        assert np.abs(r.gradient - ref[i % 4].gradient).max() < 1e-9
