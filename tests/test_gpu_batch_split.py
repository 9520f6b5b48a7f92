"""Batches long enough for the near kernel alone, and for the near and far
kernels, against the same batch on the undivided kernels (an explicit task
width), and a batch on either side of the line.  The kernels screen the same
quartets; they differ in rounding and, in the split kernels, in the primitive
and density-product cuts, all far below the tests' 1e-8 of the batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def compare(engine, clusters, precision, tol, **kw):
    mols = [engine.Molecule(s, x, **kw) for s, x in clusters]
    a = engine.run_batch(mols, gradient=True, precision=precision)
    b = engine.run_batch(mols, gradient=True, precision=precision, task_width=32)
    for x, y in zip(a, b):
        assert x.converged and y.converged
        assert x.energy == pytest.approx(y.energy, abs=tol)
        assert np.abs(x.gradient - y.gradient).max() < 10 * tol


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-8), ("mixed", 1e-6)])
@pytest.mark.parametrize("count", [10, 40])
def test_near_lists(engine, precision, tol, count):
    from pyfacc import geometry as G
    compare(engine, G.water_clusters(count, 5, 3, 16), precision, tol)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-8), ("mixed", 1e-6)])
def test_far_lists(engine, precision, tol):
    from pyfacc import geometry as G
    compare(engine, [G.alkane(10 + i, seed=i) for i in range(11)], precision, tol)


def test_deep_contractions(engine):
    from pyfacc import geometry as G
    compare(engine, G.water_clusters(24, 9, 6, 10), "fp64", 1e-8, basis="sto-6g")
