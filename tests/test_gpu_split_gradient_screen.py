"""The split kernels' gradient takes the quartets that the undivided ones take:
at a loose screening threshold, where a quartet more or less shows, the two
gradients of a batch (its explicit task width is for the undivided kernels)
agree far below the threshold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_same_quartets_at_a_loose_threshold(engine):
    from pyfacc import _native as N
    from pyfacc import geometry as G
    mols = [engine.Molecule(s, x) for s, x in G.water_clusters(40, 5, 6, 16)]
    thresh = 1e-8
    before = N.lib().pyfacc_split_launch_count(0)
    a = engine.run_batch(mols, gradient=False, schwarz_thresh=thresh)
    build = N.lib().pyfacc_split_launch_count(0) - before
    a = engine.run_batch(mols, gradient=True, schwarz_thresh=thresh)
    assert N.lib().pyfacc_split_launch_count(0) - before > 2 * build > 0, "the gradient was not split"
    b = engine.run_batch(mols, gradient=True, schwarz_thresh=thresh, task_width=32)
    # the densities agree to the builds' 1e-11; a quartet at the threshold adds
    # up to 1e-8 times its density factors
    for x, y in zip(a, b):
        assert np.abs(x.gradient - y.gradient).max() < 1e-2 * thresh
