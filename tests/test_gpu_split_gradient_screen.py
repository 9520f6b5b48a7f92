"""The split kernels' gradient takes the quartets that the undivided ones take:
at a loose screening threshold, where a quartet more or less shows, a chain's
gradient from its own system (split) and from a batch of one (undivided) agree
far below the threshold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_same_quartets_at_a_loose_threshold(engine):
    from pyfacc import _native as N
    from pyfacc import geometry as G
    mol = engine.Molecule(*G.alkane(22, seed=22))
    opt = dict(schwarz_thresh=1e-8, eps_diis=1e-10)
    with engine.System(mol, **opt) as s:
        s.scf()
        before = [N.lib().pyfacc_split_launch_count(h) for h in (0, 1)]
        g = s.gradient()
        assert all(N.lib().pyfacc_split_launch_count(h) > b for h, b in zip((0, 1), before))
    ref = engine.run_batch([mol], gradient=True, task_width=32, **opt)[0].gradient
    # left out on one side only, a quartet at the threshold moves an atom by up
    # to 1e-8; the primitive cut is 1e-2 of it, and far pairs on one atom take
    # all their primitives at once, cut or not: ten of those
    assert np.abs(g - ref).max() < 1e-9
