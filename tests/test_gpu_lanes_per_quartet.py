"""J/K lists too short for one lane per quartet: 16, 4 and 1 lanes share a
quartet's primitives depending on the list's length.  Tasks of 16 kets keep
one lane per quartet, so the same molecule with task_width=16 is the
reference; 4, 9, 16 and 36 primitive pairs per shell pair do not divide evenly
among the lanes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,basis", [("water", 1, "sto-3g"), ("water", 3, "sto-2g"), ("water", 6, "sto-3g"),
                                          ("water", 9, "sto-4g"), ("water", 2, "sto-6g"), ("alkane", 3, "sto-6g")])
def test_shared_quartets_match_one_lane_each(engine, kind, n, basis):
    import torch
    from pyfacc import geometry as G
    sp, xyz = G.water_cluster(n, np.random.default_rng(n)) if kind == "water" else G.alkane(n, seed=n)
    mol = engine.Molecule(sp, xyz, basis)
    with engine.System(mol) as s, engine.System(mol, task_width=16) as r:
        D = torch.tensor(np.random.default_rng(1).standard_normal((2, s.nbf, s.nbf)), device="cuda")
        D = 0.3 * (D + D.transpose(1, 2))
        for nk in (1, 2):
            Dk = D[0] if nk == 1 else D
            for precision, rel in (("fp64", 1e-13), ("mixed", 2.0 ** -22)):
                # FP64: sums of up to 1296 primitives in another order; mixed:
                # its FP32 quartets, too, in another order
                J, K = s.jk(D[0], Dk, precision=precision)
                Jr, Kr = r.jk(D[0], Dk, precision=precision)
                assert (J - Jr).abs().max().item() <= rel * Jr.abs().max().item(), precision
                assert (K - Kr).abs().max().item() <= rel * Kr.abs().max().item(), precision
