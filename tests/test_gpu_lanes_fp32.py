"""All-FP32 builds of lists too short for one lane per quartet (the coarse
iterations of a mixed SCF), against one lane per quartet (tasks of 16 kets)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,basis,prims", [("water", 1, "sto-3g", 3), ("water", 3, "sto-2g", 2),
                                                ("water", 9, "sto-4g", 4), ("water", 2, "sto-6g", 6),
                                                ("alkane", 3, "sto-6g", 6)])
def test_shared_fp32_quartets(engine, kind, n, basis, prims):
    import torch
    from pyfacc import geometry as G
    sp, xyz = G.water_cluster(n, np.random.default_rng(n)) if kind == "water" else G.alkane(n, seed=n)
    mol = engine.Molecule(sp, xyz, basis)
    with engine.System(mol) as s, engine.System(mol, task_width=16) as r:
        D = torch.tensor(np.random.default_rng(1).standard_normal((s.nbf, s.nbf)), device="cuda")
        D = 0.3 * (D + D.T)
        J, K = s.jk(D, precision="fp32")
        Jr, Kr = r.jk(D, precision="fp32")
    # either sums prims^4 terms a quartet in another order: each is off by
    # prims^2 roundings of 2^-24 of the largest
    tol = 2 * prims ** 2 * 2.0 ** -24
    assert (J - Jr).abs().max().item() <= tol * Jr.abs().max().item()
    assert (K - Kr).abs().max().item() <= tol * Kr.abs().max().item()
