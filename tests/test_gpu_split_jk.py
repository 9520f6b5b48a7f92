"""The split J/K kernels (far and near quartets of long lists apart) against
the undivided ones.

``pyfacc_jk_noalloc`` builds J and K with the undivided kernels only; a
System of an extended molecule takes the split ones, which shows in the number
of kernels a build launches.  Chains long enough for it, with 4, 9 and 36
primitive pairs per shell pair (an even and an odd bra count for the packed
FP32 pairs, and a staged bra larger than a warp), one and two exchange
densities, densities that leave the far quartets to J alone (local) or give
them to K too (spread).
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL64 = 1e-10   # the J/K tolerance of the FP64 parity tests
TOLMIX = 1e-7   # and of the mixed ones


def _noalloc(engine, mol, D):
    import torch
    from pyfacc import _native as N
    m, keep = mol._struct()
    J, K = torch.empty_like(D), torch.empty_like(D)
    torch.cuda.synchronize()
    st = N.lib().pyfacc_jk_noalloc(ctypes.byref(m), N.DATA_DIR.encode(), 1e-12, D.data_ptr(), J.data_ptr(), K.data_ptr())
    assert st == N.OK, N.lib().pyfacc_last_message()
    return J, K


def _density(n, reach, seed):
    """Symmetric, decaying over `reach` basis functions of the chain's order."""
    import torch
    rng = np.random.default_rng(seed)
    i = np.arange(n)
    d = rng.standard_normal((n, n)) * np.exp(-np.abs(i[:, None] - i[None, :]) / reach)
    return torch.tensor(0.3 * (d + d.T), device="cuda")


@pytest.mark.parametrize("n,basis,reach", [(26, "sto-3g", 3.0), (26, "sto-3g", 200.0), (30, "sto-2g", 3.0),
                                           (22, "sto-6g", 10.0)])
def test_split_matches_undivided(engine, n, basis, reach):
    import torch
    from pyfacc import _native as N
    from pyfacc import geometry as G
    mol = engine.Molecule(*G.alkane(n, seed=n), basis)
    with engine.System(mol) as s:
        Da, Db = _density(s.nbf, reach, 1), _density(s.nbf, reach, 2)
        before = N.lib().pyfacc_launch_count()
        J, K = s.jk(Da)
        launches = N.lib().pyfacc_launch_count() - before
        Jr, Kr = _noalloc(engine, mol, Da)
        assert launches > 9, "no list of this molecule was split"  # undivided: 6 classes, density bound, symmetrising
        assert (J - Jr).abs().max().item() < TOL64
        assert (K - Kr).abs().max().item() < TOL64
        # two exchange densities, J of their sum
        J2, K2 = s.jk(Da + Db, torch.stack([Da, Db]))
        Jb, Kb = _noalloc(engine, mol, Db)
        assert (J2 - Jr - Jb).abs().max().item() < TOL64
        assert (K2[0] - Kr).abs().max().item() < TOL64
        assert (K2[1] - Kb).abs().max().item() < TOL64
        Jm, Km = s.jk(Da, precision="mixed")
        assert (Jm - Jr).abs().max().item() < TOLMIX
        assert (Km - Kr).abs().max().item() < TOLMIX
        # every quartet in FP32: a few units in the last place of the largest element
        Jf, Kf = s.jk(Da, precision="fp32")
        assert (Jf - Jr).abs().max().item() < 2.0 ** -20 * Jr.abs().max().item()
        assert (Kf - Kr).abs().max().item() < 2.0 ** -20 * Kr.abs().max().item()


def test_split_matches_oracle(engine, oracle):
    from pyfacc import geometry as G
    from conftest import basis_file
    sp, xyz = G.alkane(24, seed=9)
    mol = engine.Molecule(sp, xyz)
    om = oracle.molecule(sp, xyz, basis_file("sto-3g"))
    with engine.System(mol) as s:
        D = _density(s.nbf, 6.0, 4)
        J, K = s.jk(D)
    Jo, Ko = oracle.jk(om, D.cpu().numpy())
    assert np.abs(J.cpu().numpy() - Jo).max() < TOL64
    assert np.abs(K.cpu().numpy() - Ko).max() < TOL64
