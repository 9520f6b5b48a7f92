"""A molecule far from the origin: the split kernels test distances in float,
where coordinates of 1e8 bohr lie 8 bohr apart.  J and K against the undivided
kernels' for the same coordinates."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [1e3, 1e8])
def test_split_kernels_far_from_the_origin(engine, offset):
    import torch
    from pyfacc import _native as N
    from pyfacc import geometry as G
    sp, xyz = G.alkane(26, seed=26)
    mol = engine.Molecule(sp, xyz + offset * np.array([1.0, -0.7, 0.4]))
    rng = np.random.default_rng(1)
    with engine.System(mol) as s:
        d = rng.standard_normal((s.nbf, s.nbf))
        D = torch.tensor(0.3 * (d + d.T), device="cuda")
        before = N.lib().pyfacc_split_launch_count(1)
        J, K = s.jk(D)
        assert N.lib().pyfacc_split_launch_count(1) > before
    m, keep = mol._struct()
    Jr, Kr = torch.empty_like(D), torch.empty_like(D)
    torch.cuda.synchronize()
    assert N.lib().pyfacc_jk_noalloc(ctypes.byref(m), N.DATA_DIR.encode(), 1e-12, D.data_ptr(), Jr.data_ptr(),
                                     Kr.data_ptr()) == N.OK
    # a product centre P = (a A + b B) / p is rounded to 2^-53 |A| and a
    # quartet's value has a derivative of the order of itself: 1e-10 as
    # elsewhere, or four such roundings of the largest element
    for a, b in ((J, Jr), (K, Kr)):
        assert (a - b).abs().max().item() < 1e-10 + 4 * 2.0 ** -53 * offset * b.abs().max().item()
