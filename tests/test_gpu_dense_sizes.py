"""The dense products and the TC2 purification at the sizes where the kernel
changes: one block up to 72 rows, 16 x 16 tiles, 32 x 32 tiles from 400 rows;
whole and ragged 8-, 16- and 32-wide tiles on both sides of each line."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-12  # relative to the largest |C|, as in the products' other tests


@pytest.mark.parametrize("m,n,k", [(399, 399, 399), (400, 400, 400), (401, 433, 65), (416, 416, 31), (450, 400, 1)])
@pytest.mark.parametrize("ta,tb", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_products_around_the_tile_change(engine, m, n, k, ta, tb):
    import torch
    from pyfacc import _native as N
    g = torch.Generator(device="cuda").manual_seed(m + 3 * n + 7 * k)
    A = torch.randn((k, m) if ta else (m, k), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn((n, k) if tb else (k, n), dtype=torch.float64, device="cuda", generator=g)
    C = torch.full((m, n), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert N.lib().pyfacc_dense_gemm_dev(m, n, k, ta, A.data_ptr(), tb, B.data_ptr(), C.data_ptr(), 0, 0) == 0
    ref = (A.T if ta else A) @ (B.T if tb else B)
    assert ((C - ref).abs().max() / ref.abs().max()).item() < TOL


@pytest.mark.parametrize("n", [400, 417])
def test_symmetric_and_commutator_products_in_large_tiles(engine, n):
    import torch
    from pyfacc import _native as N
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g)
    C = torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert N.lib().pyfacc_dense_gemm_dev(n, n, n, 0, A.data_ptr(), 1, A.data_ptr(), C.data_ptr(), 1, 0) == 0
    ref = A @ A.T
    assert (C - C.T).abs().max().item() == 0.0
    assert ((C - ref).abs().max() / ref.abs().max()).item() < TOL
    assert N.lib().pyfacc_dense_gemm_dev(n, n, n, 0, A.data_ptr(), 0, B.data_ptr(), C.data_ptr(), 0, 1) == 0
    ref = (A - A.T) @ B
    assert ((C - ref).abs().max() / ref.abs().max()).item() < TOL


@pytest.mark.parametrize("n,nocc", [(2, 1), (8, 3), (9, 8), (25, 12), (64, 20), (71, 50), (72, 36), (73, 36), (128, 5),
                                    (399, 180), (400, 200), (433, 210)])
def test_purification_at_the_kernel_changes(engine, n, nocc):
    import torch
    from pyfacc import _native as N
    g = torch.Generator(device="cuda").manual_seed(n + nocc)
    Q, _ = torch.linalg.qr(torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g))
    lev = torch.cat([-0.2 - 20 * torch.rand(nocc, dtype=torch.float64, device="cuda", generator=g),
                     0.3 + 5 * torch.rand(n - nocc, dtype=torch.float64, device="cuda", generator=g)])
    F = (Q * lev) @ Q.T
    F = 0.5 * (F + F.T)
    P = torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda")
    steps = ctypes.c_int(0)
    torch.cuda.synchronize()
    assert N.lib().pyfacc_purify_dev(n, nocc, F.data_ptr(), P.data_ptr(), ctypes.byref(steps)) == 0
    _, V = torch.linalg.eigh(F)
    ref = V[:, :nocc] @ V[:, :nocc].T
    assert (P - ref).abs().max().item() < 1e-10
    assert abs(torch.trace(P).item() - nocc) < 1e-10
    assert 2 <= steps.value < 200
