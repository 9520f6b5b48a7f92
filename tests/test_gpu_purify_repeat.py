"""The one-block purification gives the same projector, bit for bit, in the
same number of steps every time: its sums over the block run in a fixed order,
so a trace read while another step's is being written would show.  One warp, a
few warps, and the most (72 rows), with the GPU idle and with it kept busy by
other work."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 9, 24, 40, 56, 72])
@pytest.mark.parametrize("busy", [False, True])
def test_repeats_are_identical(engine, n, busy):
    import torch
    from pyfacc import _native as N
    g = torch.Generator(device="cuda").manual_seed(n)
    F = torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g)
    F = F + F.T
    ref, first = None, None
    load = torch.randn((2048, 2048), device="cuda", generator=g)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(150):
        if busy:
            with torch.cuda.stream(side):
                load @ load
        P = torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda")
        steps = ctypes.c_int(0)
        torch.cuda.current_stream().synchronize()
        assert N.lib().pyfacc_purify_dev(n, n // 2, F.data_ptr(), P.data_ptr(), ctypes.byref(steps)) == 0
        if ref is None:
            ref, first = P, steps.value
            assert abs(torch.trace(P).item() - n // 2) < 1e-10
        assert steps.value == first
        assert torch.equal(P, ref)
