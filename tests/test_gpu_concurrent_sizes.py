"""Systems of different sizes in several threads: a kernel's allowance of
shared memory is one value per device, and one thread's launch must not lower
it under another's (one-block purifications of 50 to 72 functions, and the
dense steps of batches of small and large molecules)."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _together(*jobs):
    errors = []

    def guard(job):
        try:
            job()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=guard, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_purifications(engine):
    import torch
    from pyfacc import _native as N

    def job(n):
        g = torch.Generator(device="cuda").manual_seed(n)
        F = torch.randn((n, n), dtype=torch.float64, device="cuda", generator=g)
        F = F + F.T
        P = torch.empty_like(F)
        torch.cuda.synchronize()

        def run():
            for _ in range(1500):
                st = N.lib().pyfacc_purify_dev(n, n // 2, F.data_ptr(), P.data_ptr(), ctypes.byref(ctypes.c_int(0)))
                assert st == N.OK, (n, N.lib().pyfacc_last_message())
        return run

    _together(*[job(n) for n in (72, 50, 72, 56)])


def test_batches(engine):
    from pyfacc import geometry as G
    large = [engine.Molecule(s, x) for s, x in G.water_clusters(2, 5, 18, 20)]
    small = [engine.Molecule(s, x) for s, x in G.water_clusters(3, 7, 1, 2)]
    alone = {id(m): [r.energy for r in engine.run_batch(m)] for m in (large, small)}

    def job(mols, count):
        def run():
            for _ in range(count):
                e = [r.energy for r in engine.run_batch(mols)]
                assert np.abs(np.array(e) - alone[id(mols)]).max() < 1e-9
        return run

    _together(job(large, 12), job(small, 60))
