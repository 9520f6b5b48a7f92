"""Which calls take the kernels for long quartet lists, on either side of each
line (the launch counters tell), and their lists divided over shards."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _split(f):
    """(near, far) launches of the split kernels in f()."""
    from pyfacc import _native as N
    before = [N.lib().pyfacc_split_launch_count(h) for h in (0, 1)]
    out = f()
    return out, tuple(N.lib().pyfacc_split_launch_count(h) - b for h, b in zip((0, 1), before))


def test_batches(engine):
    from pyfacc import geometry as G
    waters = [engine.Molecule(s, x) for s, x in G.water_clusters(40, 5, 3, 16)]
    chains = [engine.Molecule(*G.alkane(10 + i, seed=i)) for i in range(11)]
    deep = [engine.Molecule(s, x, "sto-6g") for s, x in G.water_clusters(24, 9, 6, 10)]
    for precision in ("fp64", "mixed"):
        _, (near, far) = _split(lambda: engine.run_batch(waters, precision=precision))
        assert near > 0 and far == 0
        assert _split(lambda: engine.run_batch(waters, precision=precision, gradient=True))[1] == (near, 0)
        _, (near, far) = _split(lambda: engine.run_batch(chains, precision=precision))
        assert near > 0 and far > 0
        assert _split(lambda: engine.run_batch(waters, precision=precision, gradient=True, task_width=32))[1] == (0, 0)
        assert _split(lambda: engine.run_batch(waters[:3], precision=precision, gradient=True))[1] == (0, 0)
    assert _split(lambda: engine.run_batch(deep))[1][0] > 0


@pytest.mark.parametrize("precision", ["fp64", "mixed", "fp32"])
def test_builds(engine, precision):
    import torch
    from pyfacc import geometry as G
    for n, long in ((26, True), (4, False)):
        with engine.System(engine.Molecule(*G.alkane(n, seed=n))) as s:
            D = torch.eye(s.nbf, dtype=torch.float64, device="cuda")
            _, (near, far) = _split(lambda: s.jk(D, precision=precision))
        assert (near > 0 and far == near) if long else (near, far) == (0, 0)


@pytest.mark.parametrize("open_shell", [False, True])
def test_gradients(engine, open_shell):
    from pyfacc import geometry as G
    make = G.radical if open_shell else G.alkane
    # FP64 lists from 3e5 far quartets, FP32 lists from 6e5
    for n, precision, long in ((24, "fp64", True), (32, "mixed", True), (18, "mixed", False), (6, "fp64", False)):
        with engine.System(engine.Molecule(*make(n, seed=n)), precision=precision) as s:
            s.scf()
            g, (near, far) = _split(s.gradient)
        assert (near > 0 and far == near) if long else (near, far) == (0, 0), (n, precision)


def test_shards_of_split_lists(engine):
    """Three shards' partial J and K add up to the whole."""
    import torch
    from pyfacc import geometry as G
    mol = engine.Molecule(*G.alkane(30, seed=30))
    rng = np.random.default_rng(4)
    with engine.System(mol) as s:
        d = rng.standard_normal((s.nbf, s.nbf))
        D = torch.tensor(0.3 * (d + d.T), device="cuda")
        whole = {p: s.jk(D, precision=p) for p in ("fp64", "mixed")}
    for precision, (J, K) in whole.items():
        Jt, Kt = torch.zeros_like(J), torch.zeros_like(K)
        for rank in range(3):
            with engine.System(mol, shard_rank=rank, shard_count=3) as s:
                (Jp, Kp), (near, far) = _split(lambda: s.jk(D, precision=precision))
            assert near > 0 and far == near
            Jt += Jp
            Kt += Kp
        # the whole's mixed lists follow the density, the shards' the Schwarz factors alone: the J/K tolerances
        tol = 1e-10 if precision == "fp64" else 1e-7
        assert (Jt - J).abs().max().item() < tol
        assert (Kt - K).abs().max().item() < tol


def test_sharded_gradient_of_split_lists(engine):
    from pyfacc import geometry as G
    from pyfacc.distributed import attach_reducer
    from test_distributed import _HostSum
    mol = engine.Molecule(*G.alkane(24, seed=24))
    ref = engine.run(mol, gradient=True)
    hs, results = _HostSum(2), {}

    def shard(rank):
        s = engine.System(mol, shard_rank=rank, shard_count=2)

        class R:
            cb = hs.make(rank)
        attach_reducer(s, R())
        results[rank] = (s.scf().energy, s.gradient())
        s.close()

    def run():
        th = [threading.Thread(target=shard, args=(r,)) for r in range(2)]
        for t in th:
            t.start()
        for t in th:
            t.join()

    _, (near, far) = _split(run)
    assert near > 0 and far == near
    for rank in range(2):
        assert results[rank][0] == pytest.approx(ref.energy, abs=1e-9)
        assert np.abs(results[rank][1] - ref.gradient).max() < 1e-8


def test_deep_contractions_split_fp64_lists_later(engine):
    """STO-6G: between the lines of FP32 and FP64 lists, and above both."""
    import torch
    from pyfacc import geometry as G
    for n, fp64 in ((17, False), (24, True)):
        with engine.System(engine.Molecule(*G.alkane(n, seed=n), "sto-6g")) as s:
            D = torch.eye(s.nbf, dtype=torch.float64, device="cuda")
            (J, K), (near, _) = _split(lambda: s.jk(D))
            assert (near > 0) == fp64
            for precision in ("fp32", "mixed"):
                (Jf, Kf), (near, far) = _split(lambda: s.jk(D, precision=precision))
                assert precision == "mixed" or near == far > 0
                # 36 roundings of 2^-24 of the largest element (1296 primitive quartets)
                assert (Jf - J).abs().max().item() < 36 * 2.0 ** -24 * J.abs().max().item()
                assert (Kf - K).abs().max().item() < 36 * 2.0 ** -24 * K.abs().max().item()


def test_lists_that_come_and_go_with_the_geometry(engine):
    """One handle through a stretched chain, a coiled-up one without far
    quartets and the first again: the records are made anew each time."""
    import torch
    from pyfacc import geometry as G
    sp, xyz = G.alkane(26, seed=26)
    # the same chain wound up: a helix of 4 bohr radius
    c = xyz - xyz.mean(0)
    t, u, v = (c @ np.linalg.svd(c)[2].T).T
    coil = np.stack([(4.0 + u) * np.cos(t / 4.0), (4.0 + u) * np.sin(t / 4.0), t / 4.0 + v], 1)
    mol = engine.Molecule(sp, xyz)
    with engine.System(mol) as s:
        d = np.random.default_rng(3).standard_normal((s.nbf, s.nbf))
        D = torch.tensor(0.3 * (d + d.T), device="cuda")
        first, far0 = _split(lambda: s.jk(D))
        s.set_coords(coil)
        wound, far1 = _split(lambda: s.jk(D))
        s.set_coords(xyz)
        again, far2 = _split(lambda: s.jk(D))
    with engine.System(engine.Molecule(sp, coil)) as s:
        ref = s.jk(D)
    assert far0[1] > 0 and far1 == (0, 0) and far2 == far0
    for x, y in ((first, again), (wound, ref)):
        for m, n in zip(x, y):
            assert (m - n).abs().max().item() < 1e-12 * n.abs().max().item()
