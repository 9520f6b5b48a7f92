"""The functions that stand in for the Boys function, 1/sqrt and exp in the
split kernels, value by value: the short table and the far limit against the
mpmath fixture and the oracle (which is pinned to it), the reciprocal square
root and the exponential against CUDA's."""
import json
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")
EPS = 2.0 ** -52


def _values(what, fp32, L, x):
    import torch
    from pyfacc import _native as N
    N.lib()
    xd = torch.tensor(np.asarray(x, dtype=np.float64), device="cuda")
    out = torch.full((len(x), L + 1), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert N.lib().pyfacc_split_values_dev(what, fp32, L, len(x), xd.data_ptr(), out.data_ptr()) == N.OK
    return out.cpu().numpy()


def _fixture():
    ref = json.load(open(os.path.join(GOLDEN, "boys_mpmath.json")))["values"]
    return sorted({x for _, x, _ in ref}), {(m, x): v for m, x, v in ref}


@pytest.mark.parametrize("L", range(5))
def test_table_fp64(engine, L):
    # F_L: 13 coefficients, rounded once each and summed with falling weights,
    # 2 eps, or 2 L + 2 roundings of the asymptote; three more a step downward
    xs, ref = _fixture()
    F = _values(0, 0, L, xs)
    for i, x in enumerate(xs):
        for m in range(L + 1):
            assert F[i, m] == pytest.approx(ref[m, x], rel=(2 * L + 2 + 3 * (L - m)) * EPS, abs=0), (m, x)


@pytest.mark.parametrize("L", range(5))
def test_table_fp64_between_its_points(engine, oracle, L):
    # every interval of the table, its ends and the change to the asymptote;
    # the oracle adds its own 1e-14 (test_boys_accurate_vs_mpmath_fixture)
    h = (36.0 + 3 * L) / 31.5
    xs = np.concatenate([np.linspace(0, 33 * h, 997), (np.arange(32) + 0.5) * h, (np.arange(32) + 0.5) * h - 1e-9])
    F = _values(0, 0, L, xs)
    for i, x in enumerate(xs):
        for m in range(L + 1):
            assert F[i, m] == pytest.approx(oracle.boys(m, float(x), 0), rel=2e-14), (m, x)


@pytest.mark.parametrize("L", range(5))
def test_table_fp32(engine, oracle, L):
    # 2^-24 a rounding: six coefficients, or the asymptote's 2 L + 1 factors of
    # rsqrt (two units in the last place), expf and three a step downward
    h = (17.0 + 3 * L) / 31.5
    xs = np.float32(np.concatenate([np.linspace(0, 33 * h, 499), (np.arange(32) + 0.5) * h, [50.0, 200.0, 1e4]]))
    F = _values(0, 1, L, xs)
    for i, x in enumerate(xs):
        for m in range(L + 1):
            tol = (8 + 4 * (2 * L + 1) + 8 * (L - m)) * 2.0 ** -24
            assert F[i, m] == pytest.approx(oracle.boys(m, float(x), 0), rel=tol), (m, x)


@pytest.mark.parametrize("fp32,eps,first", [(0, EPS, 36.0), (1, 2.0 ** -22, 17.0)])
@pytest.mark.parametrize("L", range(5))
def test_far_limit(engine, oracle, fp32, eps, first, L):
    # from its bound on: the neglected part (3e-16; 3e-8 in FP32), the square
    # root that makes |PQ| and 2 m + 1 reciprocal ones; the oracle's 1e-14
    t0 = first + 3 * L
    xs = np.concatenate([t0 * np.linspace(1.0, 1.3, 40), t0 * np.geomspace(1.3, 1e4, 40)])
    F = _values(1, fp32, L, xs)
    for i, x in enumerate(xs):
        for m in range(L + 1):
            tol = (3e-8 if fp32 else 1e-14) + (2 * (2 * m + 1) + 2) * eps
            assert F[i, m] == pytest.approx(oracle.boys(m, float(x), 0), rel=tol), (m, x)
    if not fp32:
        xs, ref = _fixture()
        xs = [x for x in xs if x >= t0]
        F = _values(1, 0, L, xs)
        for i, x in enumerate(xs):
            for m in range(L + 1):
                assert F[i, m] == pytest.approx(ref[m, x], rel=3e-16 + (2 * m + 2) * EPS, abs=0), (m, x)


def test_reciprocal_square_root(engine):
    import torch
    rng = np.random.default_rng(2)
    x = np.concatenate([1.0 + 3.0 * rng.random(200000), 10.0 ** rng.uniform(-290, 290, 50000)])
    y = _values(2, 0, 0, x)[:, 0]
    ref = torch.rsqrt(torch.tensor(x, device="cuda")).cpu().numpy()  # within one unit in the last place
    assert (np.abs(y - ref) <= 2 * EPS * ref).all()
    y = _values(2, 1, 0, np.float32(x[:200000]))[:, 0]
    assert (np.abs(y - ref[:200000]) <= 4 * 2.0 ** -23 * ref[:200000]).all()


def test_exponential(engine):
    import torch
    x = np.concatenate([np.linspace(0.0, 99.99, 200001), np.log(2.0) * (np.arange(144) + 0.5)])
    y = _values(3, 0, 0, x)[:, 0]
    ref = torch.exp(-torch.tensor(x, device="cuda")).cpu().numpy()  # within one unit in the last place
    # the reduced argument: 144 times the error of the two-part ln 2's product, half an eps; eleven falling terms
    assert (np.abs(y - ref) <= 3 * EPS * ref).all()
    assert (_values(3, 0, 0, [100.0, 1e3, 1e300])[:, 0] == 0.0).all()
