"""Memory that holds a calculation but not the transposed records of the split
kernels: the undivided kernels take over, with the same result.  Each run is a
process of its own that first fills the GPU up to a given rest.  The molecule:
a chain beside a helium atom of 24 primitives, whose pair makes the records
(a row for each of its 576 primitive pairs, for every pair of the class) ten
times as large as all the rest.  The batch: its records fit but leave little, or nothing
for the matrices, or do not fit, or would be larger than they may be."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import PKG, basis_file

pytestmark = pytest.mark.gpu
MB = 2 ** 20

CHILD = r"""
import json, sys
import numpy as np
import torch
import pyfacc
from pyfacc import _native as N
from pyfacc import geometry as G
kind, rest, data = sys.argv[1], int(sys.argv[2]), sys.argv[3]
pyfacc.run(pyfacc.Molecule(*G.water()))
if kind == "system":
    sp, x = G.alkane(50, seed=3)
    mol = pyfacc.Molecule(sp + ["He"], np.vstack([x, x.max(0) + 4.0]), "deep")
    job = lambda: [pyfacc.run(mol, data_dir=data)]
else:
    mols = [pyfacc.Molecule(s, x) for s, x in G.water_clusters(120, 5, 14, 18)]
    job = lambda: pyfacc.run_batch(mols)
if rest:
    fill = torch.empty(torch.cuda.mem_get_info()[0] - rest, dtype=torch.uint8, device="cuda")
try:
    out = [r.energy for r in job()]
except pyfacc.PyfaccError as e:
    assert "out of memory" in str(e), e
    out = None
print(json.dumps([out, N.lib().pyfacc_split_launch_count(0)]))
"""


def _run(kind, rest_mb, data="-"):
    env = dict(os.environ, PYTHONPATH=PKG)
    p = subprocess.run([sys.executable, "-c", CHILD, kind, str(rest_mb * MB), data], env=env, capture_output=True,
                       text=True, timeout=120)
    assert p.returncode == 0, p.stderr[-2000:]
    return json.loads(p.stdout.strip().splitlines()[-1])


def _deep_helium(folder):
    """STO-3G with a helium of 24 primitives, as the basis "deep" in folder."""
    (folder / "basis_set").mkdir()
    a = np.geomspace(2000.0, 0.1, 24)
    c = np.exp(-0.5 * ((np.log(a) - 0.5) / 1.5) ** 2)
    text = open(basis_file("sto-3g")).read()
    lo = text.index("He     0")
    hi = text.index("****", lo)
    rows = "".join(f"  {x:.10E}  {y:.10E}\n" for x, y in zip(a, c / c.sum()))
    (folder / "basis_set" / "deep.txt").write_text(text[:lo] + "He     0\nS   24   1.00\n" + rows + text[hi:])


def test_one_molecule(engine, tmp_path):
    _deep_helium(tmp_path)
    plenty, split = _run("system", 0, str(tmp_path))
    short, none = _run("system", 320, str(tmp_path))
    assert split > 0 and none == 0
    assert short is not None, "out of memory without need"
    assert short[0] == pytest.approx(plenty[0], abs=1e-8)


def test_batch(engine):
    plenty, split = _run("batch", 0)
    assert split > 0
    for rest in (1300, 950, 800):
        out, undivided = _run("batch", rest)
        assert undivided == 0 and out is not None
        assert np.abs(np.array(out) - np.array(plenty)).max() < 1e-8


def test_records_beyond_their_limit(engine, tmp_path):
    """48 clusters with a helium of 24 primitives each: the batch's records
    would take more than 4 GB, half of them less."""
    from pyfacc import _native as N
    from pyfacc import geometry as G
    _deep_helium(tmp_path)
    mols = [engine.Molecule(list(s) + ["He"], np.vstack([x, x.max(0) + 6.0]), "deep")
            for s, x in G.water_clusters(48, 5, 16, 16)]

    def run(ms):
        before = N.lib().pyfacc_split_launch_count(0)
        return [r.energy for r in engine.run_batch(ms, data_dir=str(tmp_path))], N.lib().pyfacc_split_launch_count(0) - before

    whole, none = run(mols)
    half, split = run(mols[:24])
    assert split > 0 and none == 0
    assert np.abs(np.array(whole[:24]) - np.array(half)).max() < 1e-8
