"""Limb laws on grids whose tiles of 32 bins reach a few of the g* points, all of them, and the edge terms of either end,
for even, odd and the most points, against the oracle on the same tables."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import sys
import numpy as np
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
import oracle_lib
import relxill_gb300 as R
from tolerance import assert_close
oracle_lib.lib(sys.argv[2])
R.init(sys.argv[2])
log = lambda lo, hi, n: np.exp(np.linspace(np.log(lo), np.log(hi), n + 1))
grids = [log(0.5, 12.0, 5000), log(5.0, 7.5, 1500), log(0.5, 12.0, 65), log(0.3, 80.0, 1000), log(0.5, 12.0, 31)]
for model in ("relline", "relconv"):
    names = [k for k, _ in R.PARAMS[model]]
    for limb in (1, 2):
        p = np.tile(R.default_params(model), (len(grids), 1))
        p[:, names.index("limb")] = limb
        p[:, names.index("a")] = (0.998, 0.3, 0.7, -0.4, 0.9)
        p[:, names.index("Incl")] = (70.0, 20.0, 45.0, 33.0, 84.0)
        flux = [np.linspace(1.0, 2.0, len(e) - 1) for e in grids] if model == "relconv" else None
        out, st = R.eval_batch(model, p, grids, flux)
        for i, e in enumerate(grids):
            st1, ref = oracle_lib.evaluate(model, p[i], e, None if flux is None else flux[i])
            assert st[i] == st1 == 0
            assert_close(out[i], ref, f"{model} law {limb} grid {i}")
"""


@pytest.mark.parametrize("points", [20, 39, 40, 61, 64])
def test_points(small_tables, tmp_path, points):
    from relxill_gb300 import synth_tables

    d = tmp_path / "tables"
    d.mkdir()
    for f in os.listdir(small_tables):
        if not f.startswith("rel_table"):
            os.symlink(os.path.join(small_tables, f), d / f)
    name = next(f for f in os.listdir(small_tables) if f.startswith("rel_table"))
    synth_tables.write_relline_table(str(d / name), n_a=5, n_mu0=6, n_g=points)
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", CHILD, root, str(d)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, RELXILL_TABLE_PATH=str(d)))
    assert r.returncode == 0, r.stderr[-2000:]
