"""Emission-angle histograms for relline tables with fewer and more g* points than the usual 40 (lanes without
points, eight points per lane), against the oracle on the same tables."""
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
e = np.exp(np.linspace(np.log(0.5), np.log(50.0), 201))
for model in ("relxill", "relxilllp"):
    for spin, incl in ((0.3, 25.0), (0.97, 70.0)):
        p = R.default_params(model)
        names = [k for k, _ in R.PARAMS[model]]
        p[names.index("a")], p[names.index("Incl")] = spin, incl
        out, st = R.eval_batch(model, [p], [e])
        st1, ref = oracle_lib.evaluate(model, p, e)
        assert st[0] == st1 == 0
        assert_close(out[0], ref, f"{model} a {spin} incl {incl}")
"""


@pytest.mark.parametrize("points", [20, 33, 64])
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
