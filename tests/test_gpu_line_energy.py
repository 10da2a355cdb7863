"""The line's energy grid e / lineE from a reciprocal: ordinary line energies, and ones whose reciprocal or quotient
overflows or vanishes, against the oracle's division."""
import numpy as np
import pytest

import oracle_lib
from tolerance import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("line", [1.0, 6.4, 6.69999, 0.5, 1e-3, 300.0, 1e-310, 1e308])
def test_line_energy(gpu, oracle, line):
    p = gpu.default_params("relline")
    p[0] = line
    scale = line if 1e-3 <= line <= 300.0 else 6.4
    e = scale * np.exp(np.linspace(np.log(0.05), np.log(1.5), 301))
    out, st = gpu.eval_batch("relline", [p], [e], check=False)
    st1, ref = oracle_lib.evaluate("relline", p, e)
    assert st[0] == st1
    if scale == line:
        assert_close(out[0], ref, f"lineE {line}")
    else:  # no bin of the grid is reached
        assert np.array_equal(np.isfinite(out[0]), np.isfinite(ref)) and not np.nan_to_num(out[0]).any()
