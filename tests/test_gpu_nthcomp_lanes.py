"""nthcomp: the shortest systems (kTe near the seed temperature), the longest, lengths that leave lanes of the last
four points or chunks empty, and the same numbers by one CTA per continuum and by four lanes per continuum."""
import numpy as np
import pytest

import oracle_lib
from tolerance import assert_close

pytestmark = pytest.mark.gpu

GRID = np.exp(np.linspace(np.log(0.1), np.log(200.0), 301))


@pytest.mark.parametrize("kte", [5.0, 5.2, 5.4, 20.0, 60.0, 61.5, 100.0, 400.0, 3000.0])
@pytest.mark.parametrize("gamma", [1.2, 2.0, 3.4])
def test_against_oracle(gpu, oracle, kte, gamma):
    p = gpu.default_params("xillverCp")
    p[0], p[2], p[7] = gamma, kte, 1.0
    out, st = gpu.eval_batch("xillverCp", [p], [GRID])
    st1, ref = oracle_lib.evaluate("xillverCp", p, GRID)
    assert st[0] == st1 == 0
    assert_close(out[0], ref, f"kTe {kte} Gamma {gamma}")


@pytest.mark.parametrize("n", [1400, 15000, 30000])  # four, two and one lanes per continuum
def test_few_and_many(gpu, n):
    p = np.tile(gpu.default_params("xillverCp"), (n, 1))
    p[:, 2] = np.linspace(5.0, 400.0, n)
    p[:, 7] = 1.0
    grid = GRID[::60]
    many, st = gpu.eval_batch("xillverCp", p, [grid] * n)
    assert not st.any()
    for i in (0, 1, 700, n // 2, n - 1):
        few, _ = gpu.eval_batch("xillverCp", p[i:i + 1], [grid])
        assert np.array_equal(few[0], many[i])
