"""relconv on grids whose last edge is an edge of the convolution grid: the conv bin above holds nothing of the caller's
spectrum, of the set that follows or of an earlier call."""
import numpy as np
import pytest

import oracle_lib
from tolerance import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("step", [1, 16, 37])
@pytest.mark.parametrize("last", [2200, 2777, 3300])
def test_last_edge_on_conv_edge(gpu, oracle, last, step):
    ce = oracle_lib.conv_grid()
    e = ce[last - 40 * step:last + 1:step].copy()
    above = ce[last:last + 40 * step + 1:step].copy()  # the next set's grid starts where this one ends
    f, g = np.linspace(3.0, 1.0, len(e) - 1), np.linspace(1.0, 2.0, len(above) - 1)
    p = gpu.default_params("relconv")
    # an earlier call leaves large values in the staging
    gpu.eval_batch("relconv", [p] * 2, [e, above], [1e6 * f, 1e6 * g])
    two, st = gpu.eval_batch("relconv", [p] * 2, [e, above], [f, g])
    one, st1 = gpu.eval_batch("relconv", [p], [e], [f])
    assert not st.any() and not st1.any()
    assert np.array_equal(two[0], one[0])
    # an ulp below the conv edge the two grids do not meet: the same spectrum up to its rounding to FP32
    below = e.copy()
    below[-1] = np.nextafter(e[-1], 0.0)
    near, _ = gpu.eval_batch("relconv", [p], [below], [f])
    np.testing.assert_allclose(one[0], near[0], rtol=1e-6)
    st2, ref = oracle_lib.evaluate("relconv", p, below, f)
    assert st2 == 0
    assert_close(one[0], ref, f"last conv edge {last} step {step}")
