"""The convolution's tiles and sums: grids of one bin up to several tiles of 16 conv bins, at the ends of the
0.01-1000 keV band (where the windows of the normalisation leave it) and inside, narrow and wide profiles."""
import numpy as np
import pytest

import oracle_lib
from tolerance import assert_close

pytestmark = pytest.mark.gpu

SPANS = [(1, 6.0, 6.02), (2, 0.3, 0.31), (15, 1.0, 1.1), (17, 6.3, 6.75), (33, 90.0, 110.0), (64, 0.011, 0.03),
         (64, 600.0, 990.0), (300, 0.008, 1200.0)]


@pytest.mark.parametrize("rin,rout", [(-1.0, 400.0), (60.0, 90.0)])
@pytest.mark.parametrize("bins,lo,hi", SPANS)
def test_conv_tiles(gpu, oracle, bins, lo, hi, rin, rout):
    e = np.exp(np.linspace(np.log(lo), np.log(hi), bins + 1))
    line = [3.0, 3.0, 15.0, 0.9, 30.0, rin, rout, 0.0]
    jobs = [("relconv", line, np.linspace(1.0, 2.0, bins))]
    if lo > 0.1 and hi < 200.0:  # inside the reflection table's range
        jobs.append(("relxill", line + [2.0, 2.0, 1.0, 300.0, 1.0], None))
    for model, p, f in jobs:
        out, st = gpu.eval_batch(model, [p], [e], flux_in=None if f is None else [f])
        assert not st.any()
        st1, ref = oracle_lib.evaluate(model, p, e, f)
        assert st1 == 0
        assert_close(out[0], ref, f"{model} {bins} bins {lo}-{hi} keV")
