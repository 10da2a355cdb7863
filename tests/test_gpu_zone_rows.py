"""xillver spectra of sets with more than 16 zones (or rows beyond the shared list): distinct rows read once
for all zones that name them.  Zone counts at the limits, both tables, gradients that spread the zones
over many brackets and none (every zone in the same bracket)."""
import numpy as np
import pytest

import oracle_lib
from tolerance import assert_close

pytestmark = pytest.mark.gpu

GRID = np.exp(np.linspace(np.log(0.3), np.log(60.0), 201))


@pytest.mark.parametrize("zones", [16, 17, 50])
@pytest.mark.parametrize("model,igt", [("relxilllp", 0), ("relxilllp", 1), ("relxilllp", 2), ("relxilllpCp", 0),
                                       ("relxilllpCp", 2)])
def test_zone_rows(gpu, oracle, monkeypatch, model, igt, zones):
    monkeypatch.setenv("RELXILL_NUM_RZONES", str(zones))
    rng = np.random.default_rng(zones + 7 * igt)
    if model == "relxilllp":
        p = [[rng.uniform(3, 20), 0.0, rng.uniform(0, 0.998), rng.uniform(10, 80), -1.0, 400.0, 0.0,
              rng.uniform(1.5, 2.7), rng.uniform(0.5, 4.4), rng.choice([1.0, 1.7]), rng.uniform(60, 400), 1.0, 0.0, 0.0]
             for _ in range(5)]
    else:
        p = [[rng.uniform(10, 80), rng.uniform(0, 0.998), -1.0, 400.0, rng.uniform(3, 20), 0.0, rng.uniform(1.5, 2.7),
              rng.uniform(0.5, 4.4), rng.uniform(15, 19), 1.0, rng.uniform(20, 200), 1.0, 0.0, 1.5, float(igt), 0.0, 0.0]
             for _ in range(5)]
    kw = {"ion_grad_type": [igt] * 5, "iongrad_index": [1.5] * 5} if model == "relxilllp" else {}
    out, st = gpu.eval_batch(model, p, [GRID] * 5, **kw)
    assert not st.any()
    for i in range(2):
        st1, ref = oracle_lib.evaluate(model, p[i], GRID, None, igt if model == "relxilllp" else 0, 1.5)
        assert st1 == 0
        assert_close(out[i], ref, f"{model} {zones} zones, gradient {igt}, set {i}")
