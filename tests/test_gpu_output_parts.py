"""Few sets' output bins are spread over several CTAs: grids of fewer bins than CTAs, of one bin, of uneven
parts, in one batch, and a renormalised spectrum whose parts do not hold the bin at 3 keV."""
import numpy as np
import pytest

import oracle_lib
from tolerance import assert_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["xillver", "xillverCp", "relxill", "relxilllpCp", "relconv"])
@pytest.mark.parametrize("bins", [[1, 1, 4000], [3000], [2, 700, 511, 513, 1030]])
def test_parts(gpu, oracle, model, bins):
    grids = [np.exp(np.linspace(np.log(0.4), np.log(60.0), n + 1)) for n in bins]
    flux = [1.0 / e[:-1] for e in grids] if model == "relconv" else None
    p = np.tile(gpu.default_params(model), (len(bins), 1))
    out, st = gpu.eval_batch(model, p, grids, flux)
    assert not st.any()
    for i, e in enumerate(grids):
        st1, ref = oracle_lib.evaluate(model, p[i], e, None if flux is None else flux[i])
        assert st1 == 0
        assert_close(out[i], ref, f"{model} {bins[i]} bins")


@pytest.mark.parametrize("lo,hi", [(0.4, 60.0), (5.0, 40.0), (0.3, 2.0)])
def test_parts_renormalised(gpu, monkeypatch, lo, hi):
    monkeypatch.setenv("RELXILL_RENORMALIZE", "1")
    e = np.exp(np.linspace(np.log(lo), np.log(hi), 3001))
    p = gpu.default_params("relxill")
    whole, st = gpu.eval_batch("relxill", [p] * 320, [e] * 320)  # one CTA per set
    parts, st1 = gpu.eval_batch("relxill", [p], [e])
    assert not st.any() and not st1.any()
    assert np.array_equal(whole[0], parts[0])
