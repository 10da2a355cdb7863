"""The two line-profile kernels: a zone summed by one warp (many sets) and by the warps of a CTA (few
sets) give the same numbers, at grid sizes around the edges of their tiles (32 and 128 bins) and set
counts around the rule that chooses between them, and agree with the oracle."""
import numpy as np
import pytest

import oracle_lib
from tolerance import assert_close

pytestmark = pytest.mark.gpu

BINS = (1, 2, 31, 32, 33, 63, 127, 128, 129, 255, 400)


def _sets(model, n, limb, seed):
    rng = np.random.default_rng(seed)
    a, incl = rng.uniform(-0.5, 0.998, n), rng.uniform(5, 85, n)
    if model == "relline":
        p = [[rng.uniform(1.0, 7.0), rng.uniform(2, 5), rng.uniform(2, 4), 15.0, a[i], incl[i], -1.0,
              rng.uniform(20, 990), 0.0, limb] for i in range(n)]
    else:
        p = [[rng.uniform(3, 60), 0.0, a[i], incl[i], -1.0, rng.uniform(50, 990), 0.0, rng.uniform(1.5, 2.7),
              rng.uniform(0, 4.5), 1.0, 300.0, 1.0, 0.0, 0.0] for i in range(n)]
    grids = [np.exp(np.linspace(np.log(0.3), np.log(9.0), BINS[i % len(BINS)] + 1)) for i in range(n)]
    return p, grids


# the rule's lines: 256 sets of 10 zones, 1536 sets of one; a limb law stays with the team kernel
@pytest.mark.parametrize("model,n,limb,igt", [("relxilllp", 255, 0, 0), ("relxilllp", 256, 0, 0), ("relxilllp", 103, 0, 2),
                                              ("relline", 1535, 0, 0), ("relline", 1536, 0, 0), ("relline", 1536, 1, 0),
                                              ("relline", 65, 2, 0), ("relline", 129, 0, 0), ("relline", 17, 0, 0)])
def test_line_kernels(gpu, oracle, model, n, limb, igt):
    p, grids = _sets(model, n, limb, 3 * n + limb)
    many, st = gpu.eval_batch(model, p, grids, ion_grad_type=[igt] * n)
    assert not st.any()
    pick = range(0, n, max(1, n // 13))
    for i in pick:
        one, st1 = gpu.eval_batch(model, [p[i]], [grids[i]], ion_grad_type=[igt])
        assert not st1.any()
        np.testing.assert_array_equal(many[i], one[0], err_msg=f"set {i}")
    for i in list(pick)[:5]:
        st1, ref = oracle_lib.evaluate(model, p[i], grids[i], None, igt, 0.0)
        assert st1 == 0
        if np.isfinite(ref).all():
            assert_close(many[i], ref, f"{model} set {i}")
