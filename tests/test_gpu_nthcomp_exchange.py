"""nthcomp by four lanes per continuum: a point of the recurrence that one lane stores is read back by another, for
grids of every length modulo the lanes; the same numbers as by one CTA per continuum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRID = np.exp(np.linspace(np.log(0.1), np.log(200.0), 9))


def sets():
    """480 xillverCp sets: 48 grids one point longer each (kTe in steps of 0.02 dex), ten Gamma."""
    kte, gamma = np.meshgrid(5.0 * 10.0 ** (0.01 + 0.02 * np.arange(48)), np.linspace(1.2, 3.4, 10))
    p = np.zeros((kte.size, 8))
    p[:, 0], p[:, 1], p[:, 2], p[:, 3], p[:, 4] = gamma.ravel(), 1.0, kte.ravel(), 3.1, 15.0
    p[:, 6], p[:, 7] = 30.0, 1.0
    return p


def test_lengths(gpu):
    p = sets()
    many, st = gpu.eval_batch("xillverCp", p, [GRID] * len(p))  # more than 456 continua: four lanes each
    assert not st.any()
    for a in (0, 240):  # a CTA each
        few, st = gpu.eval_batch("xillverCp", p[a:a + 240], [GRID] * 240)
        assert not st.any()
        for i in range(240):
            assert np.array_equal(few[i], many[a + i]), p[a + i]
