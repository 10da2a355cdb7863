"""Line profiles of one-zone sets on either side of the number of sets at which the kernel changes: the same numbers, and
about the same time per set, for relline tables with few and with the usual 40 g* points."""
import ctypes
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FEW, MANY = 1535, 1536


@pytest.fixture
def tables(request, gpu, small_tables, tmp_path):
    from relxill_gb300 import synth_tables

    for f in os.listdir(small_tables):
        if not f.startswith("rel_table"):
            os.symlink(os.path.join(small_tables, f), tmp_path / f)
    name = next(f for f in os.listdir(small_tables) if f.startswith("rel_table"))
    synth_tables.write_relline_table(str(tmp_path / name), n_g=request.param)
    gpu.init(str(tmp_path))
    yield gpu
    gpu.init(small_tables)


def profile_ms(R, p, grids):
    L = R.lib()
    L.relx_profile_name.restype = ctypes.c_char_p
    k = next(i for i in range(9) if L.relx_profile_name(i) == b"relline")
    times = []
    for _ in range(5):
        L.relx_profile_enable(1)
        out, st = R.eval_batch("relline", p, grids)
        ms = (ctypes.c_double * 9)()
        assert L.relx_profile_read(ms, None, 9) == 0 and not st.any()
        L.relx_profile_enable(0)
        times.append(ms[k])
    return sorted(times)[2], out


@pytest.mark.parametrize("tables", [12, 20, 23, 24, 40], indirect=True)
def test_either_side(tables):
    R = tables
    rng = np.random.default_rng(7)
    p = np.tile(R.default_params("relline"), (MANY, 1))
    p[:, 4], p[:, 5] = rng.uniform(0.0, 0.998, MANY), rng.uniform(5.0, 85.0, MANY)
    grids = [np.exp(np.linspace(np.log(0.3), np.log(80.0), int(n) + 1)) for n in rng.integers(300, 1500, MANY)]
    few, a = profile_ms(R, p[:FEW], grids[:FEW])
    many, b = profile_ms(R, p, grids)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)
    assert many < 1.4 * few
