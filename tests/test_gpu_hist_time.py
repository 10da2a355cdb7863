"""Emission-angle histograms of relline tables with fewer g* points than the usual 40 take no longer than a multiple of
what the 40 points take (the work is per point; every radius by the rare path takes five times as long)."""
import ctypes
import os

import numpy as np
import pytest

from test_gpu_hist_points import test_points as check_points

pytestmark = pytest.mark.gpu

N = 512


def hist_ms(R, path):
    R.init(str(path))
    L = R.lib()
    L.relx_profile_name.restype = ctypes.c_char_p
    names = [L.relx_profile_name(k).decode() for k in range(9)]
    k = next(i for i, s in enumerate(names) if "hist" in s)
    p = np.tile(R.default_params("relxilllp"), (N, 1))
    p[:, 2], p[:, 3] = np.linspace(0.0, 0.99, N), np.linspace(5.0, 85.0, N)
    grid = np.exp(np.linspace(np.log(0.5), np.log(50.0), 65))
    times = []
    for _ in range(5):
        L.relx_profile_enable(1)
        R.eval_batch("relxilllp", p, [grid] * N)
        ms = (ctypes.c_double * 9)()
        assert L.relx_profile_read(ms, None, 9) == 0
        L.relx_profile_enable(0)
        times.append(ms[k])
    return sorted(times)[2]


@pytest.mark.parametrize("points", [20, 33, 39])
def test_fewer_points(gpu, small_tables, tmp_path, points):
    from relxill_gb300 import synth_tables

    for f in os.listdir(small_tables):
        if not f.startswith("rel_table"):
            os.symlink(os.path.join(small_tables, f), tmp_path / f)
    name = next(f for f in os.listdir(small_tables) if f.startswith("rel_table"))
    synth_tables.write_relline_table(str(tmp_path / name), n_a=5, n_mu0=6, n_g=points)
    try:
        few, full = hist_ms(gpu, tmp_path), hist_ms(gpu, small_tables)
    finally:
        gpu.init(small_tables)
    print(points, few, full)
    assert few < 1.5 * full


@pytest.mark.parametrize("points", [12, 24, 25, 39, 41])  # either side of the kernels' 24 and 40 points
def test_numbers(small_tables, tmp_path, points):
    check_points(small_tables, tmp_path, points)
