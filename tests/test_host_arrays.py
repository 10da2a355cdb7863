"""Arrays handed to the library by address (csrc/pyhost.c) and arrays that need a conversion first: the same
spectra."""
import numpy as np
import pytest

GRIDS = [np.exp(np.linspace(np.log(0.5), np.log(20.0), n + 1)) for n in (1, 40, 700)]
OTHER = {"lists": lambda e: e.tolist(), "strided": lambda e: np.repeat(e, 2)[::2],
         "big-endian": lambda e: e.astype(">f8")}


def test_addresses():
    import relxill_gb300 as R

    addr, length = R._host().arrays(GRIDS)
    assert np.frombuffer(addr, np.uint64).tolist() == [e.ctypes.data for e in GRIDS]
    assert np.frombuffer(length, np.int64).tolist() == [len(e) for e in GRIDS]
    for bad in ([], GRIDS + [GRIDS[0].astype(np.float32)], [GRIDS[1][::2]], [GRIDS[1][:40].reshape(4, 10)],
                [GRIDS[0].tolist()], [GRIDS[0].astype(">f8")], [GRIDS[0].astype(np.int64)], [None]):
        assert R._host().arrays(bad) is None


@pytest.mark.gpu
@pytest.mark.parametrize("other", OTHER)
@pytest.mark.parametrize("model", ["relline", "relconv"])
def test_same_spectra(gpu, model, other):
    p = np.tile(gpu.default_params(model), (3, 1))
    flux = [np.linspace(1.0, 2.0, len(e) - 1) for e in GRIDS] if model == "relconv" else None
    a, sa = gpu.eval_batch(model, p, GRIDS, flux)
    b, sb = gpu.eval_batch(model, p, [OTHER[other](e) for e in GRIDS], None if flux is None else [OTHER[other](f) for f in flux])
    assert not sa.any() and not sb.any()
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.gpu
def test_submit(gpu):
    p = gpu.default_params("relline")
    with gpu.Server(hbm_budget_bytes=1 << 30, max_batch=16) as srv:
        out = [np.zeros(len(GRIDS[2]) - 1) for _ in range(2)]
        ids = [srv.submit("relline", p, GRIDS[2], out[0]), srv.submit("relline", p.tolist(), GRIDS[2], out[1], None, 0, 0)]
        done = {}
        while len(done) < 2:
            done.update({i: s for i, s, _ in srv.poll()})
        assert sorted(done) == sorted(ids) and not any(done.values())
        with pytest.raises(ValueError):
            srv.submit("relline", p, GRIDS[2], out[0][:-1])
        with pytest.raises(ValueError):
            srv.submit("relline", p, GRIDS[2].astype(np.float32), out[0])
    assert np.array_equal(out[0], out[1])
