"""Arrays that reach the library by address are long enough and of its type, whichever way they are handed over: the
host layer on a library that records its calls."""
import numpy as np
import pytest

import relxill_gb300 as R

E = np.exp(np.linspace(np.log(0.5), np.log(20.0), 9))
N = len(E) - 1
P = R.default_params("relconv")


class Recorder:
    """Stands in for the library: keeps what the input spectrum's address held."""

    def __init__(self):
        self.spectra = []

    def relx_serve_submit(self, h, model, params, energy, n, flux_in, out, igt, igi):
        self.spectra.append([flux_in[i] for i in range(n)] if flux_in else None)
        return len(self.spectra)

    def relx_eval_batch(self, *a):
        self.spectra.append(a)
        return 0

    relx_eval_batch_sets = relx_eval_batch

    def relx_last_status(self):
        return 0

    def c_lmodrelconv(self, *a):
        self.spectra.append(a)


@pytest.fixture
def rec(monkeypatch):
    r = Recorder()
    monkeypatch.setattr(R, "lib", lambda: r)
    return r


@pytest.fixture
def server(rec, monkeypatch):
    s = object.__new__(R.Server)
    s._h, s._keep, s._submit, s._submit_fn = None, {}, (lambda *a: None), 0
    return s


@pytest.mark.parametrize("form", [lambda f: f.astype(np.float32), lambda f: np.repeat(f, 2)[::2],
                                  lambda f: f.astype(">f8"), lambda f: f])
def test_submit_converts(server, rec, form):
    f = np.arange(1.0, N + 1)
    rid = server.submit("relconv", P, E, np.zeros(N), form(f))
    assert rec.spectra == [f.tolist()]
    kept = [a for a in server._keep[rid] if isinstance(a, np.ndarray) and a.dtype == np.float64 and
            a.dtype.isnative and a.shape == f.shape and np.array_equal(a, f)]
    assert kept  # what was handed over stays alive


def test_submit_refuses(server, rec):
    f = np.ones(N)
    for bad in (dict(flux_in=f[:-1]), dict(flux_in=f[:-1].astype(np.float32)), dict(params=P[:-1], flux_in=f)):
        a = dict(dict(params=P), **bad)
        with pytest.raises(ValueError):
            server.submit("relconv", a["params"], E, np.zeros(N), a["flux_in"])
    assert not rec.spectra


def test_eval_batch_refuses(rec):
    p = np.tile(P, (2, 1))
    with pytest.raises(ValueError):
        R.eval_batch("relconv", p, [E, E], [np.ones(N), np.ones(N - 1)])
    assert not rec.spectra
    R.eval_batch("relconv", p, [E, E], [np.ones(N + 1), np.ones(N - 1)])  # joined as they come
    assert len(rec.spectra) == 1


def test_local_model_refuses(rec):
    for short in (np.ones(N - 1), np.ones(0)):
        with pytest.raises(ValueError):
            R.relconv(E, P, short)
    assert not rec.spectra
    assert R.relconv(E, P, np.ones(N + 2)).shape == (N + 2,)  # values beyond the bins are left alone


@pytest.mark.parametrize("short", [dict(ion_grad_type=[1]), dict(ion_grad_type=[1, 1], iongrad_index=[0.5])])
def test_gradients_refused(rec, short):
    with pytest.raises(ValueError):
        R.eval_batch("relxilllp", np.tile(R.default_params("relxilllp"), (2, 1)), [E, E], **short)
    assert not rec.spectra


@pytest.mark.gpu
def test_served_spectra(gpu):
    f = np.arange(1.0, N + 1)
    out = [np.zeros(N) for _ in range(3)]
    with gpu.Server(hbm_budget_bytes=1 << 30, max_batch=16) as srv:
        for o, g in zip(out, (f, f.astype(np.float32), np.repeat(f, 2)[::2])):
            srv.submit("relconv", P, E, o, g)
        done = 0
        while done < 3:
            for _, status, _ in srv.poll():
                assert status == 0
                done += 1
    assert out[0].any() and np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
