"""Without the extension that reads arrays' addresses (another interpreter than the one it was built for, no Python
headers at build time) the package serves the same calls by way of numpy and ctypes."""
import numpy as np
import pytest

import relxill_gb300 as R
from relxill_gb300 import build

E = np.exp(np.linspace(np.log(0.5), np.log(20.0), 9))
N = len(E) - 1


@pytest.fixture
def missing(monkeypatch, tmp_path):
    monkeypatch.setattr(R, "HOST_EXT_PATH", str(tmp_path / "missing.so"))
    monkeypatch.setattr(R, "_host_ext", None)


class Recorder:
    def __init__(self):
        self.calls = []

    def relx_eval_batch(self, model, n, *a):
        self.calls.append(("eval", n))
        return 0

    def relx_serve_create(self, *a):
        return 1

    def relx_serve_submit(self, *a):
        self.calls.append(("submit", a[4]))
        return len(self.calls)

    def relx_serve_destroy(self, h):
        pass


def test_calls(missing, monkeypatch):
    rec = Recorder()
    monkeypatch.setattr(R, "lib", lambda: rec)
    out, status = R.eval_batch("relline", np.tile(R.default_params("relline"), (2, 1)), [E, E])
    assert [len(o) for o in out] == [N, N] and not status.any()
    R.eval_batch("relconv", R.default_params("relconv"), [E], [np.ones(N)])
    with R.Server() as srv:
        assert srv.submit("relline", R.default_params("relline"), E, np.zeros(N)) == 3
    assert rec.calls == [("eval", 2), ("eval", 1), ("submit", N)]


def test_unloadable(monkeypatch, tmp_path):
    other = tmp_path / "other.so"
    other.write_bytes(b"not for this interpreter")
    monkeypatch.setattr(R, "HOST_EXT_PATH", str(other))
    monkeypatch.setattr(R, "_host_ext", None)
    assert R._host() is None


def test_build_without_headers(monkeypatch, tmp_path):
    monkeypatch.setattr(build.sysconfig, "get_paths", lambda: {"include": str(tmp_path)})
    monkeypatch.setattr(build, "HOST_EXT", str(tmp_path / "ext.so"))
    assert "Python.h" in build._compile_host_ext()


@pytest.mark.gpu
def test_same_numbers(gpu, missing):
    p = gpu.default_params("relline")
    plain, st = gpu.eval_batch("relline", p, [E])
    out = np.zeros(N)
    with gpu.Server(hbm_budget_bytes=1 << 30, max_batch=4) as srv:
        srv.submit("relline", p, E, out)
        done = []
        while not done:
            done = srv.poll()
    assert not st.any() and done[0][1] == 0
    assert gpu._host() is None and np.array_equal(out, plain[0]) and np.array_equal(gpu.relline(E, p), out)
