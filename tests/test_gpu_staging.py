"""A small host batch is read from and written to pinned memory by kernels, a large one moved by the copy engines,
and a batch split into chunks never takes the first way: the same numbers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["relline", "relconv", "relxilllp", "xillver"])
def test_small_and_large(gpu, monkeypatch, model):
    n, bins = 300, 1100  # 2.6 MB of grids
    rng = np.random.default_rng(5)
    p = np.tile(gpu.default_params(model), (n, 1))
    p[:, 0] *= rng.uniform(0.9, 1.1, n)
    grids = [np.exp(np.linspace(np.log(0.5), np.log(20.0), bins + 1 + i % 3)) for i in range(n)]
    flux = [1.0 + e[:-1] for e in grids] if model == "relconv" else None
    kw = {"ion_grad_type": [1] * n, "iongrad_index": rng.uniform(0.5, 2.0, n)} if model == "relxilllp" else {}
    large, st = gpu.eval_batch(model, p, grids, flux, **kw)
    m = 9
    cut = {k: v[:m] for k, v in kw.items()}
    small, st1 = gpu.eval_batch(model, p[:m], grids[:m], None if flux is None else flux[:m], **cut)
    monkeypatch.setenv("RELX_CHUNK_SETS", "2")
    chunks, st2 = gpu.eval_batch(model, p[:m], grids[:m], None if flux is None else flux[:m], **cut)
    assert not st.any() and not st1.any() and not st2.any()
    for i in range(m):
        assert np.array_equal(large[i], small[i]) and np.array_equal(small[i], chunks[i])


def test_flags_are_cleared(gpu):
    """A set refused in one batch leaves nothing behind for the next one of the same shape."""
    e = np.exp(np.linspace(np.log(0.5), np.log(20.0), 101))
    p = gpu.default_params("relconv")
    for _ in range(3):
        _, st = gpu.eval_batch("relconv", [p], [e], [np.zeros(100)], check=False)
        assert st[0] == 5
        out, st = gpu.eval_batch("relconv", [p], [e], [np.ones(100)])
        assert st[0] == 0 and out[0].any()
