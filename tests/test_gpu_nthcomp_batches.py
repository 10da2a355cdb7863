"""nthcomp of large batches in one launch, on either side of the sizes at which the lanes per continuum change (four up
to 14592 continua, two up to 29184, then one): the numbers of one CTA per continuum."""
import ctypes

import numpy as np
import pytest

from test_gpu_nthcomp_exchange import GRID, sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [14592, 14593, 29184, 29185])
def test_one_launch(gpu, monkeypatch, n):
    torch = pytest.importorskip("torch")
    monkeypatch.setenv("RELX_CHUNK_SETS", "0")  # never split into chunks
    p = sets()
    few = [gpu.eval_batch("xillverCp", p[a:a + 240], [GRID] * 240)[0] for a in (0, 240)]  # 240 continua: a CTA each
    ref = np.array(few[0] + few[1])
    at = np.arange(n) % len(p)
    dev = torch.device("cuda:0")
    offs = np.arange(n + 1, dtype=np.int64) * len(GRID)
    d_params = torch.from_numpy(p[at]).to(dev)
    d_e = torch.from_numpy(np.tile(GRID, n)).to(dev)
    d_off = torch.from_numpy(offs).to(dev)
    d_flux = torch.full((n, len(GRID) - 1), -1.0, dtype=torch.float64, device=dev)
    d_status = torch.full((n,), -1, dtype=torch.int32, device=dev)
    stream = torch.cuda.Stream(device=dev)
    torch.cuda.synchronize()
    # host batches of this size run as groups of about 1024 sets; device batches in one launch
    st = gpu.lib().relx_eval_batch_device(gpu.MODELS["xillverCp"], n, d_params.data_ptr(), d_e.data_ptr(),
                                          d_off.data_ptr(), offs.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)), None,
                                          d_flux.data_ptr(), d_status.data_ptr(), None, None, None, stream.cuda_stream)
    assert st == 0, gpu.last_error()
    stream.synchronize()
    assert not d_status.cpu().numpy().any()
    assert np.array_equal(d_flux.cpu().numpy(), ref[at])
