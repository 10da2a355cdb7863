"""Device buffers that a kernel of the current device cannot use where they are (here: not aligned to their elements) go
by way of the copy engines, each by itself."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 5


@pytest.mark.parametrize("shifted", ["energy", "flux_in", "flux", "status", "all", "none"])
def test_shifted_buffers(gpu, shifted):
    torch = pytest.importorskip("torch")
    grids = [np.exp(np.linspace(np.log(0.5), np.log(20.0), n + 1)) for n in (1, 40, 333, 700, 3000)]
    spectra = [np.linspace(1.0, 2.0, len(e) - 1) for e in grids]
    p = np.tile(gpu.default_params("relconv"), (N, 1))
    p[:, 3] = np.linspace(0.1, 0.9, N)
    host, st = gpu.eval_batch("relconv", p, grids, spectra)
    assert not st.any()
    edges, offs = gpu.pack_grids(grids)
    fin = np.zeros(len(edges))
    for f, o in zip(spectra, offs):
        fin[o:o + len(f)] = f
    hold = []

    def put(name, a, by):
        shift = by if shifted in (name, "all") else 0
        raw = torch.zeros(a.nbytes + 16, dtype=torch.uint8, device="cuda:0")
        at = raw[shift:shift + a.nbytes]
        at.copy_(torch.from_numpy(a.view(np.uint8)))
        hold.append(raw)
        return at

    d_p, d_off = put("params", p.reshape(-1), 0), put("offsets", offs, 0)
    d_e, d_f = put("energy", edges, 4), put("flux_in", fin, 4)
    d_out, d_st = put("flux", np.full(int(offs[-1]) - N, -1.0), 4), put("status", np.full(N, -1, np.int32), 2)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    rc = gpu.lib().relx_eval_batch_device(gpu.MODELS["relconv"], N, d_p.data_ptr(), d_e.data_ptr(), d_off.data_ptr(),
                                          offs.ctypes.data_as(ctypes.POINTER(ctypes.c_int64)), d_f.data_ptr(),
                                          d_out.data_ptr(), d_st.data_ptr(), None, None, None, stream.cuda_stream)
    assert rc == 0, gpu.last_error()
    stream.synchronize()
    assert not d_st.cpu().numpy().copy().view(np.int32).any()
    assert np.array_equal(d_out.cpu().numpy().copy().view(np.float64), np.concatenate(host))
