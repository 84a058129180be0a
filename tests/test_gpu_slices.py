"""Time-step slices between the host and a batch (set / get_timestep, set_sigma_timestep): pageable,
pinned and partly offset pinned buffers, every tile remainder of the tau grid, more slices in a row than
the batch has staging slots, both precisions.  The data are copied, so they come back bit for bit."""
import numpy as np
import pytest

from nessi_b200 import herm_matrix

pytestmark = pytest.mark.gpu


def _buffer(kind, n, s):
    if kind == "pageable":
        return np.zeros((n, s, s), np.complex128)
    import torch
    off = 3 if kind == "pinned_offset" else 0
    t = torch.zeros((n + off) * s * s, dtype=torch.complex128).pin_memory()
    return t.numpy()[off * s * s:].reshape(n, s, s)


@pytest.mark.parametrize("s,ntau", [(1, 31), (1, 32), (2, 8), (2, 33), (3, 64), (5, 40), (8, 70)])
@pytest.mark.parametrize("kind", ["pageable", "pinned", "pinned_offset"])
@pytest.mark.parametrize("mixed", [False, True])
def test_slices_come_back(s, ntau, kind, mixed):
    from nessi_b200 import gpu
    nt = 40
    rng = np.random.default_rng(s * 100 + ntau)
    b = gpu.Batch([dict(nt=nt, ntau=ntau, size1=s, sig=-1, solve_order=5, beta=2.0, h=0.1)] * 2,
                  gpu.PREC_MIXED if mixed else gpu.PREC_FP64)
    ref, sig = {}, {}
    buf = None
    for t in list(range(0, 9)) + [nt]:
        n = 2 * (t + 1) + ntau + 1
        for p in (0, 1):
            ref[p, t] = rng.normal(size=(n, s, s)) + 1j * rng.normal(size=(n, s, s))
            buf = _buffer(kind, n, s)
            buf[...] = ref[p, t]
            b.set_timestep(p, t, buf)
            buf[...] = 0  # the call owns the data once it returns
        sig[t] = rng.normal(size=(n, s, s)) + 1j * rng.normal(size=(n, s, s))
        buf = _buffer(kind, n, s)
        buf[...] = sig[t]
        b.set_sigma_timestep(0, t, buf)
        buf[...] = 0
    S = herm_matrix(nt, ntau, s, -1)
    b.get_sigma(0, S)
    for (p, t), v in ref.items():
        out = _buffer(kind, len(v), s)
        b.get_timestep(p, t, out)
        assert np.array_equal(out, v), (p, t)
    for t, v in sig.items():
        assert np.array_equal(S.ret_row(t), v[:t + 1]) and np.array_equal(S.les_col(t), v[t + 2 + ntau:])
        assert np.array_equal(S.tv[t], v[t + 1:t + 2 + ntau])
    b.close()


def test_a_slice_is_refused_during_capture():
    import ctypes
    import torch
    from nessi_b200 import gpu
    nt, ntau = 10, 8
    b = gpu.Batch([dict(nt=nt, ntau=ntau, size1=1, sig=-1, solve_order=5, beta=2.0, h=0.1)])
    stream = torch.cuda.Stream()
    handle, graph = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p()
    b.set_stream(stream.cuda_stream)
    data = np.arange(2 * 7 + ntau + 1, dtype=np.complex128).reshape(-1, 1, 1)
    out = np.zeros_like(data)
    b.set_timestep(0, 6, data)  # the staging slots exist
    cudart = ctypes.CDLL("libcudart.so.12")
    assert cudart.cudaStreamBeginCapture(handle, 1) == 0  # thread-local mode
    with pytest.raises(gpu.NessiGpuError):
        b.set_timestep(0, 6, 2 * data)
    cudart.cudaStreamEndCapture(handle, ctypes.byref(graph))  # an error if the refused call ended the capture
    b.get_timestep(0, 6, out)
    assert np.array_equal(out, data)
    b.set_timestep(0, 6, 3 * data)
    b.get_timestep(0, 6, out)
    assert np.array_equal(out, 3 * data)
    b.close()
