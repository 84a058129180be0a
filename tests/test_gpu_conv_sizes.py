"""convolution_timestep on device memory at the edges of its work split: first step with the long-sum kernels
(n = k), row and lane remainders, every size1, more problems than one launch takes (24); against the oracle
at the parity bar of the repository (1e-10 of the largest element)."""
import numpy as np
import pytest

from builders import rel_err
from nessi_b200 import herm_matrix
from test_gpu_conv import DevHM, make_sigma

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.mark.parametrize("s,k,ntau,cnt", [(1, 5, 31, 1), (1, 3, 12, 25), (2, 5, 17, 2), (3, 5, 11, 1), (4, 5, 12, 1),
                                          (5, 4, 9, 1), (6, 5, 8, 1), (7, 2, 7, 1), (8, 5, 10, 1)])
def test_convolution_sizes(oracle, s, k, ntau, cnt):
    import torch
    from nessi_b200 import gpu
    beta, h, nt = 3.0, 0.05, 70 if s == 1 else (41 if s == 2 else 14)
    rng = np.random.default_rng(s + 10 * cnt)
    A = [make_sigma(oracle, rng, nt, ntau, s, -1, beta, h, 0.8) for _ in range(cnt)]
    B = [make_sigma(oracle, rng, nt, ntau, s, -1, beta, h, 0.7) for _ in range(cnt)]
    dA, dB = [DevHM(x) for x in A], [DevHM(x) for x in B]
    dC = [DevHM(herm_matrix(nt, ntau, s, -1)) for _ in range(cnt)]
    steps = sorted({k - 1, k, k + 1, 2 * k + 2, nt - 1, nt})
    for n in steps:
        gpu.convolution_timestep_dev(n, [x.ptrs() for x in dC], [x.ptrs() for x in dA], [x.ptrs() for x in dA],
                                     [x.ptrs() for x in dB], [x.ptrs() for x in dB], nt, ntau, s, -1, -1, k, beta, h)
    torch.cuda.synchronize()
    for i in (range(cnt) if cnt < 4 else (0, cnt - 1)):
        ref, got = herm_matrix(nt, ntau, s, -1), dC[i].host()
        for n in steps:
            oracle.convolution_timestep(n, ref, A[i], A[i], B[i], B[i], beta, h, k)
        for c in ("ret", "les", "tv"):
            assert rel_err(getattr(got, c), getattr(ref, c)) < TOL, (i, c)
