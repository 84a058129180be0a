"""Blocked Volterra recursion (kernels_recursion.cuh): blocks of 128 scalar rows, so 128 // size1 time
rows, after the k + 1 start rows.  Lengths around the block edges (one row short, full, one row more,
a remainder in the last block), every size1, column counts that leave CTAs partly filled, orders k = 1
and 3, Dyson and VIE2, against the oracle at the parity bar of the repository: 1e-10 of the largest
element, which leaves four digits above the rounding of the longest sum here (~1e3 terms of 1e-16)."""
import numpy as np
import pytest

from builders import component_errors, make_H, make_sigma
from nessi_b200 import herm_matrix

pytestmark = pytest.mark.gpu
TOL = 1e-10
BETA, H_, NTAU = 4.0, 0.04, 8


def _history(rng, nt, s):
    """A smooth G: only its tv history and mat enter a late step."""
    G = herm_matrix(nt, NTAU, s, -1)
    t = np.arange(nt + 1)[:, None] * H_
    u = np.arange(NTAU + 1)[None, :] * BETA / NTAU
    for a in range(s):
        for b in range(s):
            w = rng.uniform(-1, 1, 4)
            G.tv[:, :, a, b] = 1j * np.exp(-1j * w[0] * t) * np.exp(-(0.5 + w[1] ** 2) * u) * (0.6 if a == b else 0.2)
            G.mat[:, a, b] = -np.exp(-(0.5 + w[2] ** 2) * u[0]) * (0.6 if a == b else 0.2)
    return G


def _edges(s, k):
    nbt = 128 // s
    return [k + nbt - 1, k + nbt, k + nbt + 1, k + 2 * nbt + 3]


@pytest.mark.parametrize("s,k,edge,cnt", [(s, 5, e, c) for s, c in ((1, 11), (2, 5), (3, 3), (4, 3), (5, 2), (6, 2),
                                                                    (7, 2), (8, 2)) for e in range(4)] +
                         [(1, 1, 2, 1), (2, 3, 3, 2), (1, 5, 1, 170), (2, 5, 2, 90)])
def test_dyson_block_edges(oracle, s, k, edge, cnt):
    from nessi_b200 import gpu
    n = _edges(s, k)[edge]
    rng = np.random.default_rng(1000 * s + 10 * k + edge)
    Sig = make_sigma(oracle, rng, n, NTAU, s, -1, BETA, H_)
    Hs = [make_H(rng, n, s, H_) for _ in range(cnt)]
    G = [_history(rng, n, s) for _ in range(cnt)]
    b = gpu.Batch([dict(nt=n, ntau=NTAU, size1=s, sig=-1, solve_order=k, beta=BETA, h=H_, mu=0.1)] * cnt)
    b.set_sigma(0, Sig)
    for p in range(cnt):
        b.set_H(p, Hs[p])
        b.set_G(p, G[p])
    b.dyson_timestep(n)
    b.synchronize()
    for p in range(cnt) if cnt < 20 else (0, 7, cnt // 2, cnt - 1):
        ref = G[p].copy()
        oracle.dyson_timestep(n, ref, 0.1, Hs[p], Sig, BETA, H_, k)
        got = herm_matrix(n, NTAU, s, -1)
        b.get_G(p, got)
        for comp, v in component_errors(got, ref, n, n).items():
            assert v < TOL, (p, comp, v)
    b.close()


@pytest.mark.parametrize("s,edge", [(1, 2), (2, 3), (3, 0), (4, 3), (8, 2)])
def test_vie2_block_edges(oracle, s, edge):
    from nessi_b200 import gpu
    k, cnt = 5, 3
    n = _edges(s, k)[edge]
    rng = np.random.default_rng(50 * s + edge)
    F = make_sigma(oracle, rng, n, NTAU, s, -1, BETA, H_)  # hermitian: Fcc = F
    Q = [make_sigma(oracle, rng, n, NTAU, s, -1, BETA, H_) for _ in range(cnt)]
    G = [_history(rng, n, s) for _ in range(cnt)]
    b = gpu.Batch([dict(nt=n, ntau=NTAU, size1=s, sig=-1, solve_order=k, beta=BETA, h=H_)] * cnt)
    b.set_F(0, F, F)
    for p in range(cnt):
        b.set_Q(p, Q[p])
        b.set_G(p, G[p])
    b.vie2_timestep(n)
    for p in range(cnt):
        ref = G[p].copy()
        oracle.vie2_timestep(n, ref, F, F, Q[p], BETA, H_, k)
        got = herm_matrix(n, NTAU, s, -1)
        b.get_G(p, got)
        for comp, v in component_errors(got, ref, n, n).items():
            assert v < TOL, (p, comp, v)
    b.close()
