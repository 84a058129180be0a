"""Groups of one size1 step in one launch set: groups that differ in length, tau grid, order, statistics
and number of problems, and more groups than one launch takes (64), against the oracle at the parity bar
of the repository (1e-10 of the largest element)."""
import numpy as np
import pytest

from builders import component_errors, make_H, make_sigma, solve_oracle
from nessi_b200 import herm_matrix

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.mark.parametrize("s,shapes", [
    (1, [(30, 12, 5, -1, 3), (9, 20, 5, -1, 1), (22, 8, 3, -1, 2), (26, 10, 2, 1, 1)]),
    (2, [(20, 10, 5, -1, 2), (70, 8, 5, -1, 1)]),
    (3, [(12, 8, 4, -1, 1), (16, 10, 5, -1, 2)]),
    (1, [(8 + i % 3, 8, 5, -1, 1) for i in range(66)]),
])
def test_groups_step_together(oracle, s, shapes):
    from nessi_b200 import gpu
    beta, h = 4.0, 0.05
    rng = np.random.default_rng(len(shapes) + 10 * s)
    descs, probs, sigmas = [], [], []
    for g, (nt, ntau, k, sig, cnt) in enumerate(shapes):
        mu = -1.5 if sig == 1 else 0.1
        Sig = make_sigma(oracle, rng, nt, ntau, s, sig, beta, h)
        sigmas.append(Sig)
        for _ in range(cnt):
            H = make_H(rng, nt, s, h)
            G = herm_matrix(nt, ntau, s, sig)
            Gf, Gb = solve_oracle(oracle, G, H, Sig, mu, beta, h, k)
            probs.append((H, Gf, Gb, k, nt))
            descs.append(dict(nt=nt, ntau=ntau, size1=s, sig=sig, solve_order=k, sigma_group=g, beta=beta, h=h, mu=mu))
    b = gpu.Batch(descs)
    for g, Sig in enumerate(sigmas):
        b.set_sigma(g, Sig)
    kmax = max(x[2] for x in shapes)
    for p, (H, Gf, Gb, _, _) in enumerate(probs):
        b.set_H(p, H)
        G = Gf.copy() if probs[p][3] < kmax else Gb  # groups of lower order: the oracle's steps up to kmax
        for t in range(kmax + 1, probs[p][4] + 1):
            G.set_timestep_data(t, 0 * G.get_timestep(t))
        b.set_G(p, G)
    for n in range(kmax + 1, max(x[0] for x in shapes) + 1):
        b.dyson_timestep(n)
    b.synchronize()
    for p, (H, Gf, Gb, k, nt) in enumerate(probs):
        got = herm_matrix(nt, descs[p]["ntau"], s, descs[p]["sig"])
        b.get_G(p, got)
        for comp, v in component_errors(got, Gf, kmax + 1, nt).items():
            assert v < TOL, (p, comp, v)
    b.close()
