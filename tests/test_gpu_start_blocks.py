"""Start rows of a time step (the dense k-block systems of the retarded row and the lesser column) solved by
one warp (at most size1 4) and by the CTA, over the orders and sizes on both sides, against the oracle at
the parity bar of the repository (1e-10 of the largest element)."""
import numpy as np
import pytest

from builders import component_errors, make_H, make_sigma, solve_oracle
from nessi_b200 import herm_matrix

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 3, 5])
@pytest.mark.parametrize("s", [1, 2, 4, 5, 7])
def test_start_rows(oracle, s, k):
    from nessi_b200 import gpu
    beta, h, mu, nt, ntau = 4.0, 0.05, 0.1, 2 * k + 3, 8
    rng = np.random.default_rng(100 * s + k)
    Sig = make_sigma(oracle, rng, nt, ntau, s, -1, beta, h)
    H = make_H(rng, nt, s, h)
    G, G0 = solve_oracle(oracle, herm_matrix(nt, ntau, s, -1), H, Sig, mu, beta, h, k)
    b = gpu.Batch([dict(nt=nt, ntau=ntau, size1=s, sig=-1, solve_order=k, beta=beta, h=h, mu=mu)])
    b.set_sigma(0, Sig)
    b.set_H(0, H)
    b.set_G(0, G0)
    for n in range(k + 1, nt + 1):
        b.dyson_timestep(n)
    b.synchronize()
    got = herm_matrix(nt, ntau, s, -1)
    b.get_G(0, got)
    b.close()
    for comp, v in component_errors(got, G, k + 1, nt).items():
        assert v < 1e-10, (comp, v)
