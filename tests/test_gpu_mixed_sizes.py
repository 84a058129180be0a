"""Groups of different size1 in one batch step beside each other: eager, recorded into a graph, and on a
caller's stream, against the oracle at the parity bar of the repository (1e-10 of the largest element)."""
import pytest

from builders import component_errors, make_H, make_sigma, solve_oracle
from nessi_b200 import herm_matrix
import numpy as np

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.mark.parametrize("how", ["eager", "graph", "stream"])
@pytest.mark.parametrize("shapes", [
    [(1, 30, 12, 2), (2, 24, 10, 1), (5, 12, 8, 1)],          # (size1, nt, ntau, problems) per group
    [(3, 9, 8, 2), (1, 40, 20, 3), (3, 20, 10, 1), (8, 7, 6, 1)],
])
def test_sizes_step_beside_each_other(oracle, shapes, how):
    import torch
    from nessi_b200 import gpu
    beta, h, mu, k = 4.0, 0.05, 0.1, 5
    rng = np.random.default_rng(7)
    descs, probs, sigmas = [], [], []
    for g, (s, nt, ntau, cnt) in enumerate(shapes):
        sigmas.append(make_sigma(oracle, rng, nt, ntau, s, -1, beta, h))
        for _ in range(cnt):
            H = make_H(rng, nt, s, h)
            G, G0 = solve_oracle(oracle, herm_matrix(nt, ntau, s, -1), H, sigmas[g], mu, beta, h, k)
            probs.append((H, G, G0))
            descs.append(dict(nt=nt, ntau=ntau, size1=s, sig=-1, solve_order=k, sigma_group=g, beta=beta, h=h, mu=mu))
    b = gpu.Batch(descs)
    stream = torch.cuda.Stream()
    if how == "stream":
        b.set_stream(stream.cuda_stream)
    for g, S in enumerate(sigmas):
        b.set_sigma(g, S)
    for p, (H, _, G0) in enumerate(probs):
        b.set_H(p, H)
        b.set_G(p, G0)
    n1 = max(x[1] for x in shapes)
    if how == "graph":
        b.graph_record(gpu.Batch.GRAPH_DYSON, k + 1, n1)
        b.graph_launch()
    else:
        for n in range(k + 1, n1 + 1):
            b.dyson_timestep(n)
    b.synchronize()
    for p, (H, G, _) in enumerate(probs):
        d = descs[p]
        got = herm_matrix(d["nt"], d["ntau"], d["size1"], -1)
        b.get_G(p, got)
        for comp, v in component_errors(got, G, k + 1, d["nt"]).items():
            assert v < TOL, (p, comp, v)
    b.close()
