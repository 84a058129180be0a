"""Column counts and block edges of the blocked Volterra recursion (kernels_recursion.cuh) that a few problems
do not reach, against the oracle at the parity bar of the repository (1e-10 of the largest element: four digits above
the rounding of the longest sum here).

Columns: a CTA of the diagonal kernel takes wc = 1, 2, 4 or 8 columns, doubling while there are more than
wc x 148 of them (size1 3 and 4: at most 2, larger: at most 4; less for the retarded one beside a long tau grid).
The counts here reach every wc, two columns per warp (size1 2, wc 8), CTAs whose columns belong to several
problems, and a last CTA with columns missing; the long tau grid has a case of its own."""
import numpy as np
import pytest

from builders import component_errors, make_H, make_sigma
from nessi_b200 import herm_matrix
from test_gpu_recursion import _history

pytestmark = pytest.mark.gpu
TOL, TOL_MIXED = 1e-10, 1e-8  # the repository's bars
BETA, H_, NTAU = 4.0, 0.04, 8


def _rows(s):
    return 4 * (32 // s)  # time rows of a block


def _run(oracle, s, k, n, cnt, check, vie2=False, mixed=False):
    """One late step n of cnt problems; the problems in `check` have data of their own, the others share
    one set."""
    from nessi_b200 import gpu
    rng = np.random.default_rng(100000 * s + 100 * n + cnt)
    Sig = make_sigma(oracle, rng, n, NTAU, s, -1, BETA, H_)
    own = {p: (make_sigma(oracle, rng, n, NTAU, s, -1, BETA, H_) if vie2 else make_H(rng, n, s, H_), _history(rng, n, s))
           for p in list(check) + [-1]}
    b = gpu.Batch([dict(nt=n, ntau=NTAU, size1=s, sig=-1, solve_order=k, beta=BETA, h=H_, mu=0.1)] * cnt,
                  gpu.PREC_MIXED if mixed else gpu.PREC_FP64)
    if vie2:
        b.set_F(0, Sig, Sig)  # hermitian: Fcc = F
    else:
        b.set_sigma(0, Sig)
    for p in range(cnt):
        X, G = own.get(p, own[-1])
        if vie2:
            b.set_Q(p, X)
        else:
            b.set_H(p, X)
        b.set_G(p, G)
    if vie2:
        b.vie2_timestep(n)
    else:
        b.dyson_timestep(n)
    b.synchronize()
    for p in check:
        X, G = own[p]
        ref = G.copy()
        if vie2:
            oracle.vie2_timestep(n, ref, Sig, Sig, X, BETA, H_, k)
        else:
            oracle.dyson_timestep(n, ref, 0.1, X, Sig, BETA, H_, k)
        got = herm_matrix(n, NTAU, s, -1)
        b.get_G(p, got)
        for comp, v in component_errors(got, ref, n, n).items():
            assert v < (TOL_MIXED if mixed else TOL), (p, comp, v)
    b.close()


def _some(s, cnt):
    """The first problems (of the first CTAs, whole and straddling), one in the middle and the last ones."""
    return sorted({0, 1, 2, 3, 7, 8, cnt // 2, cnt - 2, cnt - 1} & set(range(cnt)))


MANY = [(1, 301), (1, 600), (1, 603),            # wc 4, 8, 8 with three columns in the last CTA
        (2, 150), (2, 297), (2, 299),            # wc 4, 8 with two columns in the last CTA, 8 with six
        (3, 52), (3, 101),                       # wc 2, problems across CTAs, one column in the last
        (4, 40), (4, 75),                        # wc 2
        (5, 31), (5, 61), (6, 51), (7, 45), (8, 20), (8, 38)]  # wc 2, 4, 4, 4, 2, 4


@pytest.mark.parametrize("s,cnt", MANY)
def test_dyson_columns(oracle, s, cnt):
    _run(oracle, s, 5, 5 + 2 * _rows(s) + 3, cnt, _some(s, cnt))


@pytest.mark.parametrize("s,cnt", [(1, 603), (2, 299), (3, 101), (4, 75), (5, 61), (8, 38)])
def test_vie2_columns(oracle, s, cnt):
    _run(oracle, s, 5, 5 + _rows(s) + 2, cnt, _some(s, cnt), vie2=True)


@pytest.mark.parametrize("s,cnt,vie2", [(2, 299, False), (2, 299, True), (4, 75, False), (1, 603, False)])
def test_columns_of_a_mixed_step(oracle, s, cnt, vie2):
    _run(oracle, s, 5, 5 + _rows(s) + 2, cnt, _some(s, cnt), vie2, mixed=True)


@pytest.mark.parametrize("s,ntau,cnt", [(2, 150, 299), (4, 300, 40)])  # wc 4 for ret and 8 for les, 1 and 2
def test_columns_beside_a_long_tau_grid(oracle, monkeypatch, s, ntau, cnt):
    import test_gpu_recursion
    monkeypatch.setattr(test_gpu_recursion, "NTAU", ntau)
    monkeypatch.setitem(globals(), "NTAU", ntau)
    _run(oracle, s, 5, 5 + _rows(s) + 2, cnt, _some(s, cnt))


@pytest.mark.parametrize("vie2", [False, True])
@pytest.mark.parametrize("s", [3, 5, 6, 7])
@pytest.mark.parametrize("extra", [-1, 0, 1, 16])
def test_block_edges_of_sizes_that_leave_lanes_idle(oracle, s, extra, vie2):
    """32 is not a multiple of these size1: a block one row short, full, one row more, and two blocks with a
    remainder (4 (32 // size1) rows each)."""
    _run(oracle, s, 5, 5 + _rows(s) + extra, 2, [0, 1], vie2)


def test_tiled_product_beside_the_stream(oracle):
    """Sigma^< G^A in its tiled form (size1 1 and 2, at least 6 x 148 tiles of 32 x 32), ragged in both directions."""
    _run(oracle, 2, 5, 253, 903, [0, 1, 451, 901, 902])
