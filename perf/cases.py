"""Timed workloads of the Kadanoff-Baym time stepping, through the package's public entry points.

A case is one piece of work that a program on this library repeats:

* ``step``      the corrector loop of one time step of a batch: Sigma(n) is uploaded and
                ``dyson_timestep(n)`` solved ``ncorr`` times, then every problem's slice is read back
                (the loop of the reference's lattice, impurity and GW drivers).  ``groups`` lists
                "size1 x problems" per self-energy.
* ``run``       a whole propagation n = k+1..nt, G read back at the end.
* ``lattice``   predictor, k-average, Sigma_2B and Dyson correctors on the device
                (``lattice_2b_timestep``): one late step of a large lattice, or a whole recorded
                propagation of a small one.  The output is G_loc.
* ``vie2``      ``vie2_timestep(n)`` of a batch ([1 + F] G = Q).
* ``conv``      ``convolution_timestep`` of independent problems on device memory.

Inputs are smooth two-time functions of a discrete bath and of free levels, of the size and decay
that the drivers meet; late steps start from a given history, as after a restart.  ``exact``
evaluates the same discretised equations in plain torch with complex128.
"""
from fractions import Fraction
from math import comb
from types import SimpleNamespace

import numpy as np
import torch

from nessi_b200 import gpu

C128 = torch.complex128
F64 = torch.float64


# ---- the cases ------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: one level in a bath (the CPU-sized impurity quench), a single step
        dict(name="impurity_step", kind="step", groups="1x1", n=200, ntau=400, k=5, beta=10.0, h=0.02, ncorr=1,
             spread=0, mixed=False),
        # the same problem propagated from its first to its last step, one call per step
        dict(name="impurity_run", kind="run", groups="1x1", n=200, ntau=400, k=5, beta=10.0, h=0.02),
        # the two-band chain, 256 k-points, its last step with three correctors
        dict(name="chain2_step", kind="step", groups="2x256", n=1000, ntau=600, k=5, beta=20.0, h=0.01, ncorr=3,
             spread=0, mixed=False),
        # mixed precision at odd sizes
        dict(name="chain2_mixed", kind="step", groups="2x150", n=777, ntau=431, k=5, beta=20.0, h=0.01, ncorr=3,
             spread=0, mixed=True),
        # a chunk of 32 k-points of the four-band chain
        dict(name="chain4_step", kind="step", groups="4x32", n=1200, ntau=800, k=5, beta=20.0, h=0.01, ncorr=2,
             spread=0, mixed=False),
        # independent problems of uneven orbital size and length in one batch
        dict(name="uneven_step", kind="step", groups="1x21,2x19,3x20,5x18,8x18", n=600, ntau=400, k=5, beta=10.0,
             h=0.01, ncorr=1, spread=150, mixed=False),
        # momentum-dependent self-energies (GW): every k-point has its own Sigma
        dict(name="kgroups_step", kind="step", groups=",".join(["1x1"] * 32), n=400, ntau=200, k=5, beta=10.0,
             h=0.02, ncorr=2, spread=0, mixed=False),
        # the 32 x 32 square lattice with local Sigma_2B, one late step with three correctors
        dict(name="lattice_step", kind="lattice", nk=1024, n0=1000, n=1000, ntau=800, k=5, beta=20.0, h=0.01,
             ncorr=3, umat=0.0, graph=False),
        # a small lattice, its whole propagation recorded once and replayed
        dict(name="lattice_run", kind="lattice", nk=64, n0=6, n=90, ntau=200, k=5, beta=10.0, h=0.02, ncorr=3,
             umat=1.0, graph=True),
        # screened interaction / integral form: one VIE2 step of 32 problems
        dict(name="vie2_step", kind="vie2", groups="2x32", n=500, ntau=300, k=5, beta=10.0, h=0.02),
        # standalone contour convolutions on device memory (downfolding, T matrices)
        dict(name="convolution", kind="conv", count=16, s=2, n=600, ntau=400, k=5, beta=10.0, h=0.02),
    ]


def _logint(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    while True:
        kind = rng.choice(["step", "step", "step", "step", "kgroups", "run", "lattice", "lattice_run", "vie2", "conv"])
        k = rng.choice([5, 5, 5, 4, 3, 2])
        ntau = _logint(rng, 40, 800)
        beta, h = rng.choice([5.0, 10.0, 20.0]), rng.choice([0.01, 0.02, 0.04])
        case = dict(kind=kind, k=k, ntau=ntau, beta=beta, h=h)
        if kind == "step":
            s = rng.choice([1, 1, 2, 2, 3, 4, 5, 6, 8])
            case.update(groups="%dx%d" % (s, _logint(rng, 1, 512)), n=_logint(rng, 24, 1200), ncorr=rng.choice([1, 2, 3]),
                        spread=rng.choice([0, 0, 40]), mixed=rng.random() < 0.25)
        elif kind == "kgroups":
            s = rng.choice([1, 1, 2, 3])
            case.update(kind="step", groups=",".join("%dx%d" % (s, rng.choice([1, 1, 2])) for _ in range(_logint(rng, 2, 48))),
                        n=_logint(rng, 40, 500), ncorr=rng.choice([1, 2]), spread=0, mixed=False)
        elif kind == "run":
            case.update(groups="%dx%d" % (rng.choice([1, 2, 3]), _logint(rng, 1, 8)), n=_logint(rng, 40, 200))
        elif kind == "lattice":
            n = _logint(rng, 40, 1000)
            case.update(nk=_logint(rng, 16, 1024), n0=n, n=n, ncorr=rng.choice([1, 2, 3]), umat=0.0, graph=False)
        elif kind == "lattice_run":
            case.update(kind="lattice", nk=_logint(rng, 16, 256), n0=k + 1, n=_logint(rng, 30, 100),
                        ncorr=rng.choice([2, 3]), umat=1.0, graph=rng.random() < 0.5)
        elif kind == "vie2":
            case.update(groups="%dx%d" % (rng.choice([1, 2, 3, 4]), _logint(rng, 1, 64)), n=_logint(rng, 30, 700))
        else:
            case.update(count=_logint(rng, 1, 40), s=rng.choice([1, 2, 3, 4]), n=_logint(rng, 30, 700))
        w = work(case)
        if w["bytes"] < 3.0e10 and w["flops"] < 1.0e11 and _state_bytes(case) < 3.0e10:
            return case


def _groups(case):
    return [tuple(int(x) for x in g.split("x")) for g in case["groups"].split(",")]


def _state_bytes(case):
    n, M = case["n"], case["ntau"] + 1
    if case["kind"] == "conv":
        return 16.0 * case["count"] * case["s"] ** 2 * 3 * ((n + 1) ** 2 + n * M)
    grp = [(1, case["nk"])] if case["kind"] == "lattice" else _groups(case)
    n += case.get("spread", 0)
    return sum(16.0 * s * s * (c * ((n + 1) ** 2 + (n + 1) * M) + 3 * (n + 1) ** 2) for s, c in grp)


def work(case):
    """Per Dyson / VIE2 solve of a group: every G^tv history, the shared Sigma (two triangles and
    the tv rows) and the problems' time-step slices move once; 8 s^3 flops per s x s complex product
    of the history sums (ret and les recursions, Sigma^< G^A, Sigma^tv G^vt, Matsubara, tv)."""
    kind, M = case["kind"], case["ntau"] + 1

    def solve(s, c, n, hist):
        by = 16.0 * s * s * (c * (n * M * hist + 2 * M + 2 * n) + n * n + n * M)
        return by, 8.0 * s ** 3 * c * (n * n + n * n + 2 * n * M + M * M)
    if kind == "conv":
        n, s, c = case["n"], case["s"], case["count"]
        return dict(bytes=16.0 * s * s * c * (2.0 * n * n + 2 * n * M + 2 * n + M),
                    flops=8.0 * s ** 3 * c * (n * n / 2 + M * M + n * M + n * M + n * n + n * n / 2))
    if kind == "lattice":
        calls = [(1, case["nk"], n, 1.0) for n in range(case["n0"], case["n"] + 1) for _ in range(case["ncorr"])]
    elif kind == "run":
        calls = [(s, c, n, 1.0) for s, c in _groups(case) for n in range(case["k"] + 1, case["n"] + 1)]
    else:
        calls = [(s, c, case["n"], 0.5 if case.get("mixed") else 1.0) for s, c in _groups(case)] * case.get("ncorr", 1)
    tot = [solve(*c) for c in calls]
    return dict(bytes=float(sum(t[0] for t in tot)), flops=float(sum(t[1] for t in tot)))


# ---- inputs ---------------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _fermi_exp(eps, tau, beta):
    """e^{eps tau} f(eps), shapes broadcast."""
    return torch.where(eps > 0, torch.exp(-eps * (beta - tau)) / (1 + torch.exp(-beta * eps.abs())),
                       torch.exp(eps * tau) / (1 + torch.exp(-beta * eps.abs())))


class _Bath:
    """X(t, t') = a(t) g(t, t') b(t') W with g the function of a discrete semicircular bath; a, b
    real envelopes, W an s x s matrix.  Its hermitian partner has a and b exchanged and W^dagger."""

    def __init__(self, gen, nt, ntau, s, beta, h, scale, hermitian=True):
        dev = _dev()
        r = torch.rand(6, generator=gen, dtype=F64).tolist()
        eps = torch.linspace(-2, 2, 65, dtype=F64)[1:-1]
        w = torch.sqrt(4 - eps * eps)
        self.w = (w / w.sum()).to(dev)
        self.eps = (eps + 0.4 * (r[0] - 0.5)).to(dev)
        self.nt, self.ntau, self.s, self.beta, self.h = nt, ntau, s, beta, h
        t = h * torch.arange(-1, nt + 1, dtype=F64, device=dev)
        t[0] = 0.0
        self.a = scale * (1 + 0.2 * r[1] * torch.sin((1 + r[2]) * t))
        self.b = self.a if hermitian else scale * (1 + 0.2 * r[3] * torch.sin((1 + r[4]) * t))
        X = torch.randn(s, s, 2, generator=gen, dtype=F64)
        X = torch.view_as_complex(X).to(dev)
        X = 0.5 * (X + X.conj().T) if hermitian else X
        self.W = torch.eye(s, dtype=C128, device=dev) + 0.15 * X
        self.tau = torch.arange(ntau + 1, dtype=F64, device=dev) * (beta / ntau)

    def partner(self):
        o = object.__new__(_Bath)
        o.__dict__.update(self.__dict__)
        o.a, o.b, o.W = self.b, self.a, self.W.conj().T.contiguous()
        return o

    def _g(self, kind):
        d = self.h * torch.arange(self.nt + 1, dtype=F64, device=_dev())
        ph = torch.exp(1j * d[:, None] * self.eps)
        if kind == "ret":  # g(t, t - d)
            return -1j * (ph.conj() * self.w).sum(1)
        if kind == "les":  # g^<(t - d, t)
            return 1j * (ph * (self.w * _fermi_exp(self.eps, 0 * self.eps, self.beta))).sum(1)
        f = _fermi_exp(self.eps[:, None], self.tau, self.beta)
        return 1j * (ph.conj() * self.w) @ f.to(C128)

    def dense(self, kind):
        """ret: X^R(t, t') for t >= t'; les: X^<(t', t) for t' <= t, both (nt+1, nt+1, s, s)."""
        t = torch.arange(self.nt + 1, device=_dev())
        d = t[:, None] - t[None, :]
        a, b = self.a[1:], self.b[1:]
        if kind == "les":
            d = -d
        v = self._g(kind)[d.clamp(min=0)] * (d >= 0) * a[:, None] * b[None, :]
        return v[:, :, None, None] * self.W

    def tri(self, kind):
        D = self.dense(kind)
        i = torch.tril_indices(self.nt + 1, self.nt + 1, device=_dev())
        return D[i[0], i[1]] if kind == "ret" else D[i[1], i[0]]

    def tv(self):
        return (self._g("tv") * self.a[1:, None] * self.b[0])[:, :, None, None] * self.W

    def mat(self):
        f = _fermi_exp(-self.eps[:, None], self.tau, self.beta)  # e^{-eps tau} (1 - f)
        return -(self.a[0] * self.b[0] * (self.w @ f)).to(C128)[:, None, None] * self.W

    def host(self):
        return SimpleNamespace(**{c: x.cpu().numpy() for c, x in
                                  dict(ret=self.tri("ret"), les=self.tri("les"), tv=self.tv(), mat=self.mat()).items()})

    def slice(self, n, R=None, L=None, T=None):
        """[ret(n, 0..n) | tv(n, .) | les(0..n, n)]"""
        R = self.dense("ret")[n, :n + 1] if R is None else R
        L = self.dense("les")[:n + 1, n] if L is None else L
        T = self.tv()[n] if T is None else T
        return torch.cat([R, T, L])


class _Levels:
    """Problem Hamiltonians H_p(t) (levels in [-2, 2], weak hybridisation, a field pulse) and the free
    propagators of H_p(-1)."""

    def __init__(self, gen, P, nt, ntau, s, beta, h):
        dev = _dev()
        e = 4 * torch.rand(P, s, generator=gen, dtype=F64) - 2
        X = torch.view_as_complex(torch.randn(P, s, s, 2, generator=gen, dtype=F64))
        D = torch.view_as_complex(torch.randn(P, s, s, 2, generator=gen, dtype=F64))
        H0 = torch.diag_embed(e).to(C128) + 0.1 * (X + X.mH) * (s > 1)
        self.H0 = H0.to(dev)
        t = h * torch.arange(nt + 1, dtype=F64)
        A = torch.cat([torch.zeros(1, dtype=F64), torch.exp(-(t - 2) ** 2) * torch.sin(3 * t)])
        self.H = (H0[:, None] + 0.15 * A[None, :, None, None] * (D + D.mH)[:, None]).to(dev)
        self.E, self.V = torch.linalg.eigh(self.H0)
        self.nt, self.ntau, self.s, self.beta, self.h = nt, ntau, s, beta, h
        self.tau = torch.arange(ntau + 1, dtype=F64, device=dev) * (beta / ntau)

    def _mat(self, p, d):  # V diag(d[..., l]) V^dagger
        return (self.V[p] * d[..., None, :].to(C128)) @ self.V[p].mH

    def u(self, p, t):
        return torch.exp(-1j * self.h * t[:, None] * self.E[p])

    def tv(self, p, rows):
        """G^tv(0..rows-1, .)"""
        ph = self.u(p, torch.arange(rows, dtype=F64, device=_dev()))
        f = _fermi_exp(self.E[p][None, :], self.tau[:, None], self.beta)
        V = self.V[p]
        x = torch.einsum("tl,mlbc->tmbc", 1j * ph, torch.einsum("bl,ml,cl->mlbc", V, f.to(C128), V.conj()))
        return x.contiguous()

    def mat(self, p):
        return -self._mat(p, _fermi_exp(-self.E[p][None, :], self.tau[:, None], self.beta)).contiguous()

    def ret(self, p, t):
        d = torch.arange(t, -1, -1, dtype=F64, device=_dev())
        return -1j * self._mat(p, self.u(p, d))

    def les(self, p, t):
        d = torch.arange(t, -1, -1, dtype=F64, device=_dev())
        return 1j * self._mat(p, self.u(p, d).conj() * _fermi_exp(self.E[p], 0 * self.E[p], self.beta))

    def slice(self, p, t, tv=None):
        tv = self.tv(p, t + 1)[t] if tv is None else tv
        return torch.cat([self.ret(p, t), tv, self.les(p, t)])


def _problems(case, seed):
    """Per group: bath (Sigma, or F of a VIE2 group), levels, the problems' lengths and the first
    problem index."""
    gen = torch.Generator().manual_seed(seed)
    out, p0 = [], 0
    for s, c in [(1, case["nk"])] if case["kind"] == "lattice" else _groups(case):
        nts = [case["n"] + (int(torch.randint(0, case["spread"] + 1, (1,), generator=gen)) if case.get("spread") else 0)
               for _ in range(c)]
        N = max(nts)
        vie = case["kind"] == "vie2"
        bath = _Bath(gen, N, case["ntau"], s, case["beta"], case["h"], 0.6 if vie else 0.5, hermitian=not vie)
        lev = _Levels(gen, c, N, case["ntau"], s, case["beta"], case["h"])
        out.append(SimpleNamespace(s=s, c=c, N=N, nts=nts, bath=bath, lev=lev, p0=p0))
        p0 += c
    return out


def _pinned(n_cplx):
    t = torch.empty(n_cplx, dtype=C128, pin_memory=torch.cuda.is_available())
    return t, t.numpy()


def _np(x):
    return np.ascontiguousarray(x.cpu().numpy())


def _upload_history(b, p, lev, q, nt, rows):
    """G^tv(0..rows-1) and G^mat of problem p from its free propagator; later rows zero."""
    M, s = lev.ntau + 1, lev.s
    buf, arr = _pinned((nt + 1) * M * s * s)
    buf[:rows * M * s * s].copy_(lev.tv(q, rows).reshape(-1))
    buf[rows * M * s * s:].zero_()
    b.set_G(p, SimpleNamespace(ret=None, les=None, tv=arr, mat=_np(lev.mat(q))))


def _batch(case, grp):
    descs = [dict(nt=nt, ntau=case["ntau"], size1=g.s, sig=-1, solve_order=case["k"], sigma_group=i,
                  beta=case["beta"], h=case["h"], mu=0.0) for i, g in enumerate(grp) for nt in g.nts]
    return gpu.Batch(descs, gpu.PREC_MIXED if case.get("mixed") else gpu.PREC_FP64)


def _out(grp, n, M):
    """One pinned array per group for its problems' slices of time step n."""
    return [_pinned(g.c * (2 * (n + 1) + M) * g.s * g.s)[1].reshape(g.c, 2 * (n + 1) + M, g.s, g.s) for g in grp]


def prepare(case, seed):
    kind, n, k, M = case["kind"], case["n"], case["k"], case["ntau"] + 1
    if kind == "conv":
        return _prepare_conv(case, seed)
    grp = _problems(case, seed)
    b = _batch(case, grp)
    st = SimpleNamespace(case=case, b=b, grp=grp)
    for i, g in enumerate(grp):
        if kind == "vie2":
            F, Fc = g.bath.host(), g.bath.partner().host()
            Fc.mat = None
            b.set_F(i, F, Fc)
        else:
            b.set_sigma(i, g.bath.host())
        for q in range(g.c):
            if kind != "vie2":
                b.set_H(g.p0 + q, _np(g.lev.H[q][:g.nts[q] + 2]))
    if kind == "lattice":
        U = np.zeros((n + 2, 1), np.complex128)
        U[0], U[1:, 0] = case["umat"], 2 * np.minimum(np.arange(n + 1) * case["h"] / 2, 1.0)
        b.set_U(0, U)
    n0 = k + 1 if kind == "run" else case.get("n0", n)
    for g in grp:
        for q in range(g.c):
            p = g.p0 + q
            if kind == "run" or (kind == "lattice" and n0 == k + 1):
                b.set_timestep(p, -1, _np(g.lev.mat(q)))
            else:
                _upload_history(b, p, g.lev, q, g.nts[q], n)
            if kind in ("run", "lattice"):
                tv = g.lev.tv(q, n0)
                for t in range(n0 - k - 1, n0):
                    b.set_timestep(p, t, _np(g.lev.slice(q, t, tv[t])))
            if kind == "vie2":
                b.set_Q_timestep(p, n, _np(g.lev.slice(q, n)))
    if kind == "step":
        st.slices = []
        for it in range(case["ncorr"]):
            f = 1 + 0.01 * (case["ncorr"] - 1 - it)
            st.slices.append([_np(f * g.bath.slice(n)) for g in grp])
    if kind in ("step", "vie2"):
        st.out = _out(grp, n, M)
    if kind == "run":
        st.G = [SimpleNamespace(ret=np.zeros(((n + 1) * (n + 2) // 2, g.s, g.s), np.complex128),
                                les=np.zeros(((n + 1) * (n + 2) // 2, g.s, g.s), np.complex128),
                                tv=np.zeros((n + 1, M, g.s, g.s), np.complex128), mat=None)
                for g in grp for _ in range(g.c)]
    if kind == "lattice":
        if n0 == k + 1:
            for t in range(-1, k + 1):
                b.gloc_timestep(0, t)
                b.sigma_2b_timestep(0, t)
        st.stream = torch.cuda.Stream()
        b.set_stream(st.stream.cuda_stream)
        st.views = b.gloc_views(0)
        if case["graph"]:
            b.graph_record(gpu.Batch.GRAPH_LATTICE, n0, n, case["ncorr"])
    b.synchronize()
    return st


def run(st):
    case = st.case
    kind, n = case["kind"], case["n"]
    if kind == "step":
        for sl in st.slices:
            for i in range(len(st.grp)):
                st.b.set_sigma_timestep(i, n, sl[i])
            st.b.dyson_timestep(n)
    elif kind == "vie2":
        st.b.vie2_timestep(n)
    elif kind == "run":
        for t in range(case["k"] + 1, n + 1):
            st.b.dyson_timestep(t)
        for p, G in enumerate(st.G):
            st.b.get_G(p, G)
        return [[G.ret, G.les, G.tv] for G in st.G]
    elif kind == "lattice":
        if case["graph"]:
            st.b.graph_launch()
        else:
            for t in range(case["n0"], n + 1):
                st.b.lattice_2b_timestep(t, case["ncorr"])
        with torch.cuda.stream(st.stream):  # the batch's stream; the views end with the batch
            return [st.views[c].clone() for c in ("ret", "les", "tv")]
    else:
        gpu.convolution_timestep_dev(n, *st.ptrs, n, case["ntau"], case["s"], -1, -1, case["k"], case["beta"],
                                     case["h"], torch.cuda.current_stream().cuda_stream)
        return st.C[:3]
    for g, out in zip(st.grp, st.out):
        for q in range(g.c):
            st.b.get_timestep(g.p0 + q, n, out[q])
    return st.out


def _conv_baths(case, seed):
    gen = torch.Generator().manual_seed(seed)
    mk = lambda: _Bath(gen, case["n"], case["ntau"], case["s"], case["beta"], case["h"], 0.8, hermitian=False)
    return [(mk(), mk()) for _ in range(case["count"])]


def _prepare_conv(case, seed):
    st = SimpleNamespace(case=case, keep=[])
    n, M, s, cnt = case["n"], case["ntau"] + 1, case["s"], case["count"]
    tri = (n + 1) * (n + 2) // 2
    st.C = [torch.zeros((cnt,) + d + (s, s), dtype=C128, device=_dev()) for d in ((tri,), (tri,), (n + 1, M), (M,))]
    sets = [[[x[i].data_ptr() for x in st.C] for i in range(cnt)], [], [], [], []]  # C, A, Acc, B, Bcc
    for A, B in _conv_baths(case, seed):
        for i, x in ((1, A), (2, A.partner()), (3, B), (4, B.partner())):
            hm = [x.tri("ret"), x.tri("les"), x.tv().contiguous(), x.mat().contiguous()]
            st.keep.append(hm)
            sets[i].append([y.data_ptr() for y in hm])
    st.ptrs = sets
    torch.cuda.synchronize()
    return st


# ---- the discretised equations in plain torch -------------------------------------------------
def _solve_fractions(A, b):
    n = len(A)
    A = [r[:] + [x] for r, x in zip(A, b)]
    for c in range(n):
        p = next(i for i in range(c, n) if A[i][c] != 0)
        A[c], A[p] = A[p], A[c]
        A[c] = [x / A[c][c] for x in A[c]]
        for i in range(n):
            if i != c and A[i][c] != 0:
                A[i] = [x - A[i][c] * y for x, y in zip(A[i], A[c])]
    return [r[n] for r in A]


def _mul(a, b):
    o = [Fraction(0)] * (len(a) + len(b) - 1)
    for i, x in enumerate(a):
        for j, y in enumerate(b):
            o[i + j] += x * y
    return o


def _lagrange(nodes):
    out = []
    for l, xl in enumerate(nodes):
        p = [Fraction(1)]
        for xj in nodes:
            if xj != xl:
                p = _mul(p, [Fraction(-xj, xl - xj), Fraction(1, xl - xj)])
        out.append(p)
    return out


class _Tables:
    """Integration and differentiation weights of order k on unit steps."""

    def __init__(self, k, N):
        L = _lagrange(list(range(k + 1)))
        ev = lambda p, x: sum(c * x ** i for i, c in enumerate(p))
        integral = lambda p, x: sum(c * Fraction(x ** (i + 1), i + 1) for i, c in enumerate(p))
        self.diff = [[float(sum(i * c * x ** (i - 1) for i, c in enumerate(p) if i)) for p in L] for x in range(k + 1)]
        self.bd = [float(p[1]) for p in _lagrange([-l for l in range(k + 2)])]
        self.rcorr = np.zeros((max(k, 1), k + 1, k + 1))
        for m in range(1, k):
            for a in range(k + 1):
                # L_a(m - x) by composition
                comp = [Fraction(0)] * (k + 1)
                for i, c in enumerate(L[a]):
                    for j in range(i + 1):
                        comp[j] += c * comb(i, j) * m ** (i - j) * (-1) ** j
                for l in range(k + 1):
                    self.rcorr[m, a, l] = float(integral(_mul(comp, L[l]), m))
        # end weights: 1 - a_j removes the Euler-Maclaurin terms of degrees 0..k
        B = [Fraction(1)]
        for m in range(1, k + 2):
            B.append(-sum(comb(m + 1, i) * B[i] for i in range(m)) / (m + 1))
        e = [-B[m + 1] / (m + 1) for m in range(k + 1)]
        d = _solve_fractions([[Fraction(j ** m if (j or m) else 1) for j in range(k + 1)] for m in range(k + 1)], e)
        om = [1 - x for x in d]
        self.omega = [float(x) for x in om]
        W = np.zeros((N + 1, N + 1))
        af = np.ones(N + 1)
        af[:min(k, N) + 1] = [float(x) for x in om][:N + 1]
        for n in range(N + 1):
            if n <= k:
                W[n, :k + 1] = [float(integral(p, n)) for p in L]
            elif n < 2 * k + 2:
                a = [om[j] if j <= k else Fraction(1) for j in range(n + 1)]
                W[n, :n + 1] = [float(a[j] + a[n - j] - 1) for j in range(n + 1)]
            else:
                W[n, :n + 1] = 1
                W[n, :k + 1] = af[:k + 1]
                W[n, n - k:n + 1] = af[:k + 1][::-1]
        self.W = torch.tensor(W, device=_dev())
        self.k = k
        self.ext = [(-1) ** l * comb(k + 1, l + 1) for l in range(k + 1)]


def _matop(tab, A, ntau, sig, beta):
    """K with dtau * int [A(tau - x) B(x)] = K B: ((m a), (x c)) from A(tau), tau = 0..ntau."""
    k, M, s, dtau = tab.k, ntau + 1, A.shape[-1], beta / ntau
    K = torch.zeros(M, M, s, s, dtype=C128, device=A.device)
    for m in range(M):
        r = ntau - m
        if r >= k:
            K[m, :r + 1] += tab.W[r, :r + 1, None, None] * A[m:]
        else:
            for l in range(k + 1 if r > 0 else 0):
                for j in range(k + 1):
                    K[m, j] += tab.rcorr[r, l, j] * A[ntau - l]
        if m >= k:
            K[m, r:] += sig * (tab.W[m, :m + 1, None, None] * A[:m + 1].flip(0)).flip(0)
        else:
            for l in range(k + 1 if m > 0 else 0):
                for j in range(k + 1):
                    K[m, ntau - l] += sig * tab.rcorr[m, l, j] * A[j]
    return dtau * K.permute(0, 2, 1, 3).reshape(M * s, M * s)


def _rows(x):  # (i, j, a, b) -> ((i a), (j b))
    return x.permute(0, 2, 1, 3).reshape(x.shape[0] * x.shape[2], -1)


def _step(tab, case, n, S, Scc, gmat, hist, H, Q=None, sig=-1):
    """Time step n > k of P problems sharing S = dict(ret, les: dense (n+1, n+1, s, s), tv (n+1, M, s, s)):
    Dyson with Hamiltonians H (P, >= n+2, s, s), or [1 + S] G = Q with the slices Q.  hist(p) gives
    G^tv(0..n-1).  Returns (ret (P, n+1, s, s), tv (P, M, s, s), les (P, n+1, s, s))."""
    k, h, beta, ntau = tab.k, case["h"], case["beta"], case["ntau"]
    vie, M, s, P = Q is not None, ntau + 1, S["ret"].shape[-1], gmat.shape[0]
    dev, sg = S["ret"].device, 1.0 if Q is None else -1.0
    eye = torch.eye(s, dtype=C128, device=dev)
    w0, ih = h * tab.omega[0], 1j / h
    T, R = S["ret"], Scc["ret"]
    idx = torch.arange(n + 1, device=dev)
    # step matrices of every row
    if vie:
        Ml = (eye + w0 * T[idx, idx]).expand(P, -1, -1, -1)
        Mr = (eye + w0 * R[idx, idx]).expand(P, -1, -1, -1)
    else:
        Ml = ih * tab.bd[0] * eye - H[:, 1:n + 2] - w0 * T[idx, idx]
        Mr = ih * tab.bd[0] * eye - H[:, 1:n + 2].mH - w0 * R[idx, idx]
    Mli, Mri = torch.linalg.inv(Ml), torch.linalg.inv(Mr)
    # retarded row
    x = torch.zeros(P, n + 1, s, s, dtype=C128, device=dev)
    x[:, n] = Q[:, n] if vie else -1j * eye
    B = torch.zeros(P, k + 1, k + 1, s, s, dtype=C128, device=dev)  # B[l, j]
    for j in range(1, k + 1):
        for l in range(k + 1):
            st = R[n - l, n - j] if l <= j else -T[n - j, n - l].mH
            if vie:
                B[:, l, j] = (eye if l == j else 0) + h * tab.W[j, l] * st
            else:
                B[:, l, j] = ih * tab.diff[j][l] * eye - (H[:, n - j + 1] if l == j else 0) - h * tab.W[j, l] * st
    rhs = torch.stack([(Q[:, n - j] if vie else 0) - x[:, n] @ B[:, 0, j] for j in range(1, k + 1)], 1)
    A = B[:, 1:, 1:].permute(0, 1, 3, 2, 4).reshape(P, k * s, k * s)
    X = torch.linalg.solve(A, rhs.permute(0, 2, 1, 3).reshape(P, s, k * s), left=False)
    x[:, n - k:n] = X.reshape(P, s, k, s).permute(0, 2, 1, 3).flip(1)
    for j in range(n - k - 1, -1, -1):
        w = tab.W[n - j, :n - j].flip(0)
        Y = (w[None, :, None, None] * x[:, j + 1:]).permute(0, 2, 1, 3).reshape(P * s, -1)
        v = sg * h * (Y @ R[j + 1:n + 1, j].reshape(-1, s)).reshape(P, s, s)
        if vie:
            v = v + Q[:, j]
        else:
            for p in range(1, k + 2):
                v = v - ih * tab.bd[p] * x[:, j + p]
        x[:, j] = v @ Mri[:, j]
    # left-mixing row
    c = sg * h * tab.W[n, :n, None, None] * T[n, :n]
    if not vie:
        for p in range(1, k + 2):
            c[n - p] -= ih * tab.bd[p] * eye
    C = sg * _matop(tab, S["tv"][n], ntau, sig, beta) @ gmat.permute(1, 2, 0, 3).reshape(M * s, P * s)
    C = C.reshape(M, s, P, s).permute(2, 0, 1, 3)
    tv = torch.empty(P, M, s, s, dtype=C128, device=dev)
    c = c.permute(1, 0, 2).reshape(s, n * s)
    for p in range(P):
        q = (c @ hist(p)[:n].permute(0, 2, 1, 3).reshape(n * s, M * s)).reshape(s, M, s).permute(1, 0, 2) + C[p]
        if vie:
            q = q + Q[p, n + 1:n + 1 + M]
        tv[p] = Mli[p, n] @ q
    # lesser column
    bt = 1j * (beta / ntau) * sig * tab.W[ntau, :M, None, None] * tv.flip(1).mH
    ba = h * tab.W[n, :n + 1, None, None] * x.mH
    L = S["les"] - _upper(Scc["les"]).permute(1, 0, 3, 2).conj()
    gl = _rows(S["tv"][:n + 1]) @ bt.permute(1, 2, 0, 3).reshape(M * s, P * s) \
        + _rows(L) @ ba.permute(1, 2, 0, 3).reshape((n + 1) * s, P * s)
    gl = sg * gl.reshape(n + 1, s, P, s).permute(2, 0, 1, 3)
    if vie:
        gl = gl + Q[:, n + 1 + M:]
    y = torch.zeros(P, n + 1, s, s, dtype=C128, device=dev)
    j0 = 0 if vie else 1
    if not vie:
        y[:, 0] = -tv[:, 0].mH
    for j in range(k + 1):
        for m in range(k + 1):
            st = T[j, m] if j >= m else -R[m, j].mH
            if vie:
                B[:, j, m] = (eye if j == m else 0) + h * tab.W[j, m] * st
            else:
                B[:, j, m] = ih * tab.diff[j][m] * eye - (H[:, j + 1] if j == m else 0) - h * tab.W[j, m] * st
    K = k + 1 - j0
    A = B[:, j0:, j0:].permute(0, 1, 3, 2, 4).reshape(P, K * s, K * s)
    rhs = torch.stack([gl[:, j] - (0 if vie else B[:, j, 0] @ y[:, 0]) for j in range(j0, k + 1)], 1)
    y[:, j0:k + 1] = torch.linalg.solve(A, rhs.reshape(P, K * s, s)).reshape(P, K, s, s)
    for j in range(k + 1, n + 1):
        Y = (tab.W[j, :j, None, None, None] * y[:, :j].permute(1, 2, 0, 3)).reshape(j * s, P * s)
        Tj = T[j, :j].permute(1, 0, 2).reshape(s, j * s)
        v = gl[:, j] + sg * h * (Tj @ Y).reshape(s, P, s).permute(1, 0, 2)
        if not vie:
            for p in range(1, k + 2):
                v = v - ih * tab.bd[p] * y[:, j - p]
        y[:, j] = Mli[:, j] @ v
    return x, tv, y


def _dense(bath, n):
    N = n + 1
    return dict(ret=bath.dense("ret")[:N, :N], les=bath.dense("les")[:N, :N], tv=bath.tv()[:N])


def _sigma_2b(gr, gl, gtv, Un, Um, U0):
    """Sigma_2B of one orbital from G_loc(n, .): ret and les over m, tv over tau."""
    lt = -gl.conj()                    # G^<(n, m)
    gt = gr + lt                       # G^>(n, m)
    pl = Um * (-1j * gl * gt) * Un
    pr = Un * (-(1j * gt * gl - 1j * lt * (gl - gr.conj()))) * Um
    ret = 1j * gt * (pr - pl.conj()) - 1j * gl.conj() * pl.conj()
    les = 1j * gl * pl
    tv = 1j * gtv * (Un * U0 * (-1j * gtv * gtv.flip(0).conj()))
    return ret, les, tv


def _exact_lattice(case, seed):
    n0, n, k, M = case["n0"], case["n"], case["k"], case["ntau"] + 1
    g = _problems(case, seed)[0]
    dev, P = _dev(), g.c
    tab = _Tables(k, max(n, case["ntau"]))
    ret, les, tvr = {}, {}, {}  # G_k rows by time step, (P, ...)
    first = n0 - k - 1
    late = n0 > k + 1
    tvh = torch.empty(P, n + 1, M, 1, 1, dtype=C128, device=dev) if not late else None
    for t in range(first, n0):
        ret[t] = torch.stack([g.lev.ret(q, t) for q in range(P)])[..., 0, 0]
        les[t] = torch.stack([g.lev.les(q, t) for q in range(P)])[..., 0, 0]
    if late:
        hist = lambda p: g.lev.tv(p, n)
        tvr = {t: torch.empty(P, M, dtype=C128, device=dev) for t in range(first, n0)}
        for q in range(P):
            x = g.lev.tv(q, n0)[..., 0, 0]
            for t in tvr:
                tvr[t][q] = x[t]
    else:
        for q in range(P):
            tvh[q, :n0] = g.lev.tv(q, n0)
        hist = lambda p: tvh[p]
    gmat = torch.stack([g.lev.mat(q) for q in range(P)])
    Uh = torch.tensor([case["umat"]] + [2 * min(t * case["h"] / 2, 1.0) for t in range(n + 1)], dtype=F64, device=dev)
    S = _dense(g.bath, n)
    loc = dict(ret=torch.zeros(n + 1, n + 1, dtype=C128, device=dev), les=torch.zeros(n + 1, n + 1, dtype=C128, device=dev),
               tv=torch.zeros(n + 1, M, dtype=C128, device=dev))

    def gloc(t):
        loc["ret"][t, :t + 1] = ret[t].mean(0)
        loc["les"][:t + 1, t] = les[t].mean(0)
        loc["tv"][t] = (tvr[t] if late else tvh[:, t, :, 0, 0]).mean(0)

    def sigma(t):
        a, b, c = _sigma_2b(loc["ret"][t, :t + 1], loc["les"][:t + 1, t], loc["tv"][t], Uh[t + 1], Uh[1:t + 2], Uh[0])
        S["ret"][t, :t + 1, 0, 0], S["les"][:t + 1, t, 0, 0], S["tv"][t, :, 0, 0] = a, b, c
    if not late:
        for t in range(k + 1):
            gloc(t)
            sigma(t)
    for t in range(n0, n + 1):
        # polynomial predictor of step t from t-1-k..t-1
        r, l = torch.zeros(P, t + 1, dtype=C128, device=dev), torch.zeros(P, t + 1, dtype=C128, device=dev)
        v = 0
        for i, c in enumerate(tab.ext):
            u = t - 1 - i
            v = v + c * (tvr[u] if late else tvh[:, u, :, 0, 0])
            for j in range(k + 1):
                r[:, j] += c * (ret[u][:, j] if u >= j else -ret[j][:, u].conj())
                l[:, j] += c * (les[u][:, j] if u >= j else -les[j][:, u].conj())
            r[:, k + 1:] += c * ret[u][:, k - i:]
            l[:, k + 1:] += c * les[u][:, k - i:]
        ret[t], les[t] = r, l
        if late:
            tvr[t] = v
        else:
            tvh[:, t, :, 0, 0] = v
        sub = lambda: {c: (x[:t + 1, :t + 1] if c != "tv" else x[:t + 1]) for c, x in S.items()}
        for _ in range(case["ncorr"]):
            gloc(t)
            sigma(t)
            a, b, c = _step(tab, case, t, sub(), sub(), gmat, hist, g.lev.H)
            ret[t], les[t] = a[..., 0, 0], c[..., 0, 0]
            if late:
                tvr[t] = b[..., 0, 0]
            else:
                tvh[:, t] = b
        gloc(t)
    i = torch.tril_indices(n + 1, n + 1, device=dev)
    flat = lambda x: torch.view_as_real(x.contiguous()).reshape(-1)
    return [flat(loc["ret"][i[0], i[1]]), flat(loc["les"][i[1], i[0]]), flat(loc["tv"])]


def _exact_conv(case, seed):
    n, k, h, beta, ntau = case["n"], case["k"], case["h"], case["beta"], case["ntau"]
    tab, dtau = _Tables(k, max(n, ntau)), beta / ntau
    W, s, M = tab.W, case["s"], ntau + 1
    i = torch.tril_indices(n + 1, n + 1, device=_dev())
    full = lambda X, Xc: X - _lower(Xc).permute(1, 0, 3, 2).conj()
    out = []
    for A, B in _conv_baths(case, seed):
        Ac, Bc = A.partner(), B.partner()
        AR, BR = full(A.dense("ret"), Ac.dense("ret")), full(B.dense("ret"), Bc.dense("ret"))
        AL = A.dense("les") - _upper(Ac.dense("les")).permute(1, 0, 3, 2).conj()
        # retarded: weights w(n - j, n - m)
        wr = W[:n + 1, :n + 1].flip(0).flip(1)  # [j, m]
        ret = h * torch.einsum("jm,mab,mjbc->jac", wr.to(C128), AR[n], BR)
        tv = (_matop(tab, A.tv()[n], ntau, -1, beta) @ B.mat().reshape(M * s, s)).reshape(M, s, s) \
            + h * torch.einsum("j,jab,jmbc->mac", W[n, :n + 1].to(C128), A.dense("ret")[n], B.tv())
        bt = -1j * dtau * W[ntau, :M, None, None] * Bc.tv()[n].flip(0).mH
        les = torch.einsum("jmab,mbc->jac", A.tv(), bt)
        les = les + torch.einsum("jmab,mbc->jac", AL, h * W[n, :n + 1, None, None] * Bc.dense("ret")[n].mH)
        les = les + h * torch.einsum("jm,jmab,mbc->jac", W[:n + 1, :n + 1].to(C128), AR, B.dense("les")[:, n])
        C = dict(ret=torch.zeros_like(AR), les=torch.zeros_like(AR), tv=torch.zeros_like(A.tv()))
        C["ret"][n], C["les"][:, n], C["tv"][n] = ret, les, tv
        out.append([C["ret"][i[0], i[1]], C["les"][i[1], i[0]], C["tv"]])
    return [torch.stack(x) for x in zip(*out)]


def _lower(x):  # strictly lower (t > t') part of a dense (t, t', s, s) function
    t = torch.arange(x.shape[0], device=x.device)
    return x * (t[:, None] > t[None, :])[:, :, None, None]


def _upper(x):
    t = torch.arange(x.shape[0], device=x.device)
    return x * (t[:, None] < t[None, :])[:, :, None, None]


def exact(case, seed):
    kind, n, k, M = case["kind"], case["n"], case["k"], case["ntau"] + 1
    if kind == "conv":
        return _exact_conv(case, seed)
    if kind == "lattice":
        return _exact_lattice(case, seed)
    tab = _Tables(k, max(n, case["ntau"]))
    out = []
    for g in _problems(case, seed):
        S = _dense(g.bath, n)
        gmat = torch.stack([g.lev.mat(q) for q in range(g.c)])
        if kind == "run":
            tv = torch.stack([g.lev.tv(q, n + 1) for q in range(g.c)])
            i = torch.tril_indices(n + 1, n + 1, device=_dev())
            R = torch.zeros(g.c, n + 1, n + 1, g.s, g.s, dtype=C128, device=_dev())
            L = torch.zeros_like(R)
            for q in range(g.c):
                for t in range(k + 1):
                    R[q, t, :t + 1], L[q, :t + 1, t] = g.lev.ret(q, t), g.lev.les(q, t)
            for t in range(k + 1, n + 1):
                sub = {c: (x[:t + 1, :t + 1] if c != "tv" else x[:t + 1]) for c, x in S.items()}
                a, b, c = _step(tab, case, t, sub, sub, gmat, lambda p: tv[p], g.lev.H)
                R[:, t, :t + 1], tv[:, t], L[:, :t + 1, t] = a, b, c
            out += [[R[q][i[0], i[1]], L[q][i[1], i[0]], tv[q]] for q in range(g.c)]
            continue
        Sc, Q = S, None
        if kind == "vie2":
            Sc = _dense(g.bath.partner(), n)
            Q = torch.stack([g.lev.slice(q, n) for q in range(g.c)])
        x, tv, y = _step(tab, case, n, S, Sc, gmat, lambda p: g.lev.tv(p, n), g.lev.H, Q)
        out.append(torch.cat([x, tv, y], 1))
    return out
