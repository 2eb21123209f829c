"""Performance cases of the VMC hot path, through the package's public entry points.

A case is one call (or the few calls a program makes together) on a context that the program keeps:

* ``sample``       Context.make_sample and its stored samples (make_sample.f90:4)
* ``batch``        Batch.make_sample over two lattices in one launch
* ``measure``      Context.measure on stored samples: energy scalars, force and mean derivative
                   (calc_phys_quantity.f90:20)
* ``eval``         Context.eval_configs: psi, H psi and O_k of configurations in host memory
* ``eval_device``  Context.eval_configs_noalloc: the same on buffers in device memory
* ``correlation``  Context.measure_correlation (Calc_Correlation/calc_phys_quantity.f90:264)
* ``sr``           one stochastic-reconfiguration step on given samples: parameters in, measurement, S, solve,
                   new parameters out (main.f90:311-453 without make_sample)
* ``iteration``    one whole optimisation step, Context.iteration
* ``transverse``   make_sample and measure with the transverse spin projection (full skew Pfaffian matrix)

Lattices, projections, densities and sample counts are the ones of bench.py's workloads and of the tests;
parameters are formats.synthetic_problem's seeded inputs, as everywhere in this repository.
"""
import math

import numpy as np
import torch

from rbm_pp_b200 import capi
from rbm_pp_b200 import formats as fm


def _case(name, kind, L, trans, alpha, walkers, ns, **more):
    c = dict(name=name, kind=kind, L=L, trans=trans, alpha=alpha, alphac=0, orbital="full", walkers=walkers, ns=ns,
             J2=0.5, split=False, s_factor0=1e-3)
    c.update(more)
    return c


def listed():
    return [
        # a handful of configurations evaluated from host memory with complex units: the smallest call, where
        # latency counts (a driver's or a notebook's spot check)
        _case("eval_4x4_complex", "eval", 4, True, 1, 1, 24, alphac=1),
        # O_k, psi and H psi of a batch in device buffers: the derivative check on an ordinary lattice
        _case("eval_8x8_trans", "eval_device", 8, True, 2, 1, 500),
        # the 4x4 optimisation that is compared with exact diagonalisation: 1024 samples over 8 walkers per step
        _case("iteration_4x4", "iteration", 4, False, 1, 8, 128),
        # sampling of the small translation-symmetric bench workload
        _case("sample_6x6_trans", "sample", 6, True, 2, 256, 16),
        # sampling of the 10x10 translation-symmetric state, one walker per SM: the part of an SR step that takes
        # most of its time
        _case("sample_10x10_trans", "sample", 10, True, 4, 148, 1),
        # sampling without translation projection on a larger lattice (two Pfaffian blocks per walker)
        _case("sample_12x12", "sample", 12, False, 2, 256, 4),
        # two lattices of uneven Pfaffian size in one launch
        _case("batch_12_14", "batch", 12, False, 2, 75, 2, L2=14, J2=0.45),
        # estimators of the 10x10 translation-symmetric state: local energy, O_k, force
        _case("measure_10x10_trans", "measure", 10, True, 4, 256, 4),
        # spin correlations of the same state over all pairs of sites
        _case("correlation_10x10", "correlation", 10, True, 4, 148, 4),
        # SR step with the split-BF16 S and the full f_ij matrix (10404 parameters), early in a run: s_factor0 is
        # lowered by s_factor_scale from step to step
        _case("sr_split_10x10", "sr", 10, False, 4, 1024, 16, split=True, s_factor0=1e-2),
        # SR step, all FP64
        _case("sr_fp64_8x8", "sr", 8, False, 2, 512, 16),
        # the transverse projection's sampling and measurement
        _case("transverse_6x6", "transverse", 6, True, 1, 64, 4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case.  The upper ends keep a pass below the largest listed ones."""
    kind = rng.choice(["eval", "eval_device", "iteration", "sample", "sample", "batch", "measure", "measure",
                       "correlation", "sr", "transverse"])
    J2 = round(rng.uniform(0.4, 0.6), 3)
    if kind == "eval":
        return _drop(_case("", kind, rng.choice([4, 6]), rng.random() < 0.5, rng.randint(1, 2), 1,
                           _log_int(rng, 3, 200), alphac=rng.randint(0, 2),
                           orbital=rng.choice(["full", "sublattice2"]), J2=J2))
    if kind == "eval_device":
        L = rng.choice([6, 8, 10])
        return _drop(_case("", kind, L, L < 10 and rng.random() < 0.7, rng.randint(1, 4), 1, _log_int(rng, 50, 600),
                           orbital=rng.choice(["full", "full", "sublattice2"]), J2=J2))
    if kind == "iteration":
        return _drop(_case("", kind, 4, rng.random() < 0.5, rng.randint(1, 2), rng.randint(6, 16),
                           rng.randint(100, 140), split=rng.random() < 0.5, J2=J2))
    if kind == "sample":
        if rng.random() < 0.5:
            L = rng.choice([4, 6, 8])
            return _drop(_case("", kind, L, True, rng.randint(1, 4), _log_int(rng, 20, 300), rng.randint(1, 9), J2=J2))
        L = rng.choice([6, 8, 10, 12])
        return _drop(_case("", kind, L, False, rng.randint(1, 4), _log_int(rng, 20, 400), rng.randint(1, 5), J2=J2))
    if kind == "batch":
        return _drop(_case("", kind, 12, False, rng.randint(1, 2), _log_int(rng, 8, 75), rng.randint(1, 2), L2=14, J2=J2))
    if kind == "measure":
        L = rng.choice([4, 6, 8, 10, 12])
        return _drop(_case("", kind, L, L < 12 and rng.random() < 0.7, rng.randint(1, 4), _log_int(rng, 10, 220),
                           rng.randint(1, 4), orbital=rng.choice(["full", "full", "sublattice2"]), J2=J2))
    if kind == "correlation":
        L = rng.choice([4, 6, 8, 10, 12])
        return _drop(_case("", kind, L, L < 12 and rng.random() < 0.7, rng.randint(1, 4), _log_int(rng, 10, 148),
                           rng.randint(1, 3), J2=J2))
    if kind == "sr":
        L = rng.choice([6, 8])
        return _drop(_case("", kind, L, False, rng.randint(1, 4), rng.randint(400, 600), rng.randint(8, 16),
                           split=rng.random() < 0.5, J2=J2))
    return _drop(_case("", kind, rng.choice([4, 6]), rng.random() < 0.5, rng.randint(1, 2), _log_int(rng, 8, 64),
                       rng.randint(1, 4), J2=J2))


def _drop(c):
    del c["name"]
    return c


def _problem(case, seed, L=None):
    L = L or case["L"]
    p = fm.synthetic_problem(L, translations=case["trans"], alphar=case["alpha"], orbital=case["orbital"],
                             nsample=case["walkers"] * case["ns"], seed=seed, J2=case["J2"], s_factor0=case["s_factor0"])
    if case["alphac"]:
        p.inp.alphac = case["alphac"]
        rng = np.random.default_rng(seed + 77)
        shape = (L * L, case["alphac"])
        p.Wc = rng.normal(0.0, 0.05, shape) + 1j * rng.normal(0.0, 0.05, shape)
        p.bc = rng.normal(0.0, 0.05, case["alphac"]) + 1j * rng.normal(0.0, 0.05, case["alphac"])
    return p


def _uniform(L, n, seed):
    """n configurations with N/2 up spins, drawn uniformly."""
    rng = np.random.default_rng(seed)
    N = L * L
    x = -np.ones((n, N), dtype=np.int32)
    up = np.argsort(rng.random((n, N)), axis=1)[:, :N // 2]
    np.put_along_axis(x, up, 1, axis=1)
    return x


def _weighted(p, n, seed):
    """n configurations near the distribution |psi|^2 that sampling gives: each the last state of a short chain of
    independent proposals."""
    m = _Model(p)
    rng = np.random.default_rng(seed + 3)
    cand = [_uniform(p.inp.L, n, 1000 * seed + k) for k in range(12)]
    w = [m.psi(torch.from_numpy(c).cuda())[0].sum(1).abs().cpu().numpy() ** 2 for c in cand]
    x, cur = cand[0], w[0]
    for c, v in zip(cand[1:], w[1:]):
        take = rng.random(n) * cur < v
        x = np.where(take[:, None], c, x)
        cur = np.where(take, v, cur)
    return x


def _context(case, seed, L=None):
    p = _problem(case, seed, L)
    w = fm.spin_projection_weights(1, transverse=True) if case["kind"] == "transverse" else None
    g = capi.Context(p, n_walkers=case["walkers"], nsample_per_walker=case["ns"], sp_weights=w)
    g.set_params(p.br, p.Wr, p.slater, 0.0, bc=p.bc, Wc=p.Wc)
    return p, g


def prepare(case, seed):
    p, g = _context(case, seed)
    s = dict(case=case, p=p, g=g, first=True)
    kind, n, L = case["kind"], case["walkers"] * case["ns"], case["L"]
    if kind in ("sample", "transverse", "iteration"):
        g.seed(seed)
    elif kind == "batch":
        q, h = _context(case, seed + 1, case["L2"])
        g.seed(seed)
        h.seed(seed + 1)
        s.update(g2=h, batch=capi.Batch([g, h]))
    elif kind in ("measure", "correlation"):
        g.seed(seed)
        g.set_samples(_uniform(L, n, seed))
    elif kind == "sr":
        g.seed(seed)
        g.set_samples(_weighted(p, n, seed))
    elif kind == "eval":
        s["x"] = _uniform(L, n, seed)
    elif kind == "eval_device":
        d = torch.device("cuda")
        s["x"] = torch.from_numpy(_uniform(L, n, seed)).to(d)
        s["psi"] = torch.zeros((n, g.n_qp + 1), dtype=torch.complex128, device=d)
        s["hpsi"] = torch.zeros(n, dtype=torch.complex128, device=d)
        s["O"] = torch.zeros((n, g.Nv), dtype=torch.float64, device=d)
        torch.cuda.synchronize()
    return s


def _params(g):
    br, Wr, sl, _ = g.get_params()
    return dict(br=br, Wr=Wr, slater=sl)


def run(s):
    case, g, p = s["case"], s["g"], s["p"]
    kind = case["kind"]
    if kind == "sample":
        na = g.make_sample(s["first"])
        s["first"] = False
        x, psi, pf = g.samples()
        return dict(naccept=na, x=x, psi=psi, pf=pf)
    if kind == "batch":
        na = s["batch"].make_sample(s["first"])
        s["first"] = False
        return dict(naccept=na, a=list(g.samples()), b=list(s["g2"].samples()))
    if kind == "measure":
        return g.measure(want_S=False)
    if kind == "correlation":
        return g.measure_correlation()
    if kind == "eval":
        return g.eval_configs(s["x"], want_h=True, want_O=True)
    if kind == "eval_device":
        g.eval_configs_noalloc(s["x"].shape[0], s["x"].data_ptr(), s["psi"].data_ptr(), s["hpsi"].data_ptr(),
                               s["O"].data_ptr())
        return dict(psi=s["psi"], hpsi=s["hpsi"], O=s["O"])
    if kind == "sr":
        g.set_params(p.br, p.Wr, p.slater, 0.0)
        g.measure(want_S=False)
        out, dx = g.sr_step(1, p.inp.delta_tau, p.inp.s_factor0, p.inp.s_cut,
                            precision=capi.SR_SPLIT_BF16 if case["split"] else capi.SR_FP64)
        return dict(Etot=out.Etot, lam=out.lambda_, dx=dx, **_params(g))
    if kind == "iteration":
        out = g.iteration(capi.SR_SPLIT_BF16 if case["split"] else capi.SR_FP64, p.inp.delta_tau,
                          p.inp.s_factor_scale, p.inp.s_cut, p.inp.s_factor0)
        return dict(Etot=out.Etot, norm=out.norm, lam=out.lambda_, **_params(g))
    na = g.make_sample(s["first"])
    s["first"] = False
    m = g.measure(want_S=False)
    return dict(naccept=na, x=g.samples()[0], **m)


# ---- work --------------------------------------------------------------------------------------------------

def _sampling(L, n_qp, walkers, ns, alpha):
    """(bytes, flops) of make_sample: max(30, ns/100) + ns + 1 sweeps of N proposals per walker.  A proposal needs
    u^T Y of every projection's inverse block (and theta'), an accepted one (about a third) Y v and the rank-2
    update.  A walker whose blocks fit an SM's shared memory need not read them again for each proposal."""
    N = L * L
    Np = N // 2
    props = walkers * (max(30, ns // 100) + ns + 1.0) * N
    flops = props * n_qp * (2.0 * Np * Np * (1 + 3.0 / 3) + 8.0 * Np + 20.0 * alpha)
    block = 8.0 * Np * Np * n_qp
    stored = walkers * ns * (N + 24.0 * n_qp)
    moved = props * block * (1 + 2.0 / 3) if block > 200e3 else walkers * block
    return moved + stored, flops


def _evaluation(L, n_qp, n, alpha, Nv, pairs, with_o=True):
    """(bytes, flops) of psi, H psi and O_k of n configurations: per projection the inverse (2 Np^3), Y v of every up
    electron (2 Np^3), two dot products for each exchanged pair and the scatter of Y."""
    N = L * L
    Np = N // 2
    flops = n * n_qp * (4.0 * Np ** 3 + pairs * (4.0 * Np + 10.0 * alpha) + (2.0 * Np * Np if with_o else 0.0))
    return n * (N + 16.0 * n_qp + (8.0 * Nv if with_o else 0.0)) + 8.0 * n_qp * N * N, flops


def work(case):
    L, N, al = case["L"], case["L"] ** 2, case["alpha"]
    n_qp = 2 * (N if case["trans"] else 1)
    n = case["walkers"] * case["ns"]
    Np = N // 2
    nsl = N * N if case["orbital"] == "full" else 2 * N
    Nv = 2 * case["alphac"] * (N + 1) + al * (N + 1) + nsl
    kind = case["kind"]
    bonds = 2.05 * N  # antiparallel ones among 4 N
    if kind == "sample":
        b, f = _sampling(L, n_qp, case["walkers"], case["ns"], al)
    elif kind == "batch":
        b, f = _sampling(L, n_qp, case["walkers"], case["ns"], al)
        b2, f2 = _sampling(case["L2"], n_qp, case["walkers"], case["ns"], al)
        b, f = b + b2, f + f2
    elif kind in ("eval", "eval_device"):
        b, f = _evaluation(L, n_qp, n, al, Nv * (2 if case["alphac"] else 1), bonds)
    elif kind == "measure":
        b, f = _evaluation(L, n_qp, n, al, Nv, bonds)
        f += 4.0 * n * Nv
    elif kind == "correlation":
        b, f = _evaluation(L, n_qp, n, al, 0, Np * Np, with_o=False)
        b += 8.0 * N * (N + 1) * 3
    elif kind in ("sr", "iteration"):
        b, f = _evaluation(L, n_qp, n, al, Nv, bonds)
        f += 4.0 * n * Nv + (3.0 if case["split"] else 1.0) * n * Nv * Nv + Nv ** 3 / 3.0
        b += 8.0 * Nv * Nv
        if kind == "iteration":
            b2, f2 = _sampling(L, n_qp, case["walkers"], case["ns"], al)
            b, f = b + b2, f + f2
    else:  # transverse: the N x N skew matrices in place of the blocks
        props = case["walkers"] * (max(30, case["ns"] // 100) + case["ns"] + 1.0) * N
        block = 8.0 * N * N * n_qp
        b = props * block * (1 + 2.0 / 3) if block > 200e3 else case["walkers"] * block
        f = props * n_qp * (4.0 * N * N + 16.0 * N * N / 3) + n * n_qp * (2.0 * N ** 3 + bonds * 4.0 * N * N)
    return {"bytes": b, "flops": f}


# ---- values in 64 bits, plain torch --------------------------------------------------------------------------

class _Model:
    """psi, exchanged amplitudes and O_k of a Problem by dense linear algebra."""

    def __init__(self, p):
        d = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.p, self.d, L = p, d, p.inp.L
        N = self.N = L * L
        self.Np, self.n_mp = N // 2, p.sym.n_mp
        self.wmap = torch.from_numpy(p.sym.W_map.T.astype(np.int64) - 1).to(d)  # [mp][i]
        self.winv = torch.argsort(self.wmap, dim=1)
        self.orb = torch.from_numpy(p.orbital_idx.astype(np.int64) - 1).to(d)
        self.f = torch.from_numpy(p.slater).to(d)[self.orb]
        site = torch.arange(N, device=d)
        self.sb = 1.0 - 2.0 * ((site // L + site % L) % 2).double()
        self.Wr, self.br = torch.from_numpy(p.Wr).to(d), torch.from_numpy(p.br).to(d)
        self.ac = p.inp.alphac
        if self.ac:
            self.Wc, self.bc = torch.from_numpy(p.Wc).to(d), torch.from_numpy(p.bc).to(d)
        ss = math.sin(math.pi / 2) ** 2
        cc = math.cos(math.pi / 2) ** 2
        self.cs = [(1.0, 0.0), (cc, ss)]
        self.par = [1.0, 1.0 if p.inp.spin_parity == 1 else -1.0]
        self.pfsign = -1.0 if (self.Np * (self.Np - 1) // 2) % 2 else 1.0

    def electrons(self, x):
        n = x.shape[0]
        return ((x == 1).nonzero()[:, 1].reshape(n, self.Np), (x == -1).nonzero()[:, 1].reshape(n, self.Np))

    def projections(self, x, up, dn):
        """For each projection: its weight without the Pfaffian, X, the slater table and the angles."""
        xd = x.double()
        for mp in range(self.n_mp):
            wm = self.wmap[mp]
            tb = wm[torch.cat([up, dn], 1)]
            inv = torch.zeros(x.shape[0], dtype=torch.int64, device=self.d)
            for r in range(1, self.N):
                inv += (tb[:, :r] > tb[:, r:r + 1]).sum(1)
            inv += (self.sb[wm[dn]] < 0).sum(1)
            sgn = 1.0 - 2.0 * (inv % 2).double()
            ft = self.f[wm][:, wm]  # f(T p, T q)
            t0 = xd @ self.Wr[wm]
            tc = xd.to(torch.complex128) @ self.Wc[wm] if self.ac else None
            for sp in (0, 1):
                cc, ss = self.cs[sp]
                s = 1.0 - 2.0 * sp
                XF = ft * cc + ft.T * ss
                th = self.br + s * t0
                thc = self.bc + s * tc if self.ac else None
                wt = sgn * self.par[sp]
                yield mp, sp, XF, XF[up[:, :, None], dn[:, None, :]], th, thc, wt

    def rbm(self, th, thc):
        r = torch.cosh(th).prod(-1)
        return r * (0.5 * torch.cosh(thc)).prod(-1) if self.ac else r

    def psi(self, x):
        """psi of every projection [n][qp], without and (second value) with nothing else."""
        up, dn = self.electrons(x)
        out = [self.rbm(th, thc) * wt * self.pfsign * torch.linalg.det(X)
               for _, _, _, X, th, thc, wt in self.projections(x, up, dn)]
        return torch.stack(out, 1), up, dn

    def everything(self, x, with_o=True, chunk=256):
        parts = [self._chunk(x[k:k + chunk], with_o) for k in range(0, x.shape[0], chunk)]
        return [torch.cat(v) if v[0] is not None else None for v in zip(*parts)]

    def _chunk(self, x, with_o):
        """psi [n][qp], psi of every exchanged pair [n][up][down], O_k [n][Nv]."""
        n, Np, N, p = x.shape[0], self.Np, self.N, self.p
        ct = torch.complex128 if self.ac else torch.float64
        up, dn = self.electrons(x)
        xd = x.double()
        ar, ac = self.br.shape[0], self.ac
        psi, pairs = [], torch.zeros((n, Np, Np), dtype=ct, device=self.d)
        O = torch.zeros((n, p.Nv), dtype=ct, device=self.d) if with_o else None
        orr, opp = 2 * ac * (N + 1), 2 * ac * (N + 1) + ar * (N + 1)
        for mp, sp, XF, X, th, thc, wt in self.projections(x, up, dn):
            wm, s = self.wmap[mp], 1.0 - 2.0 * sp
            Y = torch.linalg.inv(X)  # [down][up]
            pf = self.pfsign * torch.linalg.det(X)
            c0 = self.rbm(th, thc) * wt
            q = c0 * pf
            psi.append(q)
            U, V = XF[dn[:, :, None], dn[:, None, :]], XF[up[:, :, None], up[:, None, :]]  # U[b][j], V[i][a]
            c = XF[dn[:, :, None], up[:, None, :]]  # [b][a]
            du = c - torch.diagonal(U, dim1=1, dim2=2)[:, :, None]
            dv = c - torch.diagonal(V, dim1=1, dim2=2)[:, None, :]
            P, Q = U @ Y, Y @ V
            Z = U @ Q
            R = ((P + du * Y) * (Q + dv * Y) - Y * (Z + du * Q + dv * P + du * dv * Y - c)).transpose(1, 2)
            ws = self.Wr[wm]
            t2 = th[:, None, None, :] - 2.0 * s * ws[up][:, :, None, :] + 2.0 * s * ws[dn][:, None, :, :]
            k2 = None
            if ac:
                wc = self.Wc[wm]
                k2 = thc[:, None, None, :] - 2.0 * s * wc[up][:, :, None, :] + 2.0 * s * wc[dn][:, None, :, :]
            sg = -self.sb[up][:, :, None] * self.sb[dn][:, None, :]
            pairs += self.rbm(t2, k2) * sg * (wt * pf)[:, None, None] * R
            if not with_o:
                continue
            xi = xd[:, self.winv[mp]]
            for f in range(ac):
                v = torch.tanh(thc[:, f]) * q
                vi = s * v[:, None] * xi
                for im in (0, 1):
                    O[:, 2 * f + im] += v * 1j ** im
                    k = 2 * ac + 2 * N * f + im
                    O[:, k:k + 2 * N:2] += vi * 1j ** im
            for f in range(ar):
                v = torch.tanh(th[:, f]) * q
                O[:, orr + f] += v
                k = orr + ar + N * f
                O[:, k:k + N] += s * v[:, None] * xi
            tu, td = wm[up][:, :, None], wm[dn][:, None, :]
            g = Y.transpose(1, 2) * q[:, None, None]
            for w, at in zip(self.cs[sp], (self.orb[tu, td], self.orb[td.expand(n, Np, Np), tu.expand(n, Np, Np)])):
                if w:
                    O.scatter_add_(1, opp + at.expand(n, Np, Np).reshape(n, -1), (w * g).reshape(n, -1))
        return torch.stack(psi, 1), pairs, O

    def bonds(self):
        L, i = self.p.inp.L, torch.arange(self.N, device=self.d)
        ix, iy = i // L, i % L
        J1, J2 = self.p.inp.J1, self.p.inp.J2
        for dx, dy, J, sg in ((1, 0, J1, -1.0), (0, 1, J1, -1.0), (1, 1, J2, 1.0), (1, -1, J2, 1.0)):
            yield i, ((ix + dx) % L) * L + (iy + dy) % L, J, sg

    def by_site(self, x, pairs):
        """psi of the exchange of sites [n][i1][i2], 0 for parallel spins."""
        n, N = x.shape
        up, dn = self.electrons(x)
        m = torch.zeros((n, N, N), dtype=pairs.dtype, device=self.d)
        k = torch.arange(n, device=self.d)[:, None, None]
        m[k, up[:, :, None], dn[:, None, :]] = pairs
        return m + m.transpose(1, 2)

    def hpsi(self, x, psi0, m):
        xd, h = x.double(), 0.0
        for i1, i2, J, sg in self.bonds():
            h = h + (J * xd[:, i1] * xd[:, i2]).sum(1) * psi0 + 2.0 * J * sg * m[:, i1, i2].sum(1)
        return h


def _measured(m, x):
    """Sums of calc_phys_quantity_opt (shift 0) and the reweighted derivatives."""
    psi, pairs, O = m.everything(x)
    psi0 = psi.sum(1)
    w = 1.0 / psi0.abs()
    e = m.hpsi(x, psi0, m.by_site(x, pairs)) * w
    Ow = O * w[:, None]
    scal = dict(Etot=float((w * psi0 * e).sum()), Etot2=float((e * e).sum()), norm=float(x.shape[0]),
                wf_av=float(psi0.abs().sum()))
    return scal, 2.0 * e @ Ow, (w * psi0) @ Ow, Ow


def _sr(p, m, x):
    """SR_pdposv.f90:1-432 on the samples x: direction, step norm and new parameters."""
    sc, g, ov, O = _measured(m, x)
    N, n, nv, nr = m.N, sc["norm"], p.Nv, p.Nv - p.n_slater
    E, g, ov = sc["Etot"] / n, g / n, ov / n
    g = g - 2.0 * E * ov
    S = O.T @ O / n - torch.outer(ov, ov)
    dg = torch.diagonal(S).clone()
    same = torch.diagonal(m.orb) + nr
    live = torch.ones(nv, dtype=torch.bool, device=m.d)
    live[same] = False
    scal = math.sqrt(float(dg[:nr].mean()) / float(dg[nr:][live[nr:]].mean()))
    v = torch.ones(nv, dtype=torch.float64, device=m.d)
    v[nr:] = scal
    S, g = S * v[:, None] * v[None, :], g * v
    S.diagonal().add_(float(torch.diagonal(S)[live].mean()) * max(1e-4, p.inp.s_factor0))
    x0 = torch.cholesky_solve(g[:, None], torch.linalg.cholesky(S))[:, 0]
    lam = math.sqrt(float(x0 @ (S @ x0))) * 5.0 / p.inp.L
    dx = (x0 / lam if lam > 1.0 else x0) * v
    step = p.inp.delta_tau * dx
    big = float(step.abs().max())
    gam = torch.cat([m.br, m.Wr.T.reshape(-1), torch.from_numpy(p.slater).to(m.d)])
    gam = gam - step * (0.04 / big if big > 0.04 else 1.0)
    gam[nr:] *= 0.25 / float(gam[nr:].abs().mean())
    ar = m.br.shape[0]
    c = gam.cpu().numpy()
    return dict(Etot=E, lam=lam, dx=dx.cpu().numpy(), br=c[:ar], Wr=c[ar:nr].reshape(ar, N).T.copy(), slater=c[nr:])


def exact(case, seed):
    kind, n, L = case["kind"], case["walkers"] * case["ns"], case["L"]
    if kind not in ("eval", "eval_device", "measure", "correlation", "sr"):
        return None  # Markov chains: configurations, and amplitudes carried along them by updates
    p = _problem(case, seed)
    m = _Model(p)
    if kind == "sr":
        return _sr(p, m, torch.from_numpy(_weighted(p, n, seed)).to(m.d))
    x = torch.from_numpy(_uniform(L, n, seed)).to(m.d)
    if kind in ("eval", "eval_device"):
        psi, pairs, O = m.everything(x)
        psi0 = psi.sum(1)
        h = m.hpsi(x, psi0, m.by_site(x, pairs))
        return dict(psi=torch.cat([psi0[:, None], psi], 1).to(torch.complex128), hpsi=h.to(torch.complex128), O=O)
    if kind == "measure":
        sc, g, ov, _ = _measured(m, x)
        return dict(sc, gvec=g, Ovec=ov)
    psi, pairs, _ = m.everything(x, with_o=False)
    psi0 = psi.sum(1)
    w, by = 1.0 / psi0.abs(), m.by_site(x, pairs)
    e = m.hpsi(x, psi0, by) * w
    N, xd = m.N, x.double()
    i2, i1 = torch.tril_indices(N, N, device=m.d)  # i1 <= i2, i2 slowest
    ws = w * w * psi0
    zz = torch.einsum("n,ni,nj->ij", ws * psi0, xd, xd)
    ex = torch.einsum("n,nij->ij", ws, by * m.sb[:, None] * m.sb[None, :])
    ex = ex + torch.eye(N, dtype=torch.float64, device=m.d) * (ws * psi0).sum()
    vbs = []
    for a, b, _, sg in m.bonds():
        sd = w[:, None] * (xd[:, a] * xd[:, b] * psi0[:, None] + 2.0 * sg * by[:, a, b])
        vbs.append((sd.T @ sd)[i1, i2])
    return dict(Etot=float((w * psi0 * e).sum()), Etot2=float((e * e).sum()), norm=float(n),
                wf_av=float(psi0.abs().sum()), wf_sgn=float((psi0 * w).sum()),
                chi_sp=torch.stack([zz[i1, i2], ex[i1, i2]]), chi_vbs=torch.stack(vbs, 1))
