"""What this framework is used for, as cases whose speed can be measured.

A user's program holds a grid, a potential and the basis of one or more partial
waves, gives them to a :class:`Propagator`, starts it from a wave packet and
then, block after block, propagates some Chebyshev iterations and reads P(E),
the norm trace and the state (the continuation file of every block).  The
bound-state program instead calls H psi on host vectors once a Lanczos step.
``prepare`` builds the first part, ``run`` is one block or one H psi.

The surface, masses, boxes, cut-offs and absorbers are the synthetic LEPS
workload's (``madwave3_gb300/host/generator.py``); the tables are made in
memory instead of through the ``pot/`` and ``func/`` files.  The packet fills
the entrance valley, the interaction region and the product valley, as a
packet does in the middle of a run, so that the flux and the projections have
something to accumulate; the iteration count stands at a block's end, as after
a restart from continuation files.  Mixed precision carries FP32 accuracy, so
such a program keeps the state it reads back in FP32.
"""
import math

import numpy as np
import torch

from madwave3_gb300 import Propagator
from madwave3_gb300.host import constants as C
from madwave3_gb300.host import generator, setup


def _case(name, op, precision, n1, n2, na, iters=0, ne=1, J=0, om=0, waves=1, photo=False):
    """op "hphi": one H psi on host vectors; "run": a block of `iters` iterations.
    `waves` partial waves J, J + 1, ... with Omega = 0..min(J, om) each."""
    c = dict(op=op, precision=precision, n1=n1, n2=n2, na=na, iters=iters, ne=ne, J=J, om=om, waves=waves,
             photo=photo)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the parity tests' grid, four coupled Omega blocks: the smallest call, all latency
        _case("hphi_fp64_40x24x10_j3", "hphi", "fp64", 24, 40, 10, J=3, om=3),
        # a Lanczos step of the bound-state program on the shipped example's grid
        _case("hphi_fp64_256x256x140", "hphi", "fp64", 256, 256, 140),
        # plain FP64, J = 0, one state, one Omega block
        _case("fp64_256x128x60_j0", "run", "fp64", 128, 256, 60, iters=20),
        # plain FP64 with eleven Coriolis-coupled Omega blocks
        _case("fp64_256x128x60_j10", "run", "fp64", 128, 256, 60, iters=4, J=10, om=10),
        # plain FP64, J = 0, the larger grid
        _case("fp64_512x256x120_j0", "run", "fp64", 256, 512, 120, iters=4),
        # plain FP64, three diabatic states, Omega = 0..2, photodissociation (autocorrelation kept)
        _case("fp64_384x192x80_e3", "run", "fp64", 192, 384, 80, iters=2, ne=3, J=2, om=2, photo=True),
        # a small two-state case, mixed: launches and latency
        _case("mixed_36x20x8_e2", "run", "mixed", 20, 36, 8, iters=96, ne=2, J=1, om=1),
        # mixed, J = 0 alone
        _case("mixed_256x128x60_j0", "run", "mixed", 128, 256, 60, iters=32),
        # mixed, eleven coupled blocks
        _case("mixed_256x128x60_j10", "run", "mixed", 128, 256, 60, iters=32, J=10, om=10),
        # mixed, a sweep of partial waves J = 0..12 with Omega <= 6 batched in one context: 70 blocks
        _case("mixed_256x128x60_j0-12", "run", "mixed", 128, 256, 60, iters=32, om=6, waves=13),
        # mixed, the larger J = 0 grid
        _case("mixed_512x256x120_j0", "run", "mixed", 256, 512, 120, iters=20),
        # mixed, three diabatic states, photodissociation
        _case("mixed_384x192x80_e3", "run", "mixed", 192, 384, 80, iters=10, ne=3, J=2, om=2, photo=True),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    while True:
        n2 = logint(32, 512)
        n1 = logint(20, min(256, n2))
        na = logint(8, 140)
        ne = rng.choice((1, 1, 1, 2, 3))
        J = rng.choice((0, 0, 1, 2, 3, 5, 8, 12))
        om = rng.randint(0, min(J, 6))
        waves = rng.choice((1, 1, 1, 3, 6)) if ne == 1 else 1
        precision = rng.choice(("fp64", "mixed"))
        blocks = sum(min(J + k, om) + 1 for k in range(waves)) * ne
        rect = blocks * n1 * n2 * na
        if rect > 2.5e7:
            continue
        if rng.random() < 0.25:
            return _case("", "hphi", precision, n1, n2, na, ne=ne, J=J, om=om)
        most = (3e7 if precision == "fp64" else 3e8) / rect
        return _case("", "run", precision, n1, n2, na, iters=max(1, min(32, int(most * rng.uniform(0.3, 1.0)))), ne=ne,
                     J=J, om=om, waves=waves, photo=ne > 1 and rng.random() < 0.5)


# ---------------------------------------------------------------------------
# the host's tables
# ---------------------------------------------------------------------------
def _params(case):
    coarse = case["n2"] < 128
    return dict(npun1=case["n1"], npun2=case["n2"], nangu=case["na"], nelecmax=case["ne"], npun1min=min(32, case["n1"]) if not coarse else 8,
                jmax=min(20, case["na"] - 2), nvmax=5 if not coarse else 2, netot=1000 if not coarse else 64,
                alpha0_bohr=0.3 if not coarse else 1.2, iphoto=1 if case["photo"] else 0,
                shifts_ev=(0.0, 0.8, 1.5) if case["ne"] != 2 else (0.0, 0.3), Jtot=0)


_grids = {}


def _grid(case):
    """The set-up that does not depend on J: grid, potential, diatomic functions."""
    key = tuple(case[k] for k in ("n1", "n2", "na", "ne", "photo"))
    if key in _grids:
        return _grids[key]
    _grids.clear()
    groups, p = generator.make_inputs(**_params(case))
    run = setup.Run(inp=setup.Inputs.from_namelists(groups))
    i, ne, na = run.inp, case["ne"], case["na"]
    setup.input_grid(run)
    setup.pot0(run)
    r1 = i.rmis1 + run.ah1 * np.arange(i.npun1)
    r2 = i.rmis2 + run.ah2 * np.arange(i.npun2)
    # diatomic functions and the reference level
    nj, nv = i.jmax + 1, i.nvmax + 1
    run.nobc = np.full((ne, nj), i.nvmax, np.int32)
    run.ediat = np.zeros((ne, nj, nv))
    run.fd = np.zeros((ne, nj, nv, i.npun1))
    far = np.full_like(r1, 100.0)
    vd = generator.diabatic_matrix(r1, far, far, p) * C.eV2cm * C.conve1
    for e in range(ne):
        for j in range(nj):
            en, v = generator.sine_dvr_states(r1, vd[e, e] + j * (j + 1) * C.hbr ** 2 / (2.0 * run.xm1red * r1 * r1),
                                              run.xm1red, nv)
            run.ediat[e, j], run.fd[e, j] = en, v.T
    run.ediatref = float(run.ediat[0, 0, 0])
    run.ediat -= run.ediatref
    # potential: a point is stored where some diabatic (and so some adiabatic) energy lies below Vcut
    RR, rr = np.meshgrid(r2, r1, indexing="ij")
    vmin, vmax, pts = 1e30, run.vcutmax, []
    for a in range(na):
        x = generator.jacobi_distances(rr, RR, run.cgamma[a], i.xm0, i.xm1)
        V = generator.diabatic_matrix(*x, p) * C.eV2cm * C.conve1
        hi = np.stack([V[e, e] - run.ediatref > run.vcutmax for e in range(ne)])
        i2, i1 = np.nonzero(~hi.all(axis=0))
        v, h = V[:, :, i2, i1], hi[:, i2, i1]
        off = np.zeros(len(i1))
        for e in range(ne):
            v[e, e] -= run.ediatref
            for f in range(ne):
                if e != f:
                    v[e, f] = np.where(h[e] | h[f], 0.0, v[e, f])
                    off = np.maximum(off, np.abs(v[e, f]))
            v[e, e] = np.where(h[e], run.vcutmax, v[e, e])
            vmin, vmax = min(vmin, float((v[e, e] - off).min())), max(vmax, float((v[e, e] + off).max()))
        pts.append((i1 + 1, i2 + 1, v))
    run.nelec = ne
    run.iomdiat, run.iomatom = np.zeros(ne, np.int32), np.zeros(ne, np.int32)
    run.sigdiat, run.sigatom = np.ones(ne), np.ones(ne)
    run.npunreal = np.array([len(q[0]) for q in pts], np.int32)
    run.npuntot = int(run.npunreal.max())
    run.indr1, run.indr2 = np.zeros((na, run.npuntot), np.int32), np.zeros((na, run.npuntot), np.int32)
    run.vvv = np.zeros((ne, ne, na, run.npuntot))
    for a, (i1, i2, v) in enumerate(pts):
        n = len(i1)
        run.indr1[a, :n], run.indr2[a, :n] = i1, i2
        run.vvv[:, :, a, :n] = v.transpose(1, 0, 2)
    run.vmintot, run.vmaxtot = vmin, vmax
    run.delta2 = 0.5 * (vmax + run.radcutmax + 3.0 * run.rotcutmax - vmin)
    run.emindlt = vmin + run.delta2
    _grids[key] = run
    return run


def _waves(case, seed):
    """The partial waves of a case with their packets."""
    import copy
    base, rng, runs = _grid(case), np.random.default_rng([seed, 17]), []
    ecol, rcol = rng.uniform(0.4, 0.7), rng.uniform(8.5, 9.5)
    n, span1, span2 = 4, base.inp.rfin1 - base.inp.rmis1, base.inp.rfin2 - base.inp.rmis2
    # pieces of the packet: entrance valley, interaction region, product valley (two)
    at = np.array([(0.78, 3.5), (1.2, 1.6), (3.4, 1.9), (4.8, 2.6)]) + rng.uniform(-0.1, 0.1, (n, 2))
    wid = np.maximum(np.array([(0.35, 1.2), (0.5, 0.6), (0.9, 0.9), (0.9, 0.9)]),
                     [3 * span1 / (case["n1"] - 1), 3 * span2 / (case["n2"] - 1)])
    mom, ph = rng.uniform(-0.5, 0.5, (n, 2)) / wid * 4, rng.uniform(0, 2 * math.pi, n)
    r1 = base.inp.rmis1 + base.ah1 * np.arange(case["n1"])
    r2 = base.inp.rmis2 + base.ah2 * np.arange(case["n2"])
    d1, d2 = r1[None] - at[:, :1], r2[None] - at[:, 1:]
    G = (np.exp(-(d1 / wid[:, :1]) ** 2)[:, :, None] * np.exp(-(d2 / wid[:, 1:]) ** 2)[:, None, :]
         * np.cos(d1[:, :, None] * mom[:, :1, None] + d2[:, None, :] * mom[:, 1:, None] + ph[:, None, None]))
    for k in range(case["waves"]):
        r = copy.copy(base)
        inp = r.inp = copy.copy(base.inp)
        inp.Jtot = case["J"] + k
        inp.iparity, inp.iommax = (-1) ** inp.Jtot, min(inp.Jtot, case["om"])
        inp.ecol_ev, inp.rcolini_ang = ecol, rcol * C.convl
        setup.basis(r)
        setup.angular_functions(r)
        r.offs = np.zeros((inp.nangu, r.ncan), np.int64)
        cnt = 0
        for a in r.angle_order():
            for b in range(r.ncan):
                r.offs[a - 1, b] = cnt
                cnt += int(r.npunreal[a - 1])
        r.ntot = cnt
        if not case["photo"]:
            setup.set_colini(r)          # the collision energy's parameters; the packet is replaced below
        else:
            r.psi0 = np.zeros(cnt)
        ang = np.zeros((n, r.ncan, inp.nangu))
        for b in range(r.ncan):
            js = [j for j in r.jbas[b, : r.nojbas[b]] if j <= r.iombas[b] + 6]
            ang[:, b] = rng.normal(size=(n, len(js))) @ r.djmmp[r.iombas[b], r.nelebas[b] - 1, js]
        for a in range(inp.nangu):
            m = int(r.npunreal[a])
            g = G[:, r.indr1[a, :m] - 1, r.indr2[a, :m] - 1]
            o = int(r.offs[a, 0])
            r.psi0[o:o + m * r.ncan] = (ang[:, :, a].T @ g).reshape(-1)
        r.psi0 /= np.linalg.norm(r.psi0)
        r.efe_zot = np.zeros(0)
        runs.append(r)
    return runs


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def prepare(case, seed):
    runs = _waves(case, seed)
    p = Propagator(runs, precision=case["precision"])
    s = dict(p=p, case=case, waves=len(runs))
    if case["op"] == "hphi":
        s["psi"] = np.random.default_rng([seed, 3]).normal(size=runs[0].ntot) * 1e-3 + runs[0].psi0
        p.hphi(s["psi"])               # the Lanczos program's context exists before its steps
        return s
    # a continuation: the state of a run that stands at a block's end
    p.start([r.psi0 for r in runs])
    km1, k, _ = p.state_all()
    p.upload_state_all(km1, k, 512)
    s["psi"] = torch.empty(sum(r.ntot for r in runs), dtype=torch.float64, pin_memory=True)
    if case["precision"] == "mixed":
        s["psi32"] = torch.empty(s["psi"].numel(), dtype=torch.float32)
    p.sync()
    return s


def run(state):
    p, case = state["p"], state["case"]
    if case["op"] == "hphi":
        h = p.hphi(state["psi"])
        return {"hpsi": h if case["precision"] == "fp64" else h.astype(np.float32)}
    p.run(case["iters"])
    low = case["precision"] == "mixed"
    P = np.stack([p.totalflux(w)[0] for w in range(state["waves"])])
    norms = np.stack([p.norms(w)[-case["iters"]:] for w in range(state["waves"])])
    p.state_k_all(state["psi"].numpy())
    psi = state["psi32"].copy_(state["psi"]) if low else state["psi"]
    return {"psi": psi, "P": P.astype(np.float32) if low else P, "norms": norms.astype(np.float32) if low else norms}


def work(case):
    """Bytes: per iteration psi_k and psi_k-1 read and psi_k+1 written in FP64, and the
    potential once per context; H psi: psi in and H psi out over the host link.
    Flops: the radial sine transforms by an FFT, the angular terms through the j basis."""
    base = _grid(case)
    pts, ne = int(base.npunreal.sum()), case["ne"]
    blocks = sum(min(case["J"] + k, case["om"]) + 1 for k in range(case["waves"])) * ne
    n = max(1, case["iters"])
    n1, n2, na = case["n1"], case["n2"], case["na"]
    flops = 2 * n1 * n2 * na * 2.5 * (math.log2(2 * n1) + math.log2(2 * n2)) + 4.0 * na * pts + 16.0 * pts
    return {"bytes": n * (24.0 * pts * blocks + 8.0 * ne * ne * pts) if case["op"] == "run" else 16.0 * pts * blocks,
            "flops": n * blocks * flops}


# ---------------------------------------------------------------------------
# the same in 64 bits with dense matrices
# ---------------------------------------------------------------------------
def _smooth(n, top):
    """The smallest 2-3-5-7-11-smooth length >= n, at most top."""
    for k in range(n, top):
        m = k
        for f in (2, 3, 5, 7, 11):
            while m % f == 0:
                m //= f
        if m == 1:
            return k
    return top


def _sine(n, dev):
    k = torch.arange(1, n + 1, device=dev, dtype=torch.int64)
    return 2.0 * torch.sin(math.pi * ((k[:, None] * k[None]) % (2 * (n + 1))).double() / (n + 1))


class _Exact:
    def __init__(self, r, dev):
        i = r.inp
        self.r, self.dev, self.n1, self.n2, self.na = r, dev, i.npun1, i.npun2, i.nangu
        t = lambda x: torch.as_tensor(np.ascontiguousarray(x), device=dev)  # noqa: E731
        n1, n2, na = self.n1, self.n2, self.na
        kin = lambda n, ah, mu: (math.pi * torch.arange(1, n + 1, device=dev).double() / ((n + 1.0) * ah)) ** 2 * (0.5 * C.hbr ** 2 / mu)  # noqa: E731
        self.S2, self.e2 = _sine(n2, dev), kin(n2, r.ah2, r.xm2red)
        self.nn = []
        for a in range(na):
            i1 = r.indr1[a, : r.npunreal[a]]
            self.nn.append(max(i.npun1min, _smooth(int(i1.max() - i1.min()) + 1, n1)))
        self.S1 = {n: (_sine(n, dev), kin(n, r.ah1, r.xm1red)) for n in set(self.nn)}
        self.D = [t(r.djmmp[r.iombas[b], r.nelebas[b] - 1]) for b in range(r.ncan)]   # [j][angle]
        self.r1 = i.rmis1 + r.ah1 * torch.arange(n1, device=dev).double()
        self.r2 = i.rmis2 + r.ah2 * torch.arange(n2, device=dev).double()
        self.flat, self.cell, V = [], [], []
        for b in range(r.ncan):
            f, c = [], []
            for a in range(na):
                m = int(r.npunreal[a])
                f.append(r.offs[a, b] + np.arange(m))
                c.append((a * n1 + r.indr1[a, :m] - 1).astype(np.int64) * n2 + r.indr2[a, :m] - 1)
            self.flat.append(t(np.concatenate(f)))
            self.cell.append(t(np.concatenate(c)))
        self.V = t(np.concatenate([r.vvv[:, :, a, : r.npunreal[a]] for a in range(na)], axis=2))
        fab = lambda x, x0, al, ni, ex: torch.where(x >= x0, torch.exp(-al * ((x - x0).clamp(min=0) / ni) ** ex), torch.ones_like(x))  # noqa: E731
        fac = (fab(self.r1, i.absr1, i.absalp1, i.ninterv1, i.n1expo)[:, None] * fab(self.r2, i.absr2, i.absalp2, i.ninterv2, i.n2expo)[None]).reshape(-1)
        self.f = torch.empty(r.ntot, device=dev, dtype=torch.float64)
        for b in range(r.ncan):
            self.f[self.flat[b]] = fac[self.cell[b] % (n1 * n2)]

    def l2(self, j):
        """l^2 between the Omegas that a j has, before the division by R^2, and its R floor."""
        i = self.r.inp
        oms = [o for o in range(i.iommin, i.iommax + 1) if o <= j]
        m, fm = np.zeros((len(oms), len(oms))), C.hbr ** 2 * 0.5 / self.r.xm2red
        for x, o in enumerate(oms):
            m[x, x] = fm * (j * (j + 1) + i.Jtot * (i.Jtot + 1) - 2 * o * o)
            if x + 1 < len(oms):
                q = o * (o + 1)
                m[x, x + 1] = m[x + 1, x] = -fm * math.sqrt((i.Jtot * (i.Jtot + 1) - q) * (j * (j + 1) - q)) * (math.sqrt(2.0) if o == 0 else 1.0)
        m[np.abs(m) <= 1e-8] = 0.0
        ev = np.linalg.eigvalsh(m)
        return {o: x for x, o in enumerate(oms)}, m, 0.5 * (ev[0] + ev[-1])

    def h(self, psi):
        r, n1, n2, na, dev = self.r, self.n1, self.n2, self.na, self.dev
        out = torch.zeros_like(psi)
        X = []
        for b in range(r.ncan):
            x = torch.zeros(na * n1 * n2, device=dev, dtype=torch.float64)
            x[self.cell[b]] = psi[self.flat[b]]
            X.append(x.view(na, n1, n2))
        B = [torch.einsum("ja,arR->jrR", self.D[b], X[b]) for b in range(r.ncan)]
        jmax = na - 1
        L = [self.l2(j) for j in range(jmax + 1)] if na > 1 else []
        yj = lambda j: torch.clamp(j * (j + 1) * C.hbr ** 2 * 0.5 / (r.xm1red * self.r1 ** 2), max=r.rotcutmax)  # noqa: E731
        for b in range(r.ncan):
            k = X[b].clone()
            for a in range(na):
                n = self.nn[a]
                S1, e1 = self.S1[n]
                y = S1 @ X[b][a, :n] @ self.S2
                y *= torch.clamp(e1[:, None] + self.e2[None], max=r.radcutmax) / (4.0 * (n + 1) * (n2 + 1))
                k[a, :n] = S1 @ y @ self.S2
            if na > 1:
                hb = torch.zeros_like(B[b])
                om, el = int(r.iombas[b]), int(r.nelebas[b])
                for j in range(jmax + 1):
                    row, m, mean = L[j]
                    if om not in row:
                        continue
                    hb[j] = yj(j)[:, None] * B[b][j]
                    den = torch.where(mean / self.r2 ** 2 > r.rotcutmax, torch.full_like(self.r2, abs(mean) / r.rotcutmax), self.r2 ** 2)
                    for s in range(r.ncan):
                        o = int(r.iombas[s])
                        if int(r.nelebas[s]) == el and o in row and m[row[om], row[o]] != 0.0:
                            hb[j] += (m[row[om], row[o]] / den)[None] * B[s][j]
                k += torch.einsum("ja,jrR->arR", self.D[b], hb)
            v = k.reshape(-1)[self.cell[b]]
            for s in range(r.ncan):
                if r.iombas[s] == r.iombas[b]:
                    v += self.V[r.nelebas[b] - 1, r.nelebas[s] - 1] * psi[self.flat[s]]
            out[self.flat[b]] = v
        return out


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    runs = _waves(case, seed)
    if case["op"] == "hphi":
        psi = np.random.default_rng([seed, 3]).normal(size=runs[0].ntot) * 1e-3 + runs[0].psi0
        return {"hpsi": _Exact(runs[0], dev).h(torch.as_tensor(psi, device=dev)).cpu()}
    outs, norms = [], []
    for r in runs:
        x = _Exact(r, dev)
        old = torch.as_tensor(r.psi0, device=dev)
        new = (x.h(old) - r.emindlt * old) / r.delta2
        nrm = []
        for _ in range(case["iters"]):
            old, new = new, (2.0 * (x.h(new) - r.emindlt * new) / r.delta2 - x.f * old) * x.f
            nrm.append(float((new * new).sum()))
        outs.append(new.cpu())
        norms.append(nrm)
    return {"psi": torch.cat(outs), "P": None, "norms": np.array(norms)}
