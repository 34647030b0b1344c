"""The digit products at the small end: vectors of subnormal numbers, and the components next to
the poles of the angular terms."""
import os

import numpy as np
import pytest

from madwave3_gb300 import Propagator
from oracle.mw3ref import Oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def shape_run(tmp_path_factory):
    from madwave3_gb300.host import generator, setup

    def make(n1, n2, na, extra):
        d = str(tmp_path_factory.mktemp("fxs") / "case")
        generator.write_case(d, **{**dict(npun1=n1, npun2=n2, nangu=na, jmax=min(na - 1, 12) // 2 * 2, nvmax=1, netot=32,
                                          npun1min=8, alpha0_bohr=1.2), **extra})
        return setup.load(os.path.join(d, "input.dat"))
    return make


#                          smallest subnormal, the vector's scale, relative rounding of the path
@pytest.mark.parametrize("precision,n1,n2,na,tiny,scale,rel", [("fp64", 24, 40, 12, -1074, -1030, 1e-12),
                                                               ("fp64", 145, 130, 2, -1074, -1035, 1e-12),
                                                               ("mixed", 150, 150, 3, -149, -124, 1e-6)])
def test_subnormal_vectors(shape_run, precision, n1, n2, na, tiny, scale, rel):
    run = shape_run(n1, n2, na, {})
    p = Propagator(run, precision)
    rng = np.random.default_rng([n1, na])
    # FP32 rectangles take entries from 2^-126 on; what the transforms leave of them is below
    psi = np.ldexp(rng.uniform(0.5, 1, run.ntot) * rng.choice([-1.0, 1.0], run.ntot), scale)
    up = 1000 if precision == "fp64" else 100
    clean = np.ldexp(p.hphi(np.ldexp(psi, up)), -up)
    # every store of an intermediate rounds to the subnormals' spacing: after the last scaling by the kinetic
    # energy the two transforms back multiply it by up to 2 npun1 2 npun2, ahead of it by that energy and
    # 2 npun1 / (4 npun1 npun2) besides; the angular terms by up to 4 nangu^2 and the rotational energy
    e = 1 + 2 * n1 * run.radcutmax + run.rotcutmax
    if precision == "fp64":
        tol = np.ldexp((4 * n1 * n2 + 4 * na * na) * e / 2, tiny)
    else:
        tol = np.ldexp(4 * n1 * n2 * (1 + run.radcutmax) / 2, tiny)
    assert tol < 2.0 ** -6 * np.abs(clean).max()
    assert p.digit_products()["dst"]
    assert np.abs(p.hphi(psi) - clean).max() <= tol + rel * np.abs(clean).max()
    p.close()


@pytest.mark.parametrize("precision,na,om0,om", [("fp64", 40, 9, 12), ("fp64", 130, 15, 16), ("mixed", 70, 13, 15),
                                                 ("mixed", 130, 15, 16)])
def test_angles_next_to_the_poles(shape_run, precision, na, om0, om):
    """Single components of the angular terms where the associated Legendre functions are tiny (1e-8 to 1e-12
    of their largest), for packets of a few j and for a single grid point, at one (r1, R)."""
    run = shape_run(24, 40, na, dict(Jtot=om, iommin=om0, iommax=om, iomref=om0, jref=om0, jmax=om0))
    p, ref = Propagator(run, precision), Oracle(run)
    at = [{(int(x), int(y)): k for k, (x, y) in enumerate(zip(run.indr1[a, :n], run.indr2[a, :n]))}
          for a, n in enumerate(run.npunreal)]
    point = sorted(set.intersection(*(set(m) for m in at)))[0]
    where = np.array([[run.offs[a, b] + at[a][point] for a in range(na)] for b in range(run.ncan)])
    D = [run.djmmp[run.iombas[b], 0] for b in range(run.ncan)]               # [j][angle]
    dmax = [np.abs(d).max(0) for d in D]
    rng = np.random.default_rng([na, om])
    top = run.ncan - 1
    assert run.iombas[top] == om and dmax[top][0] < 1e-7
    packets = []
    for b in (top, 0):
        js = [j for j in range(run.iombas[b], run.iombas[b] + 7) if j < na]
        packets.append((b, None, D[b][js].T @ rng.normal(size=len(js))))
        for a in (0, 1, na // 2):
            packets.append((b, a, np.where(np.arange(na) == a, rng.normal(), 0.0)))
    for b, only, x in packets:
        psi = np.zeros(run.ntot)
        psi[where[b]] = x
        h, e = p.hphi(psi), ref.hphi(psi)
        for t in range(max(0, b - 1), min(run.ncan, b + 2)):
            got, want = h[where[t]], e[where[t]]
            keep = np.arange(na) != (only if t == b else -1)                 # (its own angle has the radial terms)
            # an angle's value is a sum over j of entries of at most dmax: na products, each way
            size = (np.abs(want) / dmax[t])[keep].max()
            tol = 64 * na * (2.0 ** -52 if precision == "fp64" else 2.0 ** -23) * size * dmax[t]
            assert np.all(np.abs(got - want)[keep] <= tol[keep])
    assert p.digit_products()["angular"]
    p.close()
