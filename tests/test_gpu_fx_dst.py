"""The FP64 path's radial DSTs and angular terms from exact digits on the tensor cores
against the CPU oracle: even and odd R lengths, lengths along r1 and angles on both sides
of one 128-row operand, tiles and K steps with remainders, coupled blocks, several
electronic states, inc = 2, and non-finite input."""
import os

import numpy as np
import pytest

from madwave3_gb300 import Propagator
from oracle.mw3ref import Oracle

pytestmark = pytest.mark.gpu

#        npun1 npun2 nangu  extra
SHAPES = [(24, 40, 4, {}), (33, 65, 3, {}), (48, 127, 3, {}), (130, 131, 2, {}), (128, 256, 3, {"Jtot": 2, "iommax": 2}),
          (200, 257, 2, {}), (256, 300, 2, {}), (145, 385, 2, {}), (64, 512, 2, {"nelecmax": 2}),
          (24, 33, 17, {"Jtot": 4, "iommax": 3}), (28, 40, 64, {"Jtot": 1, "iommax": 1, "iparity": -1}),
          (24, 36, 129, {}), (20, 34, 145, {"Jtot": 2, "iommax": 2}), (24, 40, 12, {"inc": 2}),
          (24, 40, 9, {"nelecmax": 3, "lambdas": (0, 1, 0), "Jtot": 2, "iommax": 2})]


@pytest.fixture(scope="module")
def shape_run(tmp_path_factory):
    from madwave3_gb300.host import generator, setup

    def make(n1, n2, na, extra):
        d = str(tmp_path_factory.mktemp("fx") / "case")
        generator.write_case(d, npun1=n1, npun2=n2, nangu=na, jmax=min(na - 1, 12) // 2 * 2, nvmax=1, netot=32, npun1min=8,
                             alpha0_bohr=1.2, **extra)
        return setup.load(os.path.join(d, "input.dat"))
    return make


@pytest.mark.parametrize("n1,n2,na,extra", SHAPES)
def test_hphi_against_the_oracle(shape_run, n1, n2, na, extra):
    run = shape_run(n1, n2, na, extra)
    p, ref = Propagator(run, "fp64"), Oracle(run)
    rng = np.random.default_rng([n1, n2])
    for psi in (rng.uniform(-1, 1, run.ntot), run.psi0, rng.normal(size=run.ntot) * 10.0 ** rng.uniform(-20, 0, run.ntot)):
        h, e = p.hphi(psi), ref.hphi(psi)
        # four products of up to 512 terms and the oracle's own FP64 rounding
        assert np.abs(h - e).max() <= 1e-13 * np.abs(e).max()
    assert not p.path()["rader"]
    p.close()


# mixed shapes whose r1 lengths pass one 128-row operand
MIXED = [(150, 150, 3, {}), (256, 512, 2, {}), (145, 69, 70, {"Jtot": 2, "iommax": 2}),
         (148, 50, 129, {"Jtot": 1, "iommax": 1, "iparity": -1}),
         (160, 400, 6, {"nelecmax": 2, "lambdas": (0, 1), "Jtot": 2, "iommax": 2})]


@pytest.mark.parametrize("n1,n2,na,extra", MIXED)
def test_mixed_hphi_against_the_oracle(shape_run, n1, n2, na, extra):
    run = shape_run(n1, n2, na, extra)
    p, ref = Propagator(run, "mixed"), Oracle(run)
    rng = np.random.default_rng([n1, n2])
    for psi in (rng.uniform(-1, 1, run.ntot), run.psi0):
        h, e = p.hphi(psi), ref.hphi(psi)
        # FP32 vectors between exact products: the mixed path's bar
        assert np.abs(h - e).max() <= 1e-6 * np.abs(e).max()
    p.start()
    assert not p.path()["tc_dst"]
    ref.start(run.psi0)
    p.run(20)
    nrm = ref.run_iters(20)
    assert np.abs(p.norms()[1:] - nrm).max() <= 1e-5 * np.abs(nrm).max()
    p.close()


@pytest.mark.parametrize("n1,n2,na,extra", [(48, 64, 66, {"nelecmax": 2}), (20, 34, 145, {"Jtot": 2, "iommax": 2})])
@pytest.mark.parametrize("dst", [0, 3])
def test_mixed_angular_form_beside_the_explicit_one(shape_run, n1, n2, na, extra, dst):
    run = shape_run(n1, n2, na, extra)
    want, err = Oracle(run).hphi(run.psi0), {}
    for ang in (-1, 0):
        p = Propagator(run, "mixed")
        p.set_choices({"dst": dst, "angular": ang})
        err[ang] = np.abs(p.hphi(run.psi0) - want).max() / np.abs(want).max()
        p.close()
    # no further off than the explicit FP32 sums, up to one rounding of the vectors kept in FP32
    assert err[-1] <= err[0] + 2.0 ** -23


def test_non_finite_input_stays_non_finite(shape_run):
    run = shape_run(24, 40, 4, {})
    p = Propagator(run, "fp64")
    psi = np.random.default_rng(5).uniform(-1, 1, run.ntot)
    clean = p.hphi(psi)
    for bad in (np.nan, np.inf, -np.inf):
        x = psi.copy()
        x[7] = bad
        assert not np.isfinite(p.hphi(x)).all()
    assert np.array_equal(p.hphi(psi), clean)
    assert np.array_equal(p.hphi(np.zeros(run.ntot)), np.zeros(run.ntot))
    # subnormal and huge vectors scale as FP64 does
    assert np.allclose(p.hphi(psi * 2.0 ** 900), clean * 2.0 ** 900, rtol=1e-12)
    p.close()


# enough tiles that a CTA takes several in a row and the later ones share the vectors, their
# digits or their differences: odd and even R lengths, one and two B blocks and 128-row blocks,
# runs of tiles that begin inside a group
SHARED = [("fp64", 40, 65, 120, {}), ("fp64", 130, 257, 24, {}), ("fp64", 64, 512, 40, {}), ("fp64", 200, 96, 60, {}),
          ("fp64", 145, 255, 20, {}), ("mixed", 150, 385, 40, {}), ("mixed", 145, 129, 90, {}), ("mixed", 256, 258, 30, {})]


@pytest.mark.parametrize("precision,n1,n2,na,extra", SHARED)
def test_tiles_that_share_vectors(shape_run, precision, n1, n2, na, extra):
    run = shape_run(n1, n2, na, extra)
    p = Propagator(run, precision)
    psi = np.random.default_rng([n1, n2, na]).uniform(-1, 1, run.ntot)
    h, e = p.hphi(psi), Oracle(run).hphi(psi)
    # as the shapes with a tile a CTA
    assert np.abs(h - e).max() <= (1e-13 if precision == "fp64" else 1e-6) * np.abs(e).max()
    assert np.array_equal(p.hphi(psi), h)
    p.close()
