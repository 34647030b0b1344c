"""The digit products at the small end: vectors of subnormal numbers."""
import os

import numpy as np
import pytest

from madwave3_gb300 import Propagator

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def shape_run(tmp_path_factory):
    from madwave3_gb300.host import generator, setup

    def make(n1, n2, na, extra):
        d = str(tmp_path_factory.mktemp("fxs") / "case")
        generator.write_case(d, npun1=n1, npun2=n2, nangu=na, jmax=min(na - 1, 12) // 2 * 2, nvmax=1, netot=32, npun1min=8,
                             alpha0_bohr=1.2, **extra)
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
    assert np.abs(p.hphi(psi) - clean).max() <= tol + rel * np.abs(clean).max()
    p.close()
