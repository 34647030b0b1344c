"""mw3_hphi_noalloc where the digit products take part: r1 lengths above 128 (dense transforms
beside digit angular terms), up to 128 (both from digits), and more than 64 angles."""
import ctypes as ct
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,n1,n2,na,J,tol", [("fp64", 150, 64, 6, 2, 1e-12), ("fp64", 40, 65, 70, 2, 1e-12),
                                                      ("mixed", 145, 50, 70, 2, 1e-6), ("mixed", 40, 64, 130, 0, 1e-6)])
def test_hphi_noalloc_beside_hphi(tmp_path, precision, n1, n2, na, J, tol):
    torch = pytest.importorskip("torch")
    from madwave3_gb300 import Propagator
    from madwave3_gb300.host import generator, setup

    d = str(tmp_path / "case")
    generator.write_case(d, npun1=n1, npun2=n2, nangu=na, jmax=min(na - 1, 12) // 2 * 2, nvmax=1, netot=32, npun1min=8,
                         alpha0_bohr=1.2, Jtot=J, iommax=J)
    run = setup.load(os.path.join(d, "input.dat"))
    p = Propagator(run, precision)
    p.L.mw3_hphi_noalloc.argtypes = [ct.c_void_p, ct.c_int32, ct.c_void_p, ct.c_void_p]
    rng = np.random.default_rng([n1, na])
    for _ in range(2):
        psi = rng.uniform(-1, 1, run.ntot)
        want = p.hphi(psi)
        x = torch.tensor(psi, dtype=torch.float64, device="cuda")
        y = torch.full_like(x, float("nan"))
        torch.cuda.synchronize()
        assert p.L.mw3_hphi_noalloc(p.h, 0, ct.c_void_p(x.data_ptr()), ct.c_void_p(y.data_ptr())) == 0, p.L.mw3_last_error(p.h)
        # the bars of the other shapes of this entry point
        assert np.abs(y.cpu().numpy() - want).max() <= tol * np.abs(want).max()
    assert p.digit_products()["angular"]
    p.close()
