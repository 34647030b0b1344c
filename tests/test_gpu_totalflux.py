"""P(E) against the accumulators it is read from: chunks of flux points, several
electronic states, repeated reads with and without iterations between them."""
import numpy as np
import pytest

from madwave3_gb300 import Propagator

pytestmark = pytest.mark.gpu


def _expect(p, w=0):
    run = p.runs[w]
    acc, tab = p.accumulators(w), p.tables(w)
    im = (np.conj(acc["zcr"]) * acc["zcdr"]).imag          # [flux point][E]
    mag = np.abs(acc["zcr"]) * np.abs(acc["zcdr"])
    ah1 = (run.inp.rfin1 - run.inp.rmis1) / (run.inp.npun1 - 1)
    f = np.abs(tab["reacfct"]) / ah1
    # each term is rounded twice, each sum of n terms n times: n + 2 roundings of 2^-53 at most
    return im.sum(0) * tab["reacfct"] / ah1, (len(im) + 8) * 2.0 ** -52 * mag.sum(0) * f


@pytest.mark.parametrize("case", ["tiny_j0", "tiny_j3", "tiny_e2"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_totalflux_from_accumulators(runs, case, precision):
    p = Propagator(runs[case], precision=precision)
    p.start()
    for n in (1, 40, 0, 7):
        p.run(n)
        tot, el = p.totalflux()
        again, el2 = p.totalflux()
        assert np.array_equal(tot, again) and np.array_equal(el, el2)
        want, tol = _expect(p)
        assert np.all(np.abs(tot - want) <= tol)
        assert np.all(np.abs(el.sum(0) - tot) <= tol)
        assert np.array_equal(p.totalflux()[0], tot)
    p.close()
