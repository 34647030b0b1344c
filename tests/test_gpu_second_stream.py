"""The accumulators on a stream of their own beside the next iteration's H psi: the same bits as
in sequence (as while stages are timed), with everything that they keep switched on, and in two
contexts on two host threads at once."""
import copy
import threading

import numpy as np
import pytest

from conftest import synthetic_product_tables
from madwave3_gb300 import Propagator
from madwave3_gb300.host import constants as C

pytestmark = pytest.mark.gpu

BLOCKS = (1, 33, 5, 64, 2, 31, 40)       # single iterations, captured blocks, both parities


def _context(run, precision):
    run = copy.copy(run)
    run.efe_zot = np.array([0.3, 0.9]) * C.eV2cm * C.conve1
    p = Propagator(run, precision)
    p.set_product_projection(synthetic_product_tables(run))
    p.cvj_history(48)
    return p


def _propagate(p, read):
    p.start()
    out = []
    for n in BLOCKS:
        p.run(n)
        if read:
            out.append(p.totalflux()[0])
    out += [*p.state()[:2], p.norms(), p.totalflux()[0], p.psi_e(), *p.product()]
    acc = p.accumulators()
    out += [acc[k] for k in sorted(acc)]
    out += [np.asarray(x) for x in p.download_cvj_history(48) if x is not None]
    return out


def _same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("case", ["tiny_j3", "tiny_e2"])
@pytest.mark.parametrize("read", [False, True])
def test_beside_as_in_sequence(runs, case, precision, read):
    out = []
    for sequence in (False, True):
        p = _context(runs[case], precision)
        if sequence:
            p.profile(True)
        out.append(_propagate(p, read))
        p.close()
    _same(*out)


@pytest.mark.parametrize("precision", [("fp64", "fp64"), ("mixed", "fp64"), ("mixed", "mixed")])
def test_two_contexts_on_two_threads(runs, precision):
    cases = ("tiny_j3", "tiny_e2")
    alone = []
    for case, pr in zip(cases, precision):
        p = _context(runs[case], pr)
        alone.append(_propagate(p, True))
        p.close()
    both, errors = [None, None], []

    def drive(i):
        try:
            p = _context(runs[cases[i]], precision[i])
            for _ in range(3):
                both[i] = _propagate(p, True)
            p.close()
        except Exception as e:           # raised again below
            errors.append(e)

    threads = [threading.Thread(target=drive, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for a, b in zip(alone, both):
        _same(a, b)
