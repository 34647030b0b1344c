"""The flux accumulators through the ring of iterations: reads after any number of
iterations (inside, on and past the chunks that a read adds) against reads after each."""
import numpy as np
import pytest

from madwave3_gb300 import Propagator

pytestmark = pytest.mark.gpu

BLOCKS = (1, 30, 32, 33, 5, 127, 128, 129, 300)


@pytest.mark.parametrize("case", ["tiny_j0", "tiny_j3"])
def test_reads_between_iterations(runs, case):
    one = Propagator(runs[case], precision="mixed")
    one.start()
    blocks = Propagator(runs[case], precision="mixed")
    blocks.start()
    last = {key: one.accumulators()[key] for key in ("zcr", "zcdr")}
    mag = {key: np.abs(last[key]) for key in last}
    for n in BLOCKS:
        for _ in range(n):
            one.run(1)
            acc = one.accumulators()
            for key in last:
                mag[key] += np.abs(acc[key] - last[key])      # |C_k psi_k|, |C_k dpsi_k|
                last[key] = acc[key]
        blocks.run(n)
        got = blocks.accumulators()
        for key in last:
            # at most 128 terms of two FP32 roundings each before a sum enters the FP64
            # accumulators, here; two roundings of each term there
            assert np.all(np.abs(got[key] - last[key]) <= 2 * (128 + 2) * 2.0 ** -23 * mag[key]), (key, n)
    assert mag["zcr"].max() > 0
    one.close()
    blocks.close()
