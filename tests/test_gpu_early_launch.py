"""Kernels that start while the one ahead of them in the stream still runs: their own waits have
a limit of about a second, the kernel ahead may take as long as it likes."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

from madwave3_gb300 import Propagator, build

pytestmark = pytest.mark.gpu

AHEAD = r"""
// lets the next kernel of the stream start at once and ends by itself after `cycles`
__global__ void ahead(long long cycles)
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long t0 = clock64();
    while (clock64() - t0 < cycles) __nanosleep(1000);
}

extern "C" int launch_ahead(void *stream, long long cycles)
{
    ahead<<<1, 32, 0, static_cast<cudaStream_t>(stream)>>>(cycles);
    return cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def ahead(tmp_path_factory):
    d = tmp_path_factory.mktemp("ahead")
    src, lib = str(d / "ahead.cu"), str(d / "libahead.so")
    with open(src, "w") as f:
        f.write(AHEAD)
    subprocess.run([build._nvcc()] + build.ARCH + ["-shared", "-Xcompiler", "-fPIC", "-o", lib, src], check=True)
    L = ct.CDLL(lib)
    L.launch_ahead.argtypes = [ct.c_void_p, ct.c_longlong]
    return L


@pytest.mark.parametrize("precision,n1,n2,na,dst,form", [("fp64", 24, 40, 12, -1, "digits"), ("mixed", 150, 150, 3, -1, "digits"),
                                                         ("mixed", 48, 64, 8, 0, "dst_f16"), ("mixed", 48, 64, 8, 1, "tc_dst_fused")])
def test_a_long_kernel_ahead_is_waited_for(tmp_path, ahead, precision, n1, n2, na, dst, form):
    from madwave3_gb300.host import generator, setup
    d = str(tmp_path / "case")
    generator.write_case(d, npun1=n1, npun2=n2, nangu=na, jmax=min(na - 1, 12) // 2 * 2, nvmax=1, netot=32, npun1min=8,
                         alpha0_bohr=1.2)
    run = setup.load(os.path.join(d, "input.dat"))
    out = []
    for cycles in (0, 3_200_000_000):            # 1.5 s at the highest clock
        p = Propagator(run, precision)
        if dst >= 0:
            p.set_choices({"dst": dst})
        p.start()
        p.sync()
        assert p.digit_products()["dst"] if form == "digits" else p.path()[form]
        if cycles:
            assert ahead.launch_ahead(p.stream(), cycles) == 0
        p.run(1)                                 # H psi's first kernel is the next in the stream
        p.sync()
        out.append((p.state()[1].copy(), p.norms()))
        p.close()
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
