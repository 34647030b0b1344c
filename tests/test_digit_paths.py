"""Which kernels a context chooses, on the CPU: the library's host code over a stand-in CUDA
runtime (fake_cudart.cpp) that counts device memory and launches nothing."""
import ctypes as ct
import os
import shutil
import subprocess

import pytest

from madwave3_gb300 import Propagator, build, propagator
from test_gpu_fx_dst import MIXED, SHAPES, SHARED

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host compiler")
    build.build()
    objs = [os.path.join(build.OUT, s.replace(".cu", ".o")) for s in build.SOURCES]
    if not all(os.path.exists(o) for o in objs):
        build.build(force=True)
    lib = str(tmp_path_factory.mktemp("fake") / "libmw3fake.so")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build._nvcc()))), "include") \
        if os.path.isabs(build._nvcc()) else "/usr/local/cuda/include"
    subprocess.run([gxx, "-O1", "-std=c++17", "-fPIC", "-shared", "-I" + cuda, os.path.join(HERE, "fake_cudart.cpp")] + objs +
                   ["-o", lib, "-Wl,-z,defs", "-Wl,-Bsymbolic", "-lpthread", "-ldl"], check=True)
    mp = pytest.MonkeyPatch()
    mp.setattr(propagator, "_lib", None)
    mp.setattr(propagator, "library_path", lambda: lib)
    L = propagator.load_library()
    L.fake_budget.argtypes = [ct.c_size_t]
    L.fake_used.restype = L.fake_peak.restype = ct.c_size_t
    yield L
    mp.undo()


@pytest.fixture(scope="module")
def shape_run(tmp_path_factory):
    from madwave3_gb300.host import generator, setup

    def make(n1, n2, na, extra):
        d = str(tmp_path_factory.mktemp("paths") / "case")
        generator.write_case(d, npun1=n1, npun2=n2, nangu=na, jmax=min(na - 1, 12) // 2 * 2, nvmax=1, netot=32, npun1min=8,
                             alpha0_bohr=1.2, **extra)
        return setup.load(os.path.join(d, "input.dat"))
    return make


@pytest.mark.parametrize("precision,n1,n2,na,extra", [("fp64",) + s for s in SHAPES] +
                         [("mixed",) + s for s in MIXED] + SHARED)
def test_shapes_of_the_digit_products_take_them(fake, shape_run, precision, n1, n2, na, extra):
    run = shape_run(n1, n2, na, extra)
    p = Propagator(run, precision)
    p.start()
    digits = p.digit_products()
    assert digits["dst"]
    assert digits["angular"] == (precision == "fp64" or na > 64)
    p.close()
    p = Propagator(run, precision)
    p.set_choices({"dst": 3 if precision == "mixed" else 0, "angular": 0})
    p.start()
    digits = p.digit_products()
    assert not digits["dst"] and not digits["angular"]
    p.close()


def _context(fake, run, precision, choices=None, budget=1 << 40):
    """(a context after a start, one H psi and one iteration; its digit products) under a device-memory budget."""
    fake.fake_budget(fake.fake_used() + budget)
    fake.fake_peak()
    p = Propagator(run, precision)
    if choices:
        p.set_choices(choices)
    p.start()
    p.hphi(run.psi0)
    p.run(1)
    return p, p.digit_products()


# r1 lengths above 128 take a second rectangle; the last one has explicit angular matrices beside it
@pytest.mark.parametrize("precision,n1,n2,na", [("fp64", 150, 64, 3), ("mixed", 150, 150, 3), ("mixed", 145, 69, 70),
                                                ("fp64", 48, 127, 3)])
def test_digit_tables_never_cost_a_context_its_memory(fake, shape_run, precision, n1, n2, na):
    run = shape_run(n1, n2, na, {})
    base = fake.fake_used()
    p, digits = _context(fake, run, precision)
    assert digits["dst"]
    with_digits = fake.fake_used() - base
    p.close()
    assert fake.fake_used() == base
    p, digits = _context(fake, run, precision, {"dst": 3 if precision == "mixed" else 0})
    assert not digits["dst"]
    dense = fake.fake_peak() - base
    p.close()
    assert dense < with_digits
    # whatever the room between the two: the context works, without the digit tables
    for k in range(17):
        budget = dense + (with_digits - 1 - dense) * k // 16
        p, digits = _context(fake, run, precision, budget=budget)
        assert not digits["dst"], budget
        assert fake.fake_used() - base <= dense
        p.close()
        assert fake.fake_used() == base
    p, digits = _context(fake, run, precision, budget=with_digits)
    assert digits["dst"]
    # a later allocation that finds no room has them back
    p.cvj_history(64)
    p.run(1)
    assert not p.digit_products()["dst"]
    p.close()
    assert fake.fake_used() == base
    fake.fake_budget(1 << 40)


# the kernel's warps share out the registers that a CTA is launched with, 96 a thread
@pytest.mark.parametrize("precision,n1,n2,na", [("fp64", 24, 40, 4), ("mixed", 145, 69, 70)])
def test_a_kernel_with_fewer_registers_is_left_alone(fake, shape_run, precision, n1, n2, na):
    run = shape_run(n1, n2, na, {})
    try:
        for regs, taken in ((96, True), (88, False), (102, True)):
            fake.fake_registers(regs)
            p = Propagator(run, precision)
            p.start()
            digits = p.digit_products()
            assert digits["dst"] == digits["angular"] == taken
            p.close()
    finally:
        fake.fake_registers(96)


def test_a_call_of_one_iteration_stays_on_its_stream(fake, shape_run):
    """The accumulators run on a second stream only where another iteration of the call runs beside them."""
    p = Propagator(shape_run(24, 40, 4, {}), "fp64")
    p.start()
    fake.fake_waits()
    p.run(1)
    assert fake.fake_waits() == 0
    p.run(2)
    assert fake.fake_waits() == 2            # the second stream after the first update, the first before the call's end
    p.run(1)
    assert fake.fake_waits() == 0
    p.close()
