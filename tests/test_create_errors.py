"""Creation of a context when a call of the CUDA runtime fails, on the CPU: the library's object files linked with a
stand-in runtime on host memory (tests/c/fake_cudart.c) whose n-th call fails. Every failure has to come back as
DGPU_ERR_CUDA with the runtime's own message, and the next creation has to succeed."""
import ctypes
import glob
import os
import re
import subprocess

import pytest

from dpgsolver_gb300 import _lib
from dpgsolver_gb300.host import problem as P
from dpgsolver_gb300.host.mixed_types import mixed_tri_quad_euler, mixed_types_euler
from dpgsolver_gb300.solver import BatchSimulation, Simulation

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    _lib.build(force=not glob.glob(os.path.join(_lib.BUILD_DIR, "dgpu_batched_0.o")))
    objs = [os.path.join(_lib.BUILD_DIR, f"{os.path.splitext(s)[0]}_{k}.o")
            for s in _lib.SOURCES for k in range(_lib.PARTS.get(s, 1))]
    out = tmp_path_factory.mktemp("fake")
    obj, so = str(out / "fake_cudart.o"), str(out / "libdgpu_fake.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(_lib.nvcc_path())), "include")
    subprocess.run(["gcc", "-std=gnu11", "-O1", "-fPIC", "-Wall", "-Wextra", "-Werror", "-I", inc, "-c",
                    os.path.join(HERE, "c", "fake_cudart.c"), "-o", obj], check=True)
    subprocess.run(["g++", "-shared", "-Wl,-Bsymbolic", "-o", so] + objs + [obj], check=True)
    lib = ctypes.CDLL(so)
    for name, (res, args) in _lib.EXPORTS.items():
        fn = getattr(lib, name)
        fn.restype, fn.argtypes = res, args
    lib.fake_fail_at.argtypes, lib.fake_calls.restype = [ctypes.c_long], ctypes.c_long
    before, _lib._lib = _lib._lib, lib
    yield lib
    _lib._lib = before


@pytest.mark.parametrize("kind", ["uniform", "tri_quad", "types"])
def test_every_failing_call_is_reported(fake, kind):
    make, prob = {"uniform": lambda: (Simulation, P.euler_hex_3d(2, 2)),
                  "tri_quad": lambda: (BatchSimulation, mixed_tri_quad_euler(3, p_set=(1, 2), seed=0)),
                  "types": lambda: (BatchSimulation, mixed_types_euler(4, p_set=(1, 2), seed=0))}[kind]()
    n, failed = 0, 0
    while True:   # a failing call whose result does not matter (a query of an optional form) may be passed over
        n += 1
        fake.fake_fail_at(n)
        try:
            make(prob).close()
            if fake.fake_calls() < n:
                break
        except _lib.DGPUError as e:
            failed += 1
            assert e.status == 3 and re.fullmatch(r"dgpu status 3: [ -~]{4,}: .*out of memory.*", str(e))
    assert failed > 20
    fake.fake_fail_at(0)
    make(prob).close()
