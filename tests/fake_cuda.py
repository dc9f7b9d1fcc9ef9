"""Runs Python code in a child process whose CUDA runtime is fake_cudart.cpp: the
library's host side - which kernels it launches, what it waits for, what it does
when a call fails - without a GPU."""
import os
import subprocess
import sys
import textwrap

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
LIB = os.path.join(ROOT, "konglong_b200", "_rtm_b200.so")

PRELUDE = """
import ctypes as C
import numpy as np
from konglong_b200 import spec as S, workloads as W
from konglong_b200._lib import STATUS_CODE, RtmError
from konglong_b200.propagator import Batch, Propagator, spread_coeffs
fake = C.CDLL(None)
for f in (fake.fake_launched, fake.fake_in_flight):
    f.restype = C.c_long
launched = lambda part="": fake.fake_launched(part.encode())
in_flight = fake.fake_in_flight
fail = lambda what, after, code=2: fake.fake_fail(what.encode(), C.c_long(after), code)


def handle(shot, receivers=True):
    s = shot.spec
    p = Propagator(s)
    p.set_model(**shot.model_arrays())
    k1, k2 = W.spread_band(s)
    src = W.make_traceset([shot.src_pos], s.nx, s.ny, s.nz, 10, k1, k2, spread_coeffs)
    p.set_injection(src, shot.wavelet[None, :], s.dt_dxyz)
    if receivers:
        p.set_extraction(W.make_traceset(shot.rcv_pos, s.nx, s.ny, s.nz, 10, k1, k2, spread_coeffs), shot.nt)
    p.reset()
    return p
"""


@pytest.fixture(scope="session")
def fake_cuda(tmp_path_factory):
    """run(code): the output of `code`, run after PRELUDE on the fake runtime."""
    if not os.path.exists(LIB):
        pytest.skip("the CUDA library is not built")
    from konglong_b200.build import nvcc
    so = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc()))), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + inc, os.path.join(HERE, "fake_cudart.cpp"),
                    "-o", so], check=True)

    def run(code):
        env = dict(os.environ, LD_PRELOAD=so, PYTHONPATH=ROOT)
        r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(code)], env=env, cwd=ROOT, timeout=600,
                           capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
        return r.stdout
    return run
