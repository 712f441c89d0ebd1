"""Meshes, flows and solves when device memory is short.

Fixed-width copies of a matrix, edge tables and the dense coarse operator speed
up calls that do not depend on them: no amount of free memory that was enough
without them may be too little with them. The library's host side runs here
against a stand-in for the CUDA runtime whose device has a settable size
(fake_cudart.cpp): first without a limit, then with the largest size that has
no room for a fixed-width matrix beside the rest, and with sizes from there to
beyond the one at which everything is taken."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes as C, sys
import numpy as np
from openaccel_b200 import meshgen, runtime as rt

fake = C.CDLL(None)
for n in ("fake_used", "fake_peak"):
    getattr(fake, n).restype = C.c_size_t
fake.fake_limit.argtypes = [C.c_size_t]
case, prec = sys.argv[1], int(sys.argv[2])
if case == "flow":
    m = meshgen.cavity(24)
    width = 7
else:
    m = meshgen.conduction(16)[0]
    width = 15

def go(limit):
    "everything a program asks for, at a device of limit bytes; the most it held"
    fake.fake_limit(limit)
    fake.fake_peak()
    gm = rt.Mesh(m)
    if case == "flow":
        f = rt.Flow(gm, rt.default_settings(precision=prec))
        f.initialize()
        f.simple_iterate(1)
        f.assemble_pcorr()
        f.solve("pcorr", 1e-8, 4)
    else:
        f = rt.Diffusion(gm, rt.default_diffusion_settings(precision=prec))
        f.assemble()
        f.solve(1e-8, 4)
    f.close()
    gm.close()
    assert fake.fake_used() == 0
    return fake.fake_peak()

whole = go(1 << 40)
slots = 32 * width * ((m.nn + 31) // 32)
fixed_width = slots * (4 + (4 if prec == rt.OA_PREC_MIXED else 8))
print("bytes per row: %.0f, of them fixed width %.0f" % (whole / m.nn, fixed_width / m.nn))
small = whole - fixed_width
assert go(small) <= small
for k in range(25):
    go(small + k * m.nn * 300)
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(cuda, "include"), "-o", so,
                    os.path.join(ROOT, "tests", "fake_cudart.cpp")], check=True)
    return so


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("case", ["flow", "conduction"])
def test_no_call_is_refused_for_storage_it_can_do_without(fake, case, prec):
    r = subprocess.run([sys.executable, "-c", CHILD, case, str(prec)], cwd=ROOT, capture_output=True, text=True,
                       env={**os.environ, "LD_PRELOAD": fake, "PYTHONPATH": ROOT}, timeout=600)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]
