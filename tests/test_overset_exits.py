"""hp_overset_build_gpu and hp_overset_hole_cut_gpu leave by an error at any of
their runtime calls: nothing they queued (copies from and into the caller's
arrays) is unfinished when they return, and no buffer is left.  They change no
setting of the process's default memory pool, and give back what they took.
Over a fake of the runtime on the CPU (overset_exit_check.cu); the child
process sees no GPU."""
import os
import shutil
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "multiphase-code_b200", "csrc")

CHILD = r'''
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[2])
from hydraphase import cases
from hydraphase._lib import HpMesh, HpOverset
from hydraphase.engine import _hp_mesh
L = ctypes.CDLL(sys.argv[1])
ov = cases.overset_cylinder(bg=(24, 24, 2), comp=(12, 48, 2), box=((-6.0, -6.0, 0.0), (6.0, 6.0, 4.0)))
keep = []
hm = _hp_mesh(ov.spec.mesh, keep)
block = np.ascontiguousarray(ov.block, np.int32)
ib = np.zeros(ov.spec.mesh.neles, np.int32)
ip = ctypes.POINTER(ctypes.c_int32)
bp, op = block.ctypes.data_as(ip), ib.ctypes.data_as(ip)
rep = (ctypes.c_int * 5)()

def build():
    out = HpOverset()
    return L.hp_overset_build_gpu(ctypes.byref(hm), bp, ov.layers, ov.outer_type, op, ctypes.byref(out))

def cut():
    return L.hp_overset_hole_cut_gpu(ctypes.byref(hm), bp, 6, ctypes.c_double(0.7), op, None)

for name, fn in (("build", build), ("cut", cut)):
    k = 0
    while True:
        k += 1
        L.fake_reset(k)
        rc = fn()
        L.fake_report(rep)
        # call k was made, so it failed
        assert rc != 0 or rep[0] < k, (name, k, rc)
        print(name, k, rc, *rep)
        if rep[0] < k:
            break
'''


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    so = str(tmp_path_factory.mktemp("exits") / "libexits.so")
    subprocess.run([nvcc, "-O1", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC,-fopenmp",
                    "-shared", "-o", so, os.path.join(HERE, "overset_exit_check.cu"),
                    os.path.join(CSRC, "hp_overset.cpp")], check=True)
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")
    out = subprocess.run([sys.executable, "-c", CHILD, so, os.path.join(HERE, "..", "multiphase-code_b200")],
                         capture_output=True, text=True, timeout=300, env=env)
    assert out.returncode == 0, out.stdout[-1000:] + out.stderr[-3000:]
    rows = [line.split() for line in out.stdout.splitlines()]
    return [(r[0], *map(int, r[1:])) for r in rows if r and r[0] in ("build", "cut")]


@pytest.mark.parametrize("name", ["build", "cut"])
def test_nothing_is_unfinished_at_an_error_exit(report, name):
    rows = [r for r in report if r[0] == name]
    assert len(rows) > 12 and rows[-1][2] == 0   # the last run made all its calls
    for _, k, rc, calls, pending, live, sets, kept in rows:
        assert pending == 0 and live == 0, f"call {k} failing (status {rc}): {pending} unfinished, {live} not freed"


@pytest.mark.parametrize("name", ["build", "cut"])
def test_the_default_pool_is_left_alone(report, name):
    rows = [r for r in report if r[0] == name]
    assert all(sets == 0 and kept == 0 for *_, sets, kept in rows)
