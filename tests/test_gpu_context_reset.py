"""The standalone Poisson solves and new jobs in a new context: after
cudaDeviceReset the kernels' twiddle tables, shared-memory limits and
cluster-size attribute are those of the new context, and everything gives the
bits it gave before.

Each test runs in a process of its own: a reset ends the context of everything
else in the process.
"""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PRELUDE = """
import ctypes as C, glob, os, sys
import numpy as np
sys.path.insert(0, %r)
import replace_gb300
lib = replace_gb300.load()
paths = glob.glob("/usr/local/cuda/lib64/libcudart.so") + glob.glob(
    os.path.join(os.path.dirname(np.__file__), "..", "nvidia", "*", "lib", "libcudart.so*"))
rt = C.CDLL(paths[0])

def ok(status):
    assert status == 0, status

def solve(fn, nx, ny, phi):
    d = (0.7 + 0.4 * np.random.default_rng(nx + ny).random((ny, nx))).astype(np.float32)
    buf = []
    for _ in range(4):
        p = C.c_void_p()
        ok(rt.cudaMalloc(C.byref(p), C.c_size_t(d.nbytes)))
        ok(rt.cudaMemset(p, 0, C.c_size_t(d.nbytes)))
        buf.append(p)
    ok(rt.cudaMemcpy(buf[0], d.ctypes.data_as(C.c_void_p), C.c_size_t(d.nbytes), 1))
    rc = getattr(lib, fn)(C.c_int32(nx), C.c_int32(ny), C.c_int32(380), C.c_int32(1400), buf[0],
                          buf[1] if phi else None, buf[2], buf[3], None)
    assert rc == 0, (fn, nx, ny, rc, lib.gpl_last_error())
    ok(rt.cudaDeviceSynchronize())
    out = []
    for p in buf[1:]:
        a = np.empty_like(d)
        ok(rt.cudaMemcpy(a.ctypes.data_as(C.c_void_p), p, C.c_size_t(d.nbytes), 2))
        out.append(a)
    for p in buf:
        ok(rt.cudaFree(p))
    assert np.abs(out[1]).max() > 0
    return out
""" % ROOT

SOLVES = """
grids = [(64, 32), (64, 64), (128, 128), (256, 256), (512, 256), (256, 512), (1024, 512), (512, 512)]
cases = [(fn, nx, ny, phi) for fn in ("gpl_poisson_solve", "gpl_poisson_solve_noalloc") for nx, ny in grids
         for phi in (False, True) if fn == "gpl_poisson_solve" or nx * ny <= 512 * 512]
want = [solve(*c) for c in cases]
ok(rt.cudaDeviceReset())
for c, w in zip(cases, want):
    for a, b in zip(solve(*c), w):
        assert np.array_equal(a, b), c
print("same")
"""

# 64 x 64 tiles of bins whose sums need two window words: 83 KB of shared memory
JOBS = """
from replace_gb300 import Placer, batch_nesterov_run, netlist as N
nl = N.generate(9_000, 9_450, n_io=60, seed=5)

def outcome(batched):
    p = Placer(nl, target_density=0.75, initial_place_max_iter=1, bin_grid_cnt_x=64, bin_grid_cnt_y=64,
               poisson_path=1, scatter_tile=64)
    p.initial_place()
    p.nesterov_init()
    batch_nesterov_run([p], 5) if batched else p.nesterov_run(5)
    xy = p.gcell_coords()
    p.close()
    return xy

want = [outcome(b) for b in (False, True)]
ok(rt.cudaDeviceReset())
for b, w in zip((False, True), want):
    assert np.array_equal(outcome(b), w), b
print("same")
"""


def run(body):
    r = subprocess.run([sys.executable, "-c", PRELUDE + body], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.endswith("same\n"), r.stdout + r.stderr


def test_poisson_solves_after_a_reset(gpu_lib):
    run(SOLVES)


def test_jobs_after_a_reset(gpu_lib):
    run(JOBS)
