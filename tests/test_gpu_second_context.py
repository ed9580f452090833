"""Work in a second CUDA context of one process, as a second device would be:
what a kernel's launches need of the device (its shared-memory limit) is asked
for in the context that is current, not once a process.  A child process runs
propagator, LSRTM operator and analysis, resets its context and runs them
again; both runs give the same bits."""
import os
import subprocess
import sys

import pytest

from tests.conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes as C
import numpy as np
import swfwi_b200 as S

lib = S.lib()
rt = C.CDLL("libcudart.so.12")


def ok(status):
    assert status == 0, (status, lib.swfwi_last_error())


def dev(a=None, size=0):
    p = C.c_void_p()
    n = a.nbytes if a is not None else size
    ok(rt.cudaMalloc(C.byref(p), C.c_size_t(n)))
    if a is not None:
        ok(rt.cudaMemcpy(p, a.ctypes.data_as(C.c_void_p), C.c_size_t(n), 1))
    else:
        ok(rt.cudaMemset(p, 0, C.c_size_t(n)))
    return p


def host(p, shape, dtype=np.float32):
    a = np.empty(shape, dtype)
    ok(rt.cudaDeviceSynchronize())
    ok(rt.cudaMemcpy(a.ctypes.data_as(C.c_void_p), p, C.c_size_t(a.nbytes), 2))
    return a


def work():
    out = []
    none = C.c_void_p(0)
    # a gradient of the encoded form: both sweeps
    nx, nz, nb, nt, ns = 300, 120, 20, 260, 4
    src, geo = S.ShotPosition(5, 10, 0, 60, ns, nz), S.ShotPosition(5, 0, 0, 1, nx, nz)
    h = C.c_void_p()
    ok(lib.swfwi_damp4t10d_create(C.byref(h), C.byref(src.c), C.byref(geo.c), 0.002, 20.0, 10.0, nb, nt))
    ok(lib.swfwi_damp4t10d_set_arith(h, S.ARITH_FAST))
    v = np.full((nx, nz), 2000.0, np.float32) + 8.0 * np.arange(nz, dtype=np.float32)
    ex = np.zeros((nx + 2 * nb + 12, nz + nb + 12), np.float32)
    fp = C.POINTER(C.c_float)
    ok(lib.swfwi_damp4t10d_expand_domain(h, v.ctypes.data_as(fp), nx, nz, ex.ctypes.data_as(fp)))
    vel = dev(ex)
    ok(lib.swfwi_damp4t10d_bind_velocity(h, vel))
    enc = dev(np.repeat(S.ricker_wavelet(nt, 10.0, 0.002)[:, None], ns, 1).copy())
    rec = dev(size=4 * nt * nx)
    ok(lib.swfwi_damp4t10d_ess_forward_modeling(h, enc, rec))
    grad = dev(size=ex.nbytes)
    ok(lib.swfwi_damp4t10d_calgradient_ess(h, enc, rec, grad))
    out += [host(rec, (nt, nx)), host(grad, ex.shape)]
    ok(lib.swfwi_damp4t10d_destroy(h))
    # LSRTM: modelling and migration
    nx, nz, ng = 120, 90, 100
    p = C.c_void_p()
    vel = dev(np.full((nx, nz), 2000.0, np.float32))
    ok(lib.swfwi_prtm2d_create(C.byref(p), S.ARITH_FAST, 10.0, 10.0, 0.001, 1.0, 25.0, nz, nx, 20, nt, 2, ng, 10, 2, 50,
                               0, 5, 2, 1, 0, 0, vel, none))
    mod = dev(np.random.default_rng(1).standard_normal((nx, nz)).astype(np.float32))
    dat = dev(size=4 * 2 * ng * nt)
    ok(lib.swfwi_prtm2d_lop(p, 0, 0, nx * nz, 2 * ng * nt, mod, dat, none))
    ok(lib.swfwi_prtm2d_lop(p, 1, 0, nx * nz, 2 * ng * nt, mod, dat, none))
    out += [host(dat, (2, ng, nt)), host(mod, (nx, nz))]
    ok(lib.swfwi_prtm2d_destroy(p))
    # analysis
    rows, n = 5000, 16
    r = np.random.default_rng(2)
    ha, obs = dev(r.standard_normal((n, rows)).astype(np.float32)), dev(r.standard_normal(rows).astype(np.float32))
    t4, sigma, clip = np.zeros((n, n)), C.c_double(0.0), C.c_int()
    ok(lib.swfwi_enkf_gain_matrix(ha, obs, none, rows, n, 0.01, C.byref(sigma), 7,
                                  t4.ctypes.data_as(C.POINTER(C.c_double)), C.byref(clip), none))
    return out + [t4]


first = work()
ok(rt.cudaDeviceReset())
second = work()
for a, b in zip(first, second):
    assert np.abs(a).max() > 0 and np.array_equal(a, b)
print("same bits")
"""


def test_a_second_context_of_the_process(cuda):
    r = subprocess.run([sys.executable, "-c", CHILD], capture_output=True, text=True, timeout=120, cwd=ROOT,
                       env={**os.environ, "PYTHONPATH": ROOT})
    assert r.returncode == 0 and "same bits" in r.stdout, r.stdout + r.stderr
