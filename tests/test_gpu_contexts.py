"""Kernels that take more than 48 KB of shared memory in one CUDA context after another of the same
process: the opt-in belongs to the context. A child process with contexts of its own (driver calls),
made and destroyed in turn; every launch has to succeed in each of them."""
from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import ctypes, sys
import numpy as np
sys.path.insert(0, {pkg!r})
from fsi import _native as nat

cu = ctypes.CDLL("libcuda.so.1")
vp, u64 = ctypes.c_void_p, ctypes.c_uint64

def ok(status):
    assert status == 0, status

def put(a):
    p = u64()
    ok(cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(a.nbytes)))
    ok(cu.cuMemcpyHtoD_v2(p, a.ctypes.data_as(vp), ctypes.c_size_t(a.nbytes)))
    return p.value

def get(p, a):
    ok(cu.cuMemcpyDtoH_v2(a.ctypes.data_as(vp), u64(p), ctypes.c_size_t(a.nbytes)))
    return a

def substep():
    n, d, q = 600, nat.MpmDesc(), nat.Particles()
    d.nx = d.ny = d.nz = 16
    d.num_particles, d.dt, d.dx, d.inv_dx, d.mu, d.lam = n, 0.01, 1.0, 1.0, 1.0, 1.0
    d.boundary_width, d.apic, d.clamp_lower, d.launch_threads = 1, 1, 1.0, 512
    for a in range(3):
        d.clamp_upper[a] = 14.0
    rng = np.random.default_rng(0)
    F = np.zeros((9, n), np.float32)
    F[[0, 4, 8]] = 1.0
    v = np.full((3, n), 0.5, np.float32)
    arrays = dict(x=rng.uniform(6, 9, (3, n)).astype(np.float32), v=v, C=np.zeros((9, n), np.float32), F=F,
                  mass=np.ones(n, np.float32), volume=np.ones(n, np.float32), active=np.ones(n, np.int32),
                  force=np.zeros((3, n), np.float32))
    for name, a in arrays.items():
        setattr(q, name, put(a))
    q.capacity = n
    nat.call("fsi_mpm_substep_noalloc", d, q, None)
    ok(cu.cuCtxSynchronize())
    assert np.abs(get(q.v, np.zeros_like(v)) - 0.5).max() < 1e-5

def gemm():
    m, n, k = 128, 64, 64
    one = np.full(m * k, 0x3F80, np.uint16)  # 1 in BF16
    g = nat.ClosureGemmDesc()
    g.a, g.b, g.lda, g.ldb = put(one), put(one), k, k
    g.m, g.n, g.k, g.k_chunk, g.mode, g.ldc = m, n, k, k, nat.GEMM_STORE, n
    c = np.zeros((m, n), np.float32)
    g.c, g.err = put(c), put(np.zeros(4, np.int32))
    nat.call("fsi_closure_gemm", g, None)
    ok(cu.cuCtxSynchronize())
    assert (get(g.c, c) == k).all()

ok(cu.cuInit(0))
for _ in range(2):
    ctx = vp()
    ok(cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, 0))
    substep()
    gemm()
    ok(cu.cuCtxDestroy_v2(ctx))
for _ in range(3):  # the device's primary context, reset in between
    ctx = vp()
    ok(cu.cuDevicePrimaryCtxRetain(ctypes.byref(ctx), 0))
    ok(cu.cuCtxSetCurrent(ctx))
    substep()
    gemm()
    ok(cu.cuDevicePrimaryCtxReset_v2(0))
print("contexts ok")
"""


def test_large_shared_memory_in_contexts_of_one_process():
    pkg = str(Path(__file__).resolve().parents[1] / "taichi-mpm-lbm_gb300")
    r = subprocess.run([sys.executable, "-c", CHILD.format(pkg=pkg)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "contexts ok" in r.stdout, r.stdout + r.stderr
