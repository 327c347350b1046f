"""Kernels with more dynamic shared memory than a launch gets by default, in a second CUDA context of
the process (needs a B200).  The allowance belongs to the context -- another device's, or a host's
own as here -- so it has to be asked for in each: the same calls give the same bits in both."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


class Driver:
    """Device memory and contexts by the driver API, so that nothing is bound to the first context."""

    def __init__(self):
        self.cu = ctypes.CDLL("libcuda.so.1")
        self.ok(self.cu.cuInit(0))

    @staticmethod
    def ok(code):
        assert code == 0, f"CUDA driver error {code}"

    def primary(self):
        ctx = ctypes.c_void_p()
        self.ok(self.cu.cuDevicePrimaryCtxRetain(ctypes.byref(ctx), 0))
        self.ok(self.cu.cuCtxSetCurrent(ctx))

    def second(self):
        ctx = ctypes.c_void_p()
        self.ok(self.cu.cuCtxCreate_v2(ctypes.byref(ctx), 0, 0))       # current from here on

    def put(self, a):
        p = ctypes.c_uint64()
        self.ok(self.cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(a.nbytes)))
        self.ok(self.cu.cuMemcpyHtoD_v2(p, a.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(a.nbytes)))
        return p.value

    def get(self, p, like):
        out = np.empty_like(like)
        self.ok(self.cu.cuCtxSynchronize())
        self.ok(self.cu.cuMemcpyDtoH_v2(out.ctypes.data_as(ctypes.c_void_p), ctypes.c_uint64(p), ctypes.c_size_t(out.nbytes)))
        return out


def products(nat, lib, d):
    """lbm_gemm_bf16 of small integers: the deep ring of long sums, one tile per CTA, persistent."""
    rng = np.random.default_rng(0)
    for M, N, K, epilogue in ((64, 96, 1024, 1), (64, 96, 1024, 0), (128, 64, 256, 0), (1024, 128, 256, 0)):
        bf16 = [(rng.integers(-2, 3, (r, K)).astype(np.float32).view(np.uint32) >> 16).astype(np.uint16) for r in (M, N)]
        D, err = np.zeros((M, N), np.float32), np.zeros(1, np.int32)
        a, b, o, e = d.put(bf16[0]), d.put(bf16[1]), d.put(D), d.put(err)
        nat.check(lib.lbm_gemm_bf16(a, K, b, K, M, N, K, o, N, epilogue, None, e, None), "lbm_gemm_bf16")
        exact = [(v.astype(np.uint32) << 16).view(np.float32) for v in bf16]
        got = d.get(o, D)
        assert d.get(e, err)[0] == 0 and np.array_equal(got, exact[0] @ exact[1].T)
        yield got


def steps(nat, lib, d):
    """One step of a channel by the pipelines that stage rows in shared memory."""
    L = nat.Lattice()
    L.nx, L.ny, L.nz, L.pitch, L.cells = 160, 6, 5, 160, 160 * 30
    L.tau0, L.csmag2, L.rho_out, L.force_scale = 0.52, 0.01, 1.0, 1.0
    cell = np.zeros(L.cells, np.float32)
    solid = np.zeros((5, 6, 160), np.uint8)
    solid[:, 0] = solid[:, -1] = 1
    L.Fx, L.Fy, L.Fz, L.cfw, L.uref, L.ux, L.uy, L.uz = (d.put(cell) for _ in range(8))
    L.rho, L.uin = d.put(cell + 1), d.put(np.linspace(0.02, 0.04, 30).astype(np.float32))
    L.flags, L.status, L.colU = d.put(np.zeros(L.cells, np.uint32)), d.put(np.zeros(4, np.int32)), d.put(cell[:6 * 160])
    nat.check(lib.lbm_build_flags(ctypes.byref(L), d.put(solid), None, L.flags, None), "lbm_build_flags")
    f = np.zeros(19 * L.cells, np.float32)
    src = d.put(f)
    nat.check(lib.lbm_init_equilibrium(ctypes.byref(L), src, None), "lbm_init_equilibrium")
    for tile in ((nat.PIPE_TMA, 1, 4, 4, 0), (nat.PIPE_ASYNC, 2, 4, 3, 0)):
        dst = d.put(f)
        nat.check(lib.lbm_fused_step(ctypes.byref(L), src, dst, nat.STEP_OUTPUT, ctypes.byref(nat.Tile(*tile)), None),
                  f"lbm_fused_step {tile}")
        yield d.get(dst, f)


def in_both_contexts():
    sys.path.insert(0, ROOT)
    from water_flow_simulation_b200 import _native as nat
    lib, d, got = nat.load(), Driver(), []
    for enter in (d.primary, d.second):
        enter()
        got.append([*products(nat, lib, d), *steps(nat, lib, d)])
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    print("equal", len(got[0]))


@pytest.mark.gpu
def test_shared_memory_is_granted_in_every_context():
    run = subprocess.run([sys.executable, os.path.abspath(__file__)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "equal 6" in run.stdout, run.stdout + run.stderr


if __name__ == "__main__":
    in_both_contexts()
