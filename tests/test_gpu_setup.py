"""Case set-up kernels at sizes where they can go wrong (needs a B200): row padding, the
four-cell flag kernel and the all-SM list compaction against NumPy, integers equal; and each
against its one-cell-per-thread form on misaligned arrays."""
import ctypes

import numpy as np
import pytest

from oracle.oracle import wall_mask
from test_gpu_parity import _require_gpu, expected_wallfn

pytestmark = pytest.mark.gpu

SIZES = ((4, 3, 2), (7, 5, 3), (61, 4, 5), (66, 33, 9), (129, 40, 37), (200, 150, 90))


def lattice_case(nx, ny, nz, storage):
    import torch
    from water_flow_simulation_b200.lbm3d import LBM3D
    rng = np.random.default_rng(nx)
    solid = rng.random((nz, ny, nx)) < 0.02
    solid[:, : ny // 3, : nx // 2] = True                     # whole solid segments too
    F = [np.where(rng.random((nz, ny, nx)) < 0.001, 1e-5, 0).astype(np.float32) for _ in range(3)]
    cf = np.where(rng.random((nz, ny, nx)) < 0.5, 3e-3, 0).astype(np.float32)
    bw = rng.random((nz, ny, nx)) < 0.3
    uin = rng.uniform(0, 0.1, (nz, ny)).astype(np.float32)
    dev = [torch.as_tensor(a, device="cuda") for a in (solid, *F, uin, cf, bw)]
    L = LBM3D(torch.device("cuda"), *dev[:5], 0.6, 0.17, dev[5], bedwall=dev[6], uref_mode="column", storage=storage)
    return L, solid, F, cf, bw, uin


@pytest.mark.parametrize("storage", ("fp32", "fp16"))
@pytest.mark.parametrize("size", SIZES)
def test_flags_lists_and_start(size, storage):
    torch = _require_gpu()
    nx, ny, nz = size
    L, solid, F, cf, bw, uin = lattice_case(*size, storage)
    got = L._flags.cpu().numpy().view(np.uint32).reshape(nz, ny, L.pitch)
    wm = wall_mask(solid).astype(np.uint32)
    want = wm | (1 << 20) * (np.any([f != 0 for f in F], axis=0)).astype(np.uint32)
    want |= (1 << 21) * expected_wallfn(solid, cf).astype(np.uint32) | (1 << 22) * bw.astype(np.uint32)
    want = np.where(solid, 1 << 19, want)
    assert np.array_equal(got[..., :nx], want)
    assert (got[..., nx:] == (1 << 19 | 1 << 23)).all()
    # lists from the flags
    seg = 32 * L.tile.cells_per_lane
    nseg = -(-L.pitch // seg)
    fl = np.full((nz, ny, nseg * seg), 1 << 19, np.uint32)
    fl[..., :L.pitch] = got
    fl = fl.reshape(nz, ny, nseg, seg)
    x = np.arange(nseg * seg).reshape(nseg, seg)
    all_solid = ((fl >> 19) & 1).all(-1)
    special = (((fl & (0x7FFFE | 1 << 19 | 1 << 20 | 1 << 21)) != 0) & (x < nx)).any(-1)
    y, z = np.arange(ny)[None, :, None], np.arange(nz)[:, None, None]
    open_row = (y >= 1) & (y <= ny - 2) & (z >= 1)
    clear = (np.arange(nseg) > 0) & ((np.arange(nseg) + 1) * seg < nx)
    cls = np.where(all_solid, 1, np.where(open_row & ~special, np.where(clear, 0, 3), 2)).ravel()
    for k in range(4):
        n = L._wl[1][k]
        assert np.array_equal(L._wl[0][k][:n].cpu().numpy(), np.flatnonzero(cls == k)), k
    # the same flags and start state from misaligned arrays (the one-cell-per-thread kernels)
    lat = L._lattice()
    odd = torch.empty(L.cells + 1, dtype=torch.int32, device="cuda")[1:]
    assert L.lib.lbm_build_flags(ctypes.byref(lat), L._solid.data_ptr(), L._bedwall.data_ptr(), odd.data_ptr(), L._stream()) == 0
    assert torch.equal(odd, L._flags)
    f = torch.empty(19 * L.cells + 1, dtype=L.f.dtype, device="cuda")[1:]
    if storage == "fp16":
        assert L.lib.lbm_init_equilibrium_h(ctypes.byref(lat), f.data_ptr(), L.store_scale, L._stream()) == 0
    else:
        assert L.lib.lbm_init_equilibrium(ctypes.byref(lat), f.data_ptr(), L._stream()) == 0
    assert torch.equal(f, L.f) and torch.equal(f, L.f2)


def test_pitch_rows_argument_errors():
    _require_gpu()
    from water_flow_simulation_b200 import _native as nat
    lib = nat.load()
    for args in ((None, 4, 4, 4), (4096, 2, 4, 4), (4096, 4, 5, 4), (4096, 4, 4, 6), (4098, 4, 4, 8)):
        assert lib.lbm_pitch_rows(args[0], 4096, *args[1:], 3, 0, None) == -1
