"""The step's lists in one launch (k_all_lists) against one launch per list: the passes are the same,
so populations, fields and sums are equal bit for bit (needs a B200).  The last lattice has enough
passes for the spread order of float32 storage."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lattice(dims, tile, column, storage):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from water_flow_simulation_b200.lbm3d import LBM3D
    nx, ny, nz = dims
    rng = np.random.default_rng(nx)
    solid = np.zeros((nz, ny, nx), bool)
    solid[:, 0] = solid[:, -1] = True
    solid[0] = rng.random((ny, nx)) < 0.2
    F = [np.zeros((nz, ny, nx), np.float32) for _ in range(3)]
    if nx > 64:
        solid[-2:, ny // 3:ny // 2 + 1, nx // 3:nx // 2] = True
        F[0][1, ny // 2, nx // 2 + 2:nx // 2 + 9] = 1e-5
    uin = (0.03 + 0.01 * rng.random((nz, ny))).astype(np.float32)
    cf = np.where(rng.random((nz, ny, nx)) < 0.5, 0.004, 0.0).astype(np.float32)
    return torch, LBM3D(None, solid, *F, uin, 0.52, 0.1, cf, bedwall=~solid if column else None,
                        uref_mode="column" if column else "field", tile=tile, storage=storage)


@pytest.mark.parametrize("column", (True, False))
@pytest.mark.parametrize("dims", ((16, 5, 4), (65, 4, 3), (129, 9, 6), (300, 40, 9), (620, 150, 24)))
@pytest.mark.parametrize("storage", ("fp32", "fp16"))
@pytest.mark.parametrize("cells,warps", ((2, 1), (2, 4), (4, 3), (4, 4)))
def test_one_launch_equals_a_launch_per_list(storage, cells, warps, dims, column):
    from water_flow_simulation_b200 import _native as nat
    got = []
    for held in (0, 4):                     # CTAs per SM held down: one launch per list
        torch, L = lattice(dims, (nat.PIPE_SPLIT, cells, warps, 0, held), column, storage)
        L.step(3)
        L.step(4, accumulate=True)
        got.append([t.clone().view(torch.uint8) for t in (L.f, L.f2, L.rho, L.ux, L.uy, L.uz, L.avg_sum("sp"))])
    assert all(torch.equal(a, b) for a, b in zip(*got))


@pytest.mark.parametrize("dims", ((16, 5, 4), (300, 40, 9), (620, 150, 24)))
@pytest.mark.parametrize("storage", ("fp32", "fp16"))
def test_steps_back_to_back_equal_steps_one_by_one(storage, dims):
    """Steps launched while the one before drains (lattices of up to 5M cells), against the same steps each
    waited for: every step reads the whole of the last one's populations and wall fields."""
    from water_flow_simulation_b200 import _native as nat
    got = []
    for wait in (False, True):
        torch, L = lattice(dims, (nat.PIPE_SPLIT, 2, 4, 0, 0) if storage == "fp16" else None, True, storage)
        if wait:
            tile, st = L.tile, L._stream()
            lat = L._lattice_ref()
            step = L.lib.lbm_fused_step_h if storage == "fp16" else L.lib.lbm_fused_step
            scale = (L.store_scale,) if storage == "fp16" else ()
            for _ in range(120):
                nat.check(step(lat, L.f.data_ptr(), L.f2.data_ptr(), *scale, nat.STEP_UREF_COLUMN, tile, st), "step")
                torch.cuda.synchronize()
                L.f, L.f2 = L.f2, L.f
            L.step(1)
        else:
            L.step(121)
        got.append([t.clone().view(torch.uint8) for t in (L.f, L.f2, L.rho, L.ux, L.uy, L.uz)])
    assert all(torch.equal(a, b) for a, b in zip(*got))
