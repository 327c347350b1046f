"""Steps launched while the one before drains, on lattices whose outlet rows are a launch of their own (nx - 1
a multiple of the segment length): the same bits as steps each waited for (needs a B200)."""
import pytest

from test_gpu_lists import lattice

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("column", (True, False))
@pytest.mark.parametrize("dims,cells", (((65, 4, 3), 2), ((129, 9, 6), 2), ((129, 9, 6), 4), ((577, 60, 9), 2), ((513, 70, 12), 4)))
@pytest.mark.parametrize("storage", ("fp32", "fp16"))
def test_steps_with_an_outlet_launch_equal_steps_one_by_one(storage, dims, cells, column):
    from water_flow_simulation_b200 import _native as nat
    assert (dims[0] - 1) % (32 * cells) == 0
    got = []
    for wait in (False, True):
        torch, L = lattice(dims, (nat.PIPE_SPLIT, cells, 4, 0, 0), column, storage)
        if wait:
            step = L.lib.lbm_fused_step_h if storage == "fp16" else L.lib.lbm_fused_step
            scale = (L.store_scale,) if storage == "fp16" else ()
            lat, mode = L._lattice_ref(), nat.STEP_UREF_COLUMN if column else 0
            for _ in range(120):
                nat.check(step(lat, L.f.data_ptr(), L.f2.data_ptr(), *scale, mode, L.tile, L._stream()), "step")
                torch.cuda.synchronize()
                L.f, L.f2 = L.f2, L.f
            L.step(1)
        else:
            L.step(121)
        got.append([t.clone().view(torch.uint8) for t in (L.f, L.f2, L.rho, L.ux, L.uy, L.uz)])
    assert all(torch.equal(a, b) for a, b in zip(*got))
