"""Row ends of the split pipeline (k_edge, and k_cells at x = 0 and x = nx-1) against the oracle
(needs a B200): every place of the outlet cell in its lane (nx-1 mod 4), and the outlet at the
start of a 32-, 64- and 128-cell pass.

Bars, from rounding alone: a post-collision population takes at most 16 float32 roundings of terms
below 1 (2^-24 each): 2^-20.  16-bit storage rounds the deviation f - w once more, 2^-11 of it, and
where x = nx-1 starts a segment the outlet is extrapolated from the stored x = nx-2 populations g,
which adds |d g_i| + w_i sum_j |d g_j|.
"""
import numpy as np
import pytest

from parity_util import make_oracle
from test_gpu_fp16 import W, case, pitched
from test_gpu_parity import _require_gpu, make_solver

pytestmark = pytest.mark.gpu

NX = (513, 545, 577, 609, 578, 579, 580)      # nx-1 mod 128: 0, 32, 64, 96; mod 4: 1, 2, 3


@pytest.mark.parametrize("tile", [(3, 2, 4, 0, 0), (3, 4, 4, 0, 0), (3, 4, 2, 0, 1), (3, 8, 4, 0, 0)])
@pytest.mark.parametrize("nx", NX)
@pytest.mark.parametrize("storage", ("fp32", "fp16"))
def test_row_ends_against_oracle(storage, nx, tile):
    _require_gpu()
    if storage == "fp32" and tile[1] == 8:
        pytest.skip("256-cell segments are 16-bit storage's")
    c = case("long_channel")
    L = make_solver(c, storage=storage, crop=nx, tile=tile, column=False)
    rng = np.random.default_rng(nx)
    f = L.populations().reshape(19, L.nz, L.ny, nx)
    fluid = ~c.solid[..., :nx]
    f = np.where(fluid, f * (1 + 0.02 * rng.standard_normal(f.shape)), f).astype(np.float32)
    L.load_populations(pitched(L, f))
    o = make_oracle(c, crop=nx)
    o.f[:] = L.populations()                  # as stored
    L.step(1)
    o.step(1)
    got, want = (a.reshape(19, L.nz, L.ny, nx) for a in (L.populations(), o.f))
    bar = np.full(want.shape, 2.0 ** -20)
    if storage == "fp16":
        dev = 2.0 ** -11 * np.abs(want - W[:, None, None, None])
        bar += dev
        if (nx - 1) % (64 if tile[1] == 2 else 128) == 0:
            dg = dev[..., -2]
            bar[..., -1] += dg + W[:, None, None] * dg.sum(0, keepdims=True)
    assert (np.abs(got - want) <= bar)[:, fluid].all(), float((np.abs(got - want) / bar)[:, fluid].max())
