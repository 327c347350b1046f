"""Float64 readouts at the edges of their chunks (needs a B200): columns per chunk, layers read
ahead, x remainders, quads of flags; against float64 NumPy and the oracle's force sum.

Tolerances: a float64 sum of n terms in any order is within n 2^-53 sum|terms| of any other; maxima
are exact, but for the speed of instantaneous fields (three products, two sums, a square root: 8 ulp).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _solver(nx, ny, nz, seed, storage="fp32"):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    from water_flow_simulation_b200.lbm3d import LBM3D
    rng = np.random.default_rng(seed)
    solid = rng.random((nz, ny, nx)) < 0.25
    F = [(rng.random(solid.shape) < 0.1) * rng.normal(size=solid.shape).astype(np.float32) for _ in range(3)]
    F = [np.where(solid, 0, a).astype(np.float32) for a in F]
    L = LBM3D(torch.device("cuda"), solid, *F, np.zeros((nz, ny), np.float32), 0.6, 0.17, storage=storage)
    return L, solid, F, rng


@pytest.mark.parametrize("mean", (False, True))
@pytest.mark.parametrize("nx,ny,nz", ((4, 1, 1), (33, 5, 3), (130, 300, 5), (128, 257, 4), (257, 31, 9)))
def test_profile_sums(nx, ny, nz, mean):
    import torch
    L, solid, _, rng = _solver(nx, ny, nz, nx + ny)
    fl = ~solid
    names = ("ux", "uy", "uz", "rho", "sp", "uxx")
    v = {k: rng.normal(size=solid.shape).astype(np.float32) + (1 if k == "rho" else 0) for k in names}
    v["sp"] = np.abs(v["sp"])
    if mean:
        L.enable_averaging()
        avg = L._avg.view(6, nz, ny, L.pitch)
        for i, k in enumerate(names):
            avg[i, ..., :nx].copy_(torch.as_tensor(v[k], device=L.device))
        L.navg = 3
        d = {k: a.astype(np.float64) * (1.0 / 3) for k, a in v.items()}
    else:
        for k in ("ux", "uy", "uz", "rho"):
            getattr(L, "_" + k).view(nz, ny, L.pitch)[..., :nx].copy_(torch.as_tensor(v[k], device=L.device))
        d = {k: a.astype(np.float64) for k, a in v.items()}
        d["sp"] = np.sqrt(d["ux"] ** 2 + d["uy"] ** 2 + d["uz"] ** 2)
        d["uxx"] = d["ux"] ** 2
    s = L.profile_sums(mean=mean)
    terms = {"q": d["ux"], "uxx": d["uxx"], "drho": d["rho"] - 1, "mass": d["rho"], "n_fluid": np.ones(solid.shape)}
    for k, t in terms.items():
        tol = (ny * nz + 2) * EPS * (np.abs(t) * fl).sum(axis=(0, 1))
        assert np.all(np.abs(s[k] - (t * fl).sum(axis=(0, 1))) <= tol), k
    for k, t in (("top_n", "n_fluid"), ("top_drho", "drho"), ("top_ux", "q")):
        tol = (ny + 2) * EPS * (np.abs(terms[t]) * fl)[-1].sum(axis=0)
        assert np.all(np.abs(s[k] - (terms[t] * fl)[-1].sum(axis=0)) <= tol), k
    above = fl & np.concatenate([np.ones_like(solid[:1]), solid[:-1]])
    np.testing.assert_allclose(s["umax"], (d["sp"] * fl).max(axis=(0, 1)), rtol=0 if mean else 8 * EPS)
    np.testing.assert_allclose(s["bed_speed2"], (d["sp"] ** 2 * above).max(axis=0), rtol=0 if mean else 16 * EPS)


@pytest.mark.parametrize("storage", ("fp32", "fp16"))
@pytest.mark.parametrize("nx,ny,nz,nb", ((5, 4, 3, 1), (66, 9, 7, 3), (131, 40, 11, 16), (40, 12, 6, 0)))
def test_body_forces(nx, ny, nz, nb, storage):
    """Bounce-back without the wall function from random populations: every term is the same on both
    sides, so only the order of the float64 sums differs.  No body at all: the applied force alone."""
    import torch
    from oracle.oracle import OracleLBM, body_forces
    L, solid, F, rng = _solver(nx, ny, nz, nx, storage)
    body = (rng.integers(0, nb + 1, solid.shape) * solid).astype(np.uint8)
    f = L.f.view(19, nz, ny, L.pitch)
    f[..., :nx].copy_(torch.as_tensor(rng.random((19,) + solid.shape), device=L.device))
    got, applied = L.body_forces(body, nb)
    assert got.shape == (nb, 3)
    for a, b in zip(applied, F):
        assert abs(a - b.astype(np.float64).sum()) <= b.size * EPS * np.abs(b.astype(np.float64)).sum()
    if nb == 0:
        return
    o = OracleLBM(solid, *F, np.zeros((nz, ny), np.float32), 0.6, 0.17)
    w = np.array([1 / 3] + [1 / 18] * 6 + [1 / 36] * 12, np.float32).reshape(19, 1, 1, 1)
    pop = f[..., :nx].float().cpu().numpy()
    if storage == "fp16":
        pop = pop * np.float32(1 / L.store_scale) + w
    o.f = np.ascontiguousarray(pop.ravel())
    want = body_forces(o, body, nb)
    # float32 storage: the same terms.  16-bit: the device converts with one rounding, NumPy with two
    links = 18 * int((body > 0).sum())
    tol = links * 2 * float(np.abs(pop).max()) * (links * EPS if storage == "fp32" else 2.0 ** -23)
    assert float(np.abs(got - want).max()) <= tol
