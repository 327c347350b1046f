"""Performance cases of the solver: what its users have it do, over the sizes they have it do it at.

    listed()             the cases, from the 0.1M-cell test channel to the 36M-cell benchmark reach
    draw(rng)            one more case of the same kinds and ranges
    prepare(case, seed)  what a program holds before the call (solver, batch, network, inputs)
    run(state)           one pass through the public entry points, and its outputs
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the same outputs in float64, in plain torch

Kinds of case:
    solve      LBM3D.step(20): the 20-step chunk between two field outputs that every run is made
               of (column-mean wall model, inlet, outlet, one hull, one propeller disk)
    batch      BatchRun.advance(20): several boat cases of uneven sizes together
    open       LBM3D(...): flags, work lists and start state of a new case from device arrays
    readouts   LBM3D.profile_sums and LBM3D.body_forces at the end of an averaging window
    predict    SurrogateNet.forward: the warm start's network on a coarse grid
    train      SurrogateNet.loss_and_grad: one training step's forward and backward
    solve64    Solver64.step(20): the float64 runs behind the accuracy statements

The channels are trapezoids with a bumpy bed, one tapered hull under the lid and one propeller
disk behind it, as the benchmark reach is; the start state is the 1/7-power profile with seeded
velocity and pressure fluctuations of a few per cent to ten per cent, as in a developed flow.
"""
import math

import numpy as np
import torch

from water_flow_simulation_b200.batch import BatchRun
from water_flow_simulation_b200.fp64 import Solver64
from water_flow_simulation_b200.geometry import Section
from water_flow_simulation_b200.lbm3d import LBM3D
from water_flow_simulation_b200.reach3d import Fleet, Reach, ReachConfig, boat_type
from water_flow_simulation_b200.surrogate import SurrogateNet

STEPS = 20                     # steps between two field outputs (Run3D.avg_every)
TAU0, DX, DT = 0.5006, 0.1, 0.00625        # vel = DX / DT = 16: lattice <-> m/s is exact
STORE_SCALE = 2.0 ** 14        # LBM3D's default 16-bit storage scale
U_MEAN = 0.08                  # mean lattice speed

# D3Q19: velocities, weights, opposite direction and reflection in the rigid lid
C = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1),
     (1, 1, 0), (-1, -1, 0), (1, -1, 0), (-1, 1, 0), (1, 0, 1), (-1, 0, -1), (1, 0, -1), (-1, 0, 1),
     (0, 1, 1), (0, -1, -1), (0, 1, -1), (0, -1, 1)]
W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
OPP = [C.index((-x, -y, -z)) for x, y, z in C]
LID = [C.index((x, y, -z)) for x, y, z in C]

# the warm start's network (surrogate.py): layer, channels in, channels out, ReLU
NET = [("c1", 8, 64, True), ("c2", 64, 128, True), ("c3", 128, 128, True), ("c4", 128, 64, True),
       ("c5", 64, 64, True), ("c6", 64, 8, False)]


# ------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the small test channel, 192 x 50 x 12 (0.1M cells): launches and latency count
        {"name": "channel_fp32", "kind": "solve", "storage": "fp32", "nx": 192, "ny": 50, "nz": 12, "bank": 0.0,
         "average": False},
        # a small boat test at odd sizes in 16-bit storage, inside its averaging window
        {"name": "ragged_fp16", "kind": "solve", "storage": "fp16", "nx": 333, "ny": 61, "nz": 17, "bank": 1.0,
         "average": True},
        # ensemble-sized reaches in their averaging window (the trailing 40 % of every run)
        {"name": "reach3m_fp16_avg", "kind": "solve", "storage": "fp16", "nx": 577, "ny": 203, "nz": 25, "bank": 2.0,
         "average": True},
        {"name": "reach8m_fp32_avg", "kind": "solve", "storage": "fp32", "nx": 701, "ny": 305, "nz": 37, "bank": 1.0,
         "average": True},
        # the benchmark reach, 1500 x 602 x 40 = 36.1M cells, in both storages
        {"name": "reach36m_fp32", "kind": "solve", "storage": "fp32", "nx": 1500, "ny": 602, "nz": 40, "bank": 2.0,
         "average": False},
        {"name": "reach36m_fp16", "kind": "solve", "storage": "fp16", "nx": 1500, "ny": 602, "nz": 40, "bank": 2.0,
         "average": False},
        # a batch of boat cases of uneven sizes, as the boat tests run
        {"name": "batch5", "kind": "batch", "count": 5, "nx": 480, "ny": 150, "nz": 24, "bank": 1.0},
        # opening a case: what every new solver object pays before its first step
        {"name": "open_36m", "kind": "open", "storage": "fp16", "nx": 1500, "ny": 602, "nz": 40, "bank": 2.0},
        # the readouts of a finished run
        {"name": "readouts_8m", "kind": "readouts", "storage": "fp16", "nx": 701, "ny": 305, "nz": 37, "bank": 1.0},
        # the warm start's prediction for an 8M-cell case (voxels of 4 x 4 x 4 cells)
        {"name": "predict_120k", "kind": "predict", "Z": 10, "Y": 80, "X": 150},
        # one training step on a case of about 0.8M cells
        {"name": "train_12k", "kind": "train", "Z": 6, "Y": 32, "X": 64},
        # the float64 run of a 2.3M-cell case
        {"name": "solve64_2m", "kind": "solve64", "nx": 701, "ny": 101, "nz": 33, "bank": 1.0},
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def box(most):
        """Sizes of a reach of at most `most` cells: any residue of nx, ny and nz."""
        nz = log(8, 44)
        ny = log(max(32, nz + 8), 640)
        nx = log(80, 1536)
        while nx * ny * nz > most:
            nx, ny = max(72, int(nx * 0.83)), max(nz + 9, int(ny * 0.89))
        return {"nx": nx, "ny": ny, "nz": nz, "bank": rng.choice([0.0, 1.0, 2.0]) if ny > 5 * nz else 0.0}

    kind = rng.choice(["solve", "solve", "solve", "solve", "batch", "open", "readouts", "predict", "train", "solve64"])
    if kind == "solve":
        return {"kind": kind, "storage": rng.choice(["fp32", "fp16"]), **box(30_000_000), "average": rng.random() < 0.4}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(2, 6), **box(3_000_000)}
    if kind in ("open", "readouts"):
        return {"kind": kind, "storage": rng.choice(["fp32", "fp16"]), **box(30_000_000 if kind == "open" else 12_000_000)}
    if kind == "solve64":
        return {"kind": kind, **box(4_000_000)}
    big = kind == "predict"
    return {"kind": kind, "Z": 2 * rng.randint(1, 6), "Y": 2 * log(4, 40 if big else 20), "X": 2 * log(10, 100 if big else 40)}


# ------------------------------------------------------------------------------ channels
def _lid_padded(solid):
    """`solid` with the walls round it: bed below, walls on both sides in y, no wall past the x
    ends, and above the lid the top layer again (a mover through the lid comes from the layer
    it is in)."""
    p = torch.nn.functional.pad(solid, (1, 1, 1, 1, 1, 1), value=False)
    p[-1, 1:-1, 1:-1] = solid[-1]
    p[0] = True
    p[:, 0] = True
    p[:, -1] = True
    p[:, :, 0] = False
    p[:, :, -1] = False
    return p


def _source(p, i):
    """The cells direction i is pulled from, of an array padded by one cell."""
    (x, y, z), (nz, ny, nx) = C[i], (n - 2 for n in p.shape)
    return p[1 - z:1 - z + nz, 1 - y:1 - y + ny, 1 - x:1 - x + nx]


def channel(case):
    """Geometry, forces, inlet and wall friction of a case, on the GPU."""
    dev = torch.device("cuda")
    nx, ny, nz, bank = case["nx"], case["ny"], case["nz"], case["bank"]
    x = torch.arange(nx, device=dev, dtype=torch.float32)
    y = (torch.arange(ny, device=dev, dtype=torch.float32) - (ny - 1) / 2).abs()
    z = torch.arange(nz, device=dev, dtype=torch.float32)
    flat = ny / 2 - 1 - bank * nz
    zb = ((y - flat) / bank).clamp(min=0) if bank > 0 else torch.zeros_like(y)
    yy = torch.arange(ny, device=dev, dtype=torch.float32)[:, None]
    # bed bumps of 0.04 depths rms and 50 cells' correlation length, as the benchmark reach has
    bumps = sum(torch.cos((x * a + yy * b) / 50 + p)
                for a, b, p in ((0.9, 0.3, 0.4), (-0.4, 0.8, 1.9), (0.2, -0.7, 4.1), (1.1, 0.1, 2.6)))
    zb = zb[:, None] + 0.04 * nz * 0.7 * bumps.clamp(min=-1.0)
    bed = (z[:, None, None] + 0.5 < zb) | (y > ny / 2 - 1)[None, :, None]
    # a hull of a third of the depth under the lid, its bow tapered over the first quarter
    x0, length, width, draft = int(0.27 * nx), max(8, int(0.133 * nx)), max(4, int(0.1 * ny)), max(2, int(0.375 * nz))
    half = 0.5 * width * ((x - x0) / (0.25 * length)).clamp(0.3, 1.0)
    hull = ((x >= x0) & (x < x0 + length))[None, :] & (y[:, None] <= half)
    hull = (z >= nz - draft)[:, None, None] & hull & ~bed
    solid = bed | hull
    # a propeller disk behind the stern: four cells thick, tilted down a little
    d, xs = max(3, int(0.3 * nz)), x0 + length + 4
    disk = ((x >= xs) & (x < xs + 4))[None, None, :] & (y < 0.6 * d)[None, :, None] & \
        ((z >= nz - draft - d / 2) & (z < nz - draft + d / 2))[:, None, None] & ~solid
    fx, fy, fz = (disk.float() * s for s in (4e-5, 0.0, -6e-6))
    # inlet: 1/7-power profile over the water column of the first x station
    depth = (nz - zb[:, 0]).clamp(min=1.0)
    uin = 1.14 * U_MEAN * ((z[:, None] + 0.5 - zb[:, 0]) / depth).clamp(0, 1) ** (1 / 7)
    uin = torch.where(solid[:, :, 0], torch.zeros_like(uin), uin)
    # wall friction: Manning on bed and banks, the log law on the hull
    pb = _lid_padded(bed)
    ph = torch.nn.functional.pad(hull, (1, 1, 1, 1, 1, 1), value=False)
    ph[-1, 1:-1, 1:-1] = hull[-1]
    bedwall, hullwall = torch.zeros_like(solid), torch.zeros_like(solid)
    for i in range(1, 19):
        bedwall |= _source(pb, i)
        hullwall |= _source(ph, i)
    bedwall &= ~solid
    hullwall &= ~solid
    for a in (bedwall, hullwall):
        a[:, :, :2] = False
        a[:, :, -2:] = False
    cf = torch.where(bedwall, 0.0036, torch.where(hullwall, 0.0052, 0.0)).float()
    return {"solid": solid, "hull": hull, "F": (fx, fy, fz), "uin": uin, "cf": cf, "bedwall": bedwall}


def start_state(case, ch, seed):
    """Float32 (rho, ux, uy, uz) of a developed-looking flow: the inlet profile along the reach
    and seeded waves of 16 to 200 cells in each velocity component and in the pressure."""
    g = torch.Generator().manual_seed(seed)
    dev = ch["solid"].device
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ax = [torch.arange(n, device=dev, dtype=torch.float32) for n in (nz, ny, nx)]
    fluid = ~ch["solid"]

    def waves(amplitude):
        out = torch.zeros(nz, ny, nx, device=dev)
        for a in torch.rand(4, 5, generator=g).tolist():
            k = 2 * math.pi / (16 * 12.5 ** a[0])
            th, ph = 2 * math.pi * a[1], math.acos(2 * a[2] - 1)
            kx, ky, kz = (k * v for v in (math.cos(th) * math.sin(ph), math.sin(th) * math.sin(ph), math.cos(ph)))
            arg = (kz * ax[0])[:, None, None] + (ky * ax[1])[:, None] + kx * ax[2] + 2 * math.pi * a[3]
            out += torch.cos(arg) * (amplitude * (0.5 + a[4]))
        return out * fluid
    ux = ch["uin"][:, :, None] * fluid + waves(0.006)
    return 1.0 + waves(3e-4), ux, waves(0.006), waves(0.006)


def equilibrium(i, r, ux, uy, uz):
    cu = 3 * (C[i][0] * ux + C[i][1] * uy + C[i][2] * uz)
    return W[i] * r * (1 + cu + 0.5 * cu * cu - 1.5 * (ux * ux + uy * uy + uz * uz))


def start_populations(case, ch, seed, pitch):
    """Float32 start populations (19, nz, ny, pitch), at rest in solid and padding cells."""
    s = start_state(case, ch, seed)
    f = torch.empty(19, case["nz"], case["ny"], pitch, device=s[0].device)
    for i in range(19):
        f[i, :, :, :case["nx"]] = torch.where(ch["solid"], W[i], equilibrium(i, *s))
        f[i, :, :, case["nx"]:] = W[i]
    return f


def _cs(case):
    return 0.17


def solver(case, ch):
    return LBM3D(torch.device("cuda"), ch["solid"], *ch["F"], ch["uin"], TAU0, _cs(case), ch["cf"],
                 bedwall=ch["bedwall"], uref_mode="column", storage=case.get("storage", "fp16"))


def batch_cases(case):
    """The members of a batch: sizes from 0.4 to 1 times the case's, along and across."""
    out = []
    for k in range(case["count"]):
        s, t = 1 - 0.6 * ((k * 0.618) % 1), 1 - 0.3 * ((k * 0.381) % 1)
        out.append({"nx": max(72, int(case["nx"] * s)), "ny": max(int(case["ny"] * t), case["nz"] + 9),
                    "nz": case["nz"], "bank": case["bank"]})
    return out


def reach(case, ch):
    """A Reach around a channel's arrays, averaging from its first step on."""
    cfg = ReachConfig(length=case["nx"] * DX, dx=DX, cs=_cs(case), avg_frac=1.0)
    uin = ch["uin"].double().cpu().numpy() * (DX / DT)
    return Reach(sec=Section(B=case["ny"] * DX, Hb=case["nz"] * DX, z=0.0, Bf=0.0, n=0.025), cfg=cfg,
                 fleet=Fleet(boat_type("tug"), enabled=False), h=case["nz"] * DX, Q=1.0, S=3e-4, dx=DX, dt=DT,
                 nx=case["nx"], ny=case["ny"], nz=case["nz"], y=None, zc=None, solid=ch["solid"], uin_phys=uin,
                 Fx=ch["F"][0], Fy=ch["F"][1], Fz=ch["F"][2], cf=ch["cf"], bedwall=ch["bedwall"],
                 V=U_MEAN * DX / DT)


# ------------------------------------------------------------------------------ the network
def network_inputs(case, seed):
    """Weights (as a trained net's scale), input features, target and mask of one case."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    V = case["Z"] * case["Y"] * case["X"]
    weights = {}
    for name, cin, cout, relu in NET:
        sd = math.sqrt((2.0 if relu else 0.5) / (27 * cin))
        weights[name] = {"W": torch.randn(cout, 27 * cin, generator=g, device="cuda") * sd,
                         "b": torch.randn(cout, generator=g, device="cuda") * 0.02}
    x = torch.randn(V, 8, generator=g, device="cuda") * 0.6
    x[:, 0] = (x[:, 0] > -0.5).float()                          # fluid fraction
    x[:, 1:4] *= (torch.rand(V, 1, generator=g, device="cuda") < 0.02)     # forces in few voxels
    target = torch.randn(V, 4, generator=g, device="cuda") * 0.3
    mask = (torch.rand(V, generator=g, device="cuda") < 0.8).float()
    return weights, x, target, mask


# ------------------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("predict", "train"):
        weights, x, target, mask = network_inputs(case, seed)
        net = SurrogateNet()
        net.load_state(weights)
        return {"kind": kind, "net": net, "x": x, "dims": (case["Z"], case["Y"], case["X"]), "target": target,
                "mask": mask}
    if kind == "batch":
        parts = batch_cases(case)
        chs = [channel(c) for c in parts]
        batch = BatchRun([reach(c, ch) for c, ch in zip(parts, chs)], max_steps=10 ** 9)
        for k, (c, ch, r) in enumerate(zip(parts, chs, batch.runs)):
            r.lbm.load_populations(start_populations(c, ch, seed + 1000 * k, r.lbm.pitch).reshape(-1))
        return {"kind": kind, "batch": batch}
    ch = channel(case)
    if kind == "open":
        # another case of the family: the inlet's speed differs from case to case
        ch["uin"] = ch["uin"] * _inlet_factor(seed)
        return {"kind": kind, "case": case, "channel": ch}
    if kind == "solve64":
        host = {k: v.cpu().numpy() for k, v in ch.items() if k != "F"}
        host["F"] = [a.cpu().numpy() for a in ch["F"]]
        r = reach(case, {**host, "uin": ch["uin"]})
        s = Solver64(r)
        s.f.copy_(start_populations(case, ch, seed, case["nx"]).reshape(-1))
        s.f2.copy_(s.f)
        return {"kind": kind, "solver": s}
    L = solver(case, ch)
    L.load_populations(start_populations(case, ch, seed, L.pitch).reshape(-1))
    if kind == "readouts":
        L.step(1, accumulate=True)
        return {"kind": kind, "solver": L, "body": ch["hull"].to(torch.uint8)}
    return {"kind": kind, "solver": L, "average": case["average"]}


def _inlet_factor(seed):
    return 0.8 + 0.4 * torch.rand(1, generator=torch.Generator().manual_seed(seed)).item()


def _fields(L, average):
    out = {"f": L.f, "rho": L.rho, "ux": L.ux, "uy": L.uy, "uz": L.uz}
    if average:
        out.update({"sum_" + k: L.avg_sum(k) for k in ("ux", "rho", "sp")})
    return out


def run(state):
    kind = state["kind"]
    if kind == "solve":
        L = state["solver"]
        L.step(STEPS, accumulate=state["average"])
        return _fields(L, state["average"])
    if kind == "batch":
        state["batch"].advance(STEPS)
        return [_fields(r.lbm, True) for r in state["batch"].runs]
    if kind == "open":
        L = solver(state["case"], state["channel"])
        return {"f": L.f, "flags": L.flags}
    if kind == "readouts":
        L = state["solver"]
        forces, applied = L.body_forces(state["body"], 1)
        return {"profiles": L.profile_sums(mean=True), "forces": forces, "applied": applied}
    if kind == "solve64":
        s = state["solver"]
        s.step(STEPS)
        return {"f": s.f, "rho": s.rho, "ux": s.ux, "uy": s.uy, "uz": s.uz}
    net = state["net"]
    if kind == "predict":
        return net.forward(state["x"], state["dims"])
    net.zero_grad()
    loss, out = net.loss_and_grad(state["x"], state["dims"], state["target"], state["mask"])
    return {"loss": loss, "out": out, **{n + k: net.p[n][k] for n, _, _, _ in NET for k in ("dW", "db")}}


# ------------------------------------------------------------------------------ work
def work(case):
    kind = case["kind"]
    if kind in ("predict", "train"):
        V = case["Z"] * case["Y"] * case["X"]
        voxels = {"c1": V, "c2": V // 8, "c3": V // 8, "c4": V // 8, "c5": V, "c6": V}
        flops = sum(2 * 27 * cin * cout * voxels[n] for n, cin, cout, _ in NET)
        weights = sum(27 * cin * cout + cout for _, cin, cout, _ in NET)
        if kind == "predict":
            return {"bytes": V * 8 * 4 * 2 + weights * 2, "flops": flops}
        # backward: the weights' gradients, and the inputs' of every layer but the first
        back = 2 * flops - 2 * 27 * 8 * 64 * V
        return {"bytes": V * (8 * 4 * 2 + 5 * 4) + weights * (2 + 4), "flops": flops + back}
    parts = batch_cases(case) if kind == "batch" else [case]
    cells = sum(c["nx"] * c["ny"] * c["nz"] for c in parts)
    fluid = sum(int((~channel(c)["solid"]).sum()) for c in parts)
    if kind == "open":       # masks, forces, friction in; flags and both population buffers out
        return {"bytes": cells * (2 + 16 + 4 + 2 * 19 * (4 if case["storage"] == "fp32" else 2)), "flops": 19 * 8 * cells}
    if kind == "readouts":   # flags and four averages of every cell, populations of the hull's walls
        return {"bytes": cells * 4 + fluid * 16, "flops": fluid * 12}
    width = {"solve": 4 if case.get("storage") == "fp32" else 2, "batch": 2, "solve64": 8}[kind]
    fields = 4 * (8 if kind == "solve64" else 4) + (48 if kind == "batch" or case.get("average") else 0)
    return {"bytes": STEPS * fluid * 2 * 19 * width + cells * fields, "flops": STEPS * fluid * 250}


# ------------------------------------------------------------------------------ float64
def _wall_function(f, mask, idx, cf, u, rho):
    """Moving-wall bounce-back at the cells `idx` (flat): the slip velocity along the wall that
    makes the momentum given to the wall the shear rho cf U^2, U the cell's own speed along it."""
    wall = [mask[i].reshape(-1)[idx] for i in range(19)]
    c = torch.tensor(C, dtype=torch.float64, device=idx.device)
    wm = torch.stack(wall).double()
    n = -(c.T @ wm)
    face = torch.stack([wm[1] + wm[2], wm[3] + wm[4], wm[5] + wm[6]])
    nn, area = n.norm(dim=0), face.norm(dim=0)
    e = n / nn.clamp(min=1e-30)
    p = torch.stack([a.reshape(-1)[idx] for a in u])
    t = p - (p * e).sum(0) * e
    ut = t.norm(dim=0)
    ok = (nn > 0) & (area > 0) & (ut > 1e-7)
    t = t / ut.clamp(min=1e-30)
    ct = c @ t
    fw = torch.stack([f[i].reshape(-1)[idx] for i in range(19)])
    w = torch.tensor(W, dtype=torch.float64, device=idx.device)[:, None]
    D, K = (ct * fw * wm).sum(0), (w * ct * ct * wm).sum(0)
    ok &= K > 0
    r = rho.reshape(-1)[idx]
    us = (-2 * D - r * cf.reshape(-1)[idx] * ut * ut * area) / (6 * r * K.clamp(min=1e-30))
    us = torch.where(ok, torch.minimum(torch.maximum(us, -ut), ut), torch.zeros_like(us))
    for i in range(1, 19):
        f[i].view(-1)[idx] += 6 * W[i] * r * ct[i] * us * wm[i]


def solve_exact(case, ch, f, steps):
    """`steps` lattice steps in float64 from populations f (19, nz, ny, nx): pull with bounce-back
    and the rigid lid, wall function, regularized collision with the Smagorinsky relaxation time
    and forcing, then inlet and outlet.  Returns (f, rho, ux, uy, uz)."""
    solid, dev = ch["solid"], ch["solid"].device
    F = [a.double() for a in ch["F"]]
    cf, uin = ch["cf"].double(), ch["uin"].double()
    padded = _lid_padded(solid)
    mask = [_source(padded, i) & ~solid for i in range(19)]
    walls = torch.zeros_like(solid)
    for m in mask[1:]:
        walls |= m
    idx = torch.nonzero((walls & (cf > 0)).reshape(-1)).squeeze(1)
    rho, u = torch.ones(solid.shape, dtype=torch.float64, device=dev), [torch.zeros(solid.shape, dtype=torch.float64, device=dev) for _ in range(3)]
    inlet, outlet = ~(solid[:, :, 0] | solid[:, :, 1]), ~(solid[:, :, -1] | solid[:, :, -2])
    csmag2 = _cs(case) ** 2
    for _ in range(steps):
        g = torch.empty_like(f)
        for i, (x, y, z) in enumerate(C):
            torch.where(mask[i], f[OPP[i]], torch.roll(f[i], (z, y, x), (0, 1, 2)), out=g[i])
            if z == -1:
                g[i, -1] = torch.where(mask[i][-1], f[OPP[i], -1], torch.roll(f[LID[i], -1], (y, x), (0, 1)))
            if x:
                e = 0 if x == 1 else -1
                g[i, :, :, e] = f[i, :, :, e]
        _wall_function(g, mask, idx, cf, u, rho)
        rho = g.sum(0)
        u = []
        for a in range(3):
            j = 0.5 * F[a]
            for i in range(1, 19):
                if C[i][a]:
                    j = j + C[i][a] * g[i]
            u.append(j / rho)
        P = {}
        for a in range(3):
            for b in range(a, 3):
                s = -rho * u[a] * u[b]
                if a == b:
                    s -= rho / 3
                for i in range(1, 19):
                    if C[i][a] * C[i][b]:
                        s += C[i][a] * C[i][b] * g[i]
                P[a, b] = s
        qn = sum((1 if a == b else 2) * s * s for (a, b), s in P.items()).sqrt_()
        om = 2 / (TAU0 + (TAU0 ** 2 + 18 * 1.41421356 * csmag2 * qn / rho).sqrt_())
        del qn
        sf = 1 - 0.5 * om
        uF = sum(u[a] * F[a] for a in range(3))
        trace = (P[0, 0] + P[1, 1] + P[2, 2]) / 3
        for i, c in enumerate(C):
            pi, cu, cF = -trace, 0.0, 0.0
            for a in range(3):
                if c[a]:
                    cu, cF = cu + c[a] * u[a], cF + c[a] * F[a]
                for b in range(a, 3):
                    if c[a] * c[b]:
                        pi = pi + (1 if a == b else 2) * c[a] * c[b] * P[a, b]
            f[i] = equilibrium(i, rho, *u) + (1 - om) * W[i] * (4.5 * pi - 1.5 * cF) \
                + sf * W[i] * (3 * (cF - uF) + 9 * cu * cF)
        del g
        for e, n, open_, at_inlet in ((0, 1, inlet, True), (-1, -2, outlet, False)):
            gn = f[:, :, :, n].clone()
            r = gn.sum(0)
            v = [sum(C[i][a] * gn[i] for i in range(19)) / r for a in range(3)]
            zero = torch.zeros_like(r)
            rb, vb = (r, [uin, zero, zero]) if at_inlet else (torch.ones_like(r), v)
            for i in range(19):
                b = equilibrium(i, rb, *vb) + gn[i] - equilibrium(i, r, *v)
                f[i, :, :, e] = torch.where(open_, b, f[i, :, :, e])
        for i in range(19):
            f[i][solid] = W[i]
        rho[solid] = 1.0
        for a in range(3):
            u[a][solid] = 0.0
    return f, rho, *u


def _stored(case, f, storage):
    """Float64 populations as the solver's `f` holds them: rows padded to the storage's pitch, and
    16-bit storage's scaled deviations from the lattice weights."""
    align = {"fp32": 4, "fp16": 8}[storage]
    pitch = -(-case["nx"] // align) * align
    out = torch.empty(19, case["nz"], case["ny"], pitch, dtype=torch.float64, device=f.device)
    for i in range(19):
        out[i, :, :, :case["nx"]] = f[i]
        out[i, :, :, case["nx"]:] = W[i]
        if storage == "fp16":
            out[i] = (out[i] - W[i]) * STORE_SCALE
    return out.reshape(-1)


def _exact_fields(case, ch, seed, storage, steps, average):
    f = start_populations(case, ch, seed, case["nx"])
    if storage == "fp16":
        for i in range(19):
            w = torch.tensor(W[i], dtype=torch.float32).item()
            f[i] = w + ((f[i] - w) * STORE_SCALE).half().float() / STORE_SCALE
    f, rho, ux, uy, uz = solve_exact(case, ch, f.double(), steps)
    out = {"rho": rho.reshape(-1), "ux": ux.reshape(-1), "uy": uy.reshape(-1), "uz": uz.reshape(-1)}
    if average:
        out.update({"sum_ux": out["ux"], "sum_rho": out["rho"],
                    "sum_sp": (ux * ux + uy * uy + uz * uz).sqrt_().reshape(-1)})
    out["f"] = _stored(case, f, storage) if storage else f.reshape(-1)
    return out


def _exact_network(case, seed):
    weights, x, target, mask = network_inputs(case, seed)
    Z, Y, X = case["Z"], case["Y"], case["X"]
    p = {n: (w["W"].bfloat16().double().requires_grad_(case["kind"] == "train"),
             w["b"].double().requires_grad_(case["kind"] == "train")) for n, w in weights.items()}

    def conv(name, a):
        _, cin, cout, relu = next(layer for layer in NET if layer[0] == name)
        Wn, b = p[name]
        z, y, x_, _ = a.shape
        a = torch.nn.functional.pad(a, (0, 0, 1, 1, 1, 1, 1, 1))
        out = b
        for t in range(27):
            k, j, i = t // 9, t // 3 % 3, t % 3
            out = out + a[k:k + z, j:j + y, i:i + x_].reshape(-1, cin) @ Wn[:, t * cin:(t + 1) * cin].T
        out = out.reshape(z, y, x_, cout)
        return out.relu() if relu else out

    a1 = conv("c1", x.bfloat16().double().reshape(Z, Y, X, 8))
    h = a1.reshape(Z // 2, 2, Y // 2, 2, X // 2, 2, 64).mean(dim=(1, 3, 5))
    h = conv("c4", conv("c3", conv("c2", h)))
    up = h[:, None, :, None, :, None].expand(-1, 2, -1, 2, -1, 2, -1).reshape(Z, Y, X, 64)
    out = conv("c6", conv("c5", up + a1)).reshape(-1, 8)
    if case["kind"] == "predict":
        return out
    loss = (mask.double()[:, None] * (out[:, :4] - target.double()) ** 2).sum() / mask.double().sum()
    loss.backward()
    res = {"loss": loss.detach().reshape(1), "out": out.detach()}
    for n in p:
        res[n + "dW"], res[n + "db"] = p[n][0].grad, p[n][1].grad
    return res


def exact(case, seed):
    kind = case["kind"]
    if kind in ("predict", "train"):
        return _exact_network(case, seed)
    if kind == "batch":
        return [_exact_fields(c, channel(c), seed + 1000 * k, "fp16", STEPS, True)
                for k, c in enumerate(batch_cases(case))]
    ch = channel(case)
    if kind == "solve":
        return _exact_fields(case, ch, seed, case["storage"], STEPS, case["average"])
    if kind == "solve64":
        return _exact_fields(case, ch, seed, None, STEPS, False)
    if kind == "open":
        u = (ch["uin"] * _inlet_factor(seed)).double()[:, :, None] * ~ch["solid"]
        f = torch.stack([equilibrium(i, 1.0, u, torch.zeros_like(u), torch.zeros_like(u)) for i in range(19)])
        return {"f": _stored(case, f, case["storage"]), "flags": None}
    # readouts: one accumulated output, then sums over each cross-section; a speed above the bed
    e = _exact_fields(case, ch, seed, case["storage"], 1, True)
    shape, fluid = ch["solid"].shape, (~ch["solid"]).double()
    rho, ux, sp = (e[k].reshape(shape) for k in ("rho", "ux", "sum_sp"))
    above = fluid.bool() & torch.cat([torch.ones_like(ch["solid"][:1]), ch["solid"][:-1]])
    sums = {"q": ux * fluid, "uxx": ux * ux * fluid, "drho": (rho - 1) * fluid, "mass": rho * fluid, "n_fluid": fluid}
    top = {"top_n": fluid, "top_drho": (rho - 1) * fluid, "top_ux": ux * fluid}
    prof = {k: v.sum(dim=(0, 1)) for k, v in sums.items()}
    prof.update({k: v[-1].sum(dim=0) for k, v in top.items()})
    prof["umax"] = (sp * fluid).amax(dim=(0, 1))
    prof["bed_speed2"] = (sp * sp * above).amax(dim=0)
    return {"profiles": {k: np.asarray(v.cpu()) for k, v in prof.items()}, "forces": None, "applied": None}
