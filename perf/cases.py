"""The work that users of this framework have it do, as cases that can be timed and compared.

Families (``kind``):

  * ``bar``      a boundary-value run advanced by ``Simulation.step`` and its fields read back: the
                 tensile bars of vpd/case.py and the lattice sizes of the archived case files, in
                 FP64, in mixed precision and with the learned return map, with and without damage;
  * ``setup``    the bond structure of a new body on device arrays: ``build_neighbor_list``, then
                 ``shape_tensor_inverse`` (what a host that drives the modules itself does first);
  * ``modules``  one increment of such a host through the module functions: F, material update,
                 bond damage, force density (``force_density`` or its variant without allocation);
  * ``points``   material points without bonds: ``material_update``, ``corotational_update`` or
                 ``jc_return_map``;
  * ``network``  the surrogate network: ``mlp_forward`` (inference) or ``mlp_gradients``;
  * ``train``    ``train_surrogate`` on increments that the device VUMAT solves.

``prepare`` makes what such a program holds before the call, from the seed alone; ``run`` is one
pass through the public entry points; ``exact`` gives the same outputs in 64-bit torch without the
package's code; ``work`` the bytes and operations a pass cannot do without.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vumat-pd_b200"))

import vpd  # noqa: E402
from vpd import case as vcase  # noqa: E402

DEV = "cuda"
RING = 16        # displacement fields of a driven load path, forth and back
STRAIN_STEP = 2.5e-3


def listed():
    return [
        # tensile_bar_1 (4,000 points, FP64): a parameter study's run, stepped in short chunks
        dict(name="bar_4k_fp64", kind="bar", nx=40, ny=10, nz=10, ratio=3.015, jitter=0.0, precision="fp64",
             guess="", damage=False, drive="ramp", grip=1.0, preload=2000, steps=32),
        # the lattice of the archived 10,605-point case files (half-cosine pull, horizon 3 h)
        dict(name="bar_10605_fp64", kind="bar", nx=101, ny=21, nz=5, ratio=3.0, jitter=0.0, precision="fp64",
             guess="", damage=False, drive="smooth", grip=0.0, preload=2500, steps=32),
        # a ragged cross-section at the long horizon, FP64 in plastic flow: the plain path at an
        # ordinary size
        dict(name="bar_154k_fp64", kind="bar", nx=97, ny=43, nz=37, ratio=4.015, jitter=0.05, precision="fp64",
             guess="", damage=False, drive="ramp", grip=5.0, preload=1200, steps=32),
        # tensile_bar_2 (500,000 points, critical stretch, mixed precision), before its first break
        dict(name="bar_500k_mixed_damage", kind="bar", nx=200, ny=50, nz=50, ratio=3.015, jitter=0.0,
             precision="mixed", guess="", damage=True, drive="ramp", grip=1.0, preload=200, steps=32),
        # tensile_bar_3 without damage (1,000,000 points) in plastic flow with the learned return
        # map: the benchmark's workload
        dict(name="bar_1M_surrogate", kind="bar", nx=400, ny=50, nz=50, ratio=4.015, jitter=0.05,
             precision="mixed", guess="hybrid", damage=False, drive="ramp", grip=5.0, preload=2000, steps=32),
        # the bond structure of a 250,000-point body
        dict(name="setup_250k", kind="setup", nx=100, ny=50, nz=50, ratio=4.015, jitter=0.05),
        # the smallest module-level call: a body of the size of the config-1 bar
        dict(name="modules_4k", kind="modules", nx=40, ny=10, nz=10, ratio=3.015, jitter=0.0, noalloc=True),
        # the same through the allocating force call, on a ragged body
        dict(name="modules_154k", kind="modules", nx=97, ny=43, nz=37, ratio=4.015, jitter=0.05, noalloc=False),
        # 500,000 material points on a load path in plastic flow
        dict(name="points_500k", kind="points", op="material", n=500_000),
        # network inference over the points of the large bar
        dict(name="network_1M", kind="network", op="forward", batch=1_000_000),
        # the gradient of one training batch
        dict(name="network_grad_8k", kind="network", op="gradients", batch=8192),
        # a short training run (60 Adam steps at the default batch)
        dict(name="train_131k", kind="train", samples=131_072, epochs=4, batch=8192),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _lattice(rng, lo, hi):
    """A box of about log-uniform lo..hi points, odd extents as likely as even ones."""
    n = _log_int(rng, lo, hi)
    nz = rng.randint(3, max(4, min(60, int(round((n / 4) ** (1 / 3))) + 3)))
    ny = rng.randint(4, max(5, min(60, int(round((n / (4 * nz)) ** 0.5)) + 4)))
    nx = max(9, int(round(n / (ny * nz))))
    return dict(nx=nx, ny=ny, nz=nz)


def draw(rng):
    kind = rng.choice(["bar", "bar", "bar", "setup", "modules", "modules", "points", "network", "train"])
    if kind == "bar":
        precision = rng.choice(["fp64", "mixed"])
        damage = rng.random() < 0.4
        guess = "hybrid" if precision == "mixed" and not damage and rng.random() < 0.5 else ""
        drive = rng.choice(["ramp", "smooth"]) if not damage else "ramp"
        grip = 0.0 if drive == "smooth" else 1.0 if damage else rng.choice([1.0, 5.0])
        return dict(kind=kind, ratio=rng.choice([3.0, 3.015, 4.015]), jitter=rng.choice([0.0, 0.05]),
                    precision=precision, guess=guess, damage=damage, drive=drive, grip=grip,
                    preload=rng.choice([200, 600]), steps=rng.choice([8, 13, 32]), **_lattice(rng, 1500, 250_000))
    if kind == "setup":
        return dict(kind=kind, ratio=rng.choice([3.0, 3.015, 4.015]), jitter=rng.choice([0.0, 0.05]),
                    **_lattice(rng, 1500, 250_000))
    if kind == "modules":
        c = dict(kind=kind, ratio=rng.choice([3.0, 3.015, 4.015]), jitter=rng.choice([0.0, 0.05]),
                 **_lattice(rng, 1500, 150_000))
        c["noalloc"] = c["nx"] * c["ny"] * c["nz"] <= 65536 and rng.random() < 0.5
        return c
    if kind == "points":
        return dict(kind=kind, op=rng.choice(["material", "corotational", "return_map"]), n=_log_int(rng, 1000, 500_000))
    if kind == "network":
        op = rng.choice(["forward", "gradients"])
        return dict(kind=kind, op=op, batch=_log_int(rng, 200, 1_000_000 if op == "forward" else 32768))
    return dict(kind=kind, samples=_log_int(rng, 16_000, 131_072), epochs=rng.randint(1, 4), batch=rng.choice([1000, 4096, 8192]))


# ------------------------------------------------------------------ bodies and inputs
SPACING = 0.1
PROPS = vcase.steel_props(1.0e6)
DT = vcase.stable_dt(SPACING, PROPS)


def _count(c):
    return c["nx"] * c["ny"] * c["nz"]


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _body(c, seed):
    """Jittered lattice positions [n,3] and boundary-halved volumes [n] as float64 CUDA tensors."""
    axes = [torch.arange(c[k], dtype=torch.float64, device=DEV) for k in ("nx", "ny", "nz")]
    g = torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
    pos = g * SPACING
    pos[:, 1] -= 0.5 * (c["ny"] - 1) * SPACING
    pos[:, 2] -= 0.5 * (c["nz"] - 1) * SPACING
    vol = torch.full((pos.shape[0],), SPACING ** 3, dtype=torch.float64, device=DEV)
    for d, k in enumerate(("nx", "ny", "nz")):
        vol = torch.where((g[:, d] == 0) | (g[:, d] == c[k] - 1), 0.5 * vol, vol)
    if c["jitter"]:
        r = torch.rand(pos.shape, generator=_gen(seed if c["kind"] == "bar" else 20261203), dtype=torch.float64, device=DEV)
        pos = pos + (2.0 * r - 1.0) * (c["jitter"] * SPACING)
    scale = _scale(c, seed)
    return (pos * scale).contiguous(), (vol * scale ** 3).contiguous()


def _scale(c, seed):
    """The size of a body that the modules run on (its bonds, and so the shapes of the outputs, do not depend on it)."""
    return 1.0 if c["kind"] == "bar" else float(np.random.RandomState(seed % (1 << 31)).uniform(0.8, 1.25))


def _bar_case(c, seed):
    """The vpd.Case of a bar: velocity-ramp grips (the bars of vpd/case.py) or a half-cosine pull (the archived files)."""
    factor = 1.0 + 0.05 * float(np.random.RandomState(seed % (1 << 31)).uniform(-1, 1))
    kw = dict(name="bar", nx=c["nx"], ny=c["ny"], nz=c["nz"], spacing=SPACING, horizon=c["ratio"] * SPACING, dt=DT,
              steps=10000, density=vcase.STEEL_DENSITY, props=PROPS, region_layers=3,
              precision=vcase.PRECISION_MIXED if c["precision"] == "mixed" else vcase.PRECISION_FP64,
              material_mode=vcase.MATERIAL_SURROGATE if c["guess"] else vcase.MATERIAL_VUMAT)
    if c["drive"] == "ramp":
        kw.update(bc_mode=vcase.BC_VELOCITY_RAMP, grip_velocity=factor * c["grip"], ramp_time=200 * DT)
    else:
        kw.update(bc_mode=vcase.BC_SMOOTH_DISPLACEMENT, amplitude=factor * 0.06 * (c["nx"] - 1) * SPACING,
                  rise_time=20000 * DT)
    if c["damage"]:
        kw.update(damage_mode=vcase.DAMAGE_CRITICAL_STRETCH, damage_initiation=0.02)
    return vcase.Case(**kw)


_network = []


def _weights():
    """A briefly trained network: what a program that runs the learned update has trained before."""
    if not _network:
        _network.extend(vpd.train_surrogate(PROPS, samples=131_072, epochs=4)[:2])
    return _network


def _load_path(pos, seed):
    """RING displacement fields of a growing, slightly uneven stretch with lateral contraction."""
    g = _gen(seed + 1)
    rate = 1.0 + 0.2 * (torch.rand(1, generator=g, dtype=torch.float64, device=DEV).item() - 0.5)
    wave = torch.rand(3, generator=g, dtype=torch.float64, device=DEV)
    length = pos.abs().amax(0).clamp_min(1e-9)
    bump = 0.05 * torch.sin(3.0 * (pos / length) + 6.28 * wave)
    shape = pos * torch.tensor([1.0, -0.35, -0.35], dtype=torch.float64, device=DEV) * (1.0 + bump)
    return [(rate * STRAIN_STEP * (k + 1) * shape).contiguous() for k in range(RING)]


def _path_index(k):
    """0, 1, .., RING-1, RING-2, .., 1, 0, 1, ..: loading and unloading in turn."""
    k %= 2 * RING - 2
    return k if k < RING else 2 * RING - 2 - k


def _material_state(n):
    eye = torch.eye(3, dtype=torch.float64, device=DEV).reshape(1, 9).repeat(n, 1).contiguous()
    zero = lambda w: torch.zeros((n, w), dtype=torch.float64, device=DEV)  # noqa: E731
    return dict(defgrad_old=eye, left_stretch=eye.clone(), rotation=eye.clone(), strain=zero(9),
                stress_corotational=zero(9), state=zero(6),
                temperature=torch.full((n,), 293.0, dtype=torch.float64, device=DEV),
                energy_internal=zero(1)[:, 0].contiguous(), energy_inelastic=zero(1)[:, 0].contiguous())


POINT_DT = 1.0e-3


def _point_fields(n, seed):
    """RING deformation gradients per point: a growing stretch in a point's own direction, slightly rotated."""
    g = _gen(seed)
    a = torch.randn((n, 3, 3), generator=g, dtype=torch.float64, device=DEV)
    a = a - torch.eye(3, dtype=torch.float64, device=DEV) * (a.diagonal(dim1=1, dim2=2).sum(1) / 3.0)[:, None, None]
    a = a / a.flatten(1).norm(dim=1).clamp_min(1e-9)[:, None, None]
    eye = torch.eye(3, dtype=torch.float64, device=DEV)
    return [(eye + STRAIN_STEP * (k + 1) * a).reshape(n, 9).contiguous() for k in range(RING)]


def _return_map_inputs(n, seed):
    g = _gen(seed)
    r = lambda *s: torch.rand(s, generator=g, dtype=torch.float64, device=DEV)  # noqa: E731
    inc = torch.randn((n, 6), generator=g, dtype=torch.float64, device=DEV) * (10.0 ** (-6.0 + 3.0 * r(n, 1)))
    eqps = 10.0 ** (-5.0 + 4.0 * r(n))
    oldy = PROPS[2] + PROPS[3] * eqps ** PROPS[5]
    s = torch.randn((n, 6), generator=g, dtype=torch.float64, device=DEV)
    m = s[:, :3].mean(1, keepdim=True)
    s[:, :3] -= m
    q = torch.sqrt(1.5 * ((s[:, :3] ** 2).sum(1) + 2.0 * (s[:, 3:] ** 2).sum(1)))
    s = s / q[:, None] * (oldy * (0.9 + 0.1 * r(n)))[:, None]
    st = torch.zeros((n, 6), dtype=torch.float64, device=DEV)
    st[:, 0], st[:, 1], st[:, 2], st[:, 3] = 1.0, eqps, 293.0 + 300.0 * r(n), oldy
    st[:, 4] = 1.0e-5 * r(n)
    return inc.contiguous(), s.contiguous(), st


def _network_inputs(c, seed):
    g = _gen(seed)
    shapes = [(128, 16, 10), (128, 128, 128), (128, 128, 128), (16, 128, 128)]
    parts = []
    for k, (rows, cols, fan) in enumerate(shapes):
        w = (2.0 * torch.rand((rows, cols), generator=g, device=DEV) - 1.0) * math.sqrt(3.0 / fan)
        if k == 0:
            w[:, 10:] = 0.0
        if k == 3:
            w[7:] = 0.0
        parts.append(w.reshape(-1))
    w = torch.cat(parts).to(torch.bfloat16).view(torch.int16).contiguous()
    b = 0.1 * torch.randn(400, generator=g, device=DEV)
    b[384 + 7:] = 0.0
    x = 0.5 * torch.randn((c["batch"], 16), generator=g, device=DEV)
    x[:, 10:] = 0.0
    go = torch.randn((c["batch"], 16), generator=g, device=DEV) / c["batch"]
    go[:, 7:] = 0.0
    return w, b.contiguous(), x.contiguous(), go.contiguous()


# ------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, k=0)
    if kind == "bar":
        pos, vol = _body(case, seed)
        sim = vpd.Simulation(_bar_case(case, seed), positions=pos.cpu().numpy(), volumes=vol.cpu().numpy())
        if case["guess"]:
            sim.set_surrogate(*_weights(), guess=case["guess"], newton_steps=2)
        sim.step(case["preload"], diagnostics=False)
        s["sim"] = sim
        s["out"] = {f: np.empty((sim.n_points, w)) for f, w in _bar_fields(case)}
    elif kind == "setup":
        s["pos"], s["vol"] = _body(case, seed)
        s["horizon"] = case["ratio"] * SPACING * _scale(case, seed)
    elif kind == "modules":
        s["pos"], s["vol"] = _body(case, seed)
        s["row_ptr"], s["col"] = vpd.build_neighbor_list(s["pos"], case["ratio"] * SPACING * _scale(case, seed))
        s["kinv"] = vpd.shape_tensor_inverse(s["pos"], s["vol"], s["row_ptr"], s["col"])
        s["path"] = _load_path(s["pos"], seed)
        s["material"] = _material_state(_count(case))
        s["bond_damage"] = torch.zeros(s["col"].shape[0], dtype=torch.float64, device=DEV)
        s["force"] = torch.empty((_count(case), 3), dtype=torch.float64, device=DEV)
        for _ in range(2):  # past the material's initialising call, into plastic flow
            _modules_pass(s)
    elif kind == "points":
        if case["op"] == "return_map":
            s["inc"], s["sig"], s["st"] = _return_map_inputs(case["n"], seed)
        else:
            s["path"] = _point_fields(case["n"], seed)
            s["material"] = _material_state(case["n"])
            if case["op"] == "material":
                for _ in range(3):
                    vpd.material_update(PROPS, POINT_DT, s["path"][_path_index(s["k"])], s["material"])
                    s["k"] += 1
    elif kind == "network":
        s["w"], s["b"], s["x"], s["go"] = _network_inputs(case, seed)
    elif kind == "train":
        s["seed"] = int(seed)
    return s


def _bar_fields(c):
    if _count(c) > 50_000:
        return [("displacement", 3), ("energy_inelastic", 1)]
    return [("displacement", 3), ("velocity", 3), ("stress_corotational", 9), ("state", 6)]


MODULE_INITIATION = 0.03


def _modules_pass(s):
    u = s["path"][_path_index(s["k"])]
    s["k"] += 1
    F = vpd.deformation_gradients(s["pos"], u, s["vol"], s["row_ptr"], s["col"], s["kinv"])
    spatial = vpd.material_update(PROPS, POINT_DT, F, s["material"])
    index = vpd.damage_update(s["pos"], u, s["vol"], s["row_ptr"], s["col"], MODULE_INITIATION, 0.0, s["bond_damage"])
    args = (s["pos"], s["vol"], s["row_ptr"], s["col"], s["kinv"], F, spatial)
    if s["case"]["noalloc"]:
        force = vpd.force_density_noalloc(*args, s["force"], s["bond_damage"])
    else:
        force = vpd.force_density(*args, s["bond_damage"])
    return dict(F=F, spatial=spatial, index=index, force=force, state=s["material"]["state"],
                bond_damage=s["bond_damage"])


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "bar":
        sim = state["sim"]
        out = dict(rows=sim.step(c["steps"]))
        for name, buf in state["out"].items():
            out[name] = sim.field(name, out=buf)
        return out
    if kind == "setup":
        row_ptr, col = vpd.build_neighbor_list(state["pos"], state["horizon"])
        return dict(row_ptr=row_ptr, col=col,
                    kinv=vpd.shape_tensor_inverse(state["pos"], state["vol"], row_ptr, col))
    if kind == "modules":
        return _modules_pass(state)
    if kind == "points":
        if c["op"] == "return_map":
            ep, y, it = vpd.jc_return_map(PROPS, POINT_DT, state["inc"], state["sig"], state["st"])
            return dict(ep=ep, y=y, it=it)
        k = state["k"]
        state["k"] += 1
        if c["op"] == "corotational":
            m = state["material"]
            return vpd.corotational_update(state["path"][_path_index(k)], state["path"][_path_index(k + 1)],
                                           m["left_stretch"], m["rotation"], POINT_DT)
        spatial = vpd.material_update(PROPS, POINT_DT, state["path"][_path_index(k)], state["material"])
        return dict(spatial=spatial, **state["material"])
    if kind == "network":
        if c["op"] == "forward":
            return vpd.mlp_forward(state["w"], state["b"], state["x"])
        return vpd.mlp_gradients(state["w"], state["b"], state["x"], state["go"])
    w, b, report = vpd.train_surrogate(PROPS, samples=c["samples"], epochs=c["epochs"], batch=c["batch"],
                                       seed=state["seed"])
    return dict(weights=w, biases=b, loss=np.asarray(report["epoch_loss"], dtype=np.float32))


# ------------------------------------------------------------------ exact (64-bit torch)
def _neighbours(pos, c, scale):
    """Padded neighbour table [n, slots] (own index where a slot is empty) and its mask, from the lattice offsets."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    horizon = c["ratio"] * SPACING * scale
    reach = int(math.floor(c["ratio"] + 2.0 * math.sqrt(3.0) * c["jitter"] + 1e-9))
    i = torch.arange(pos.shape[0], device=DEV)
    x, y, z = i // (ny * nz), (i // nz) % ny, i % nz
    tol = 64.0 * np.finfo(float).eps * max(horizon, float(pos.abs().max()))
    idx, mask = [], []
    limit = c["ratio"] + 2.0 * math.sqrt(3.0) * c["jitter"] + 1e-6
    for dx in range(-reach, reach + 1):
        for dy in range(-reach, reach + 1):
            for dz in range(-reach, reach + 1):
                if (dx, dy, dz) == (0, 0, 0) or dx * dx + dy * dy + dz * dz > limit * limit:
                    continue
                ok = (x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny) & (z + dz >= 0) & (z + dz < nz)
                j = torch.where(ok, i + (dx * ny + dy) * nz + dz, i)
                d = pos[j] - pos
                ok &= torch.sqrt(d[:, 0] ** 2 + d[:, 1] ** 2 + d[:, 2] ** 2) <= horizon + tol
                if bool(ok.any()):
                    idx.append(torch.where(ok, j, i))
                    mask.append(ok)
    return torch.stack(idx, 1), torch.stack(mask, 1)


def _inverse(a):
    return torch.linalg.inv(a)


def _corotational(Fn, F, Vn, Rn, dt):
    eye = torch.eye(3, dtype=torch.float64, device=F.device)
    L = ((F - Fn) / dt) @ _inverse(Fn)
    D, W = 0.5 * (L + L.mT), 0.5 * (L - L.mT)
    DV = D @ Vn
    z = torch.stack([DV[:, 2, 1] - DV[:, 1, 2], DV[:, 0, 2] - DV[:, 2, 0], DV[:, 1, 0] - DV[:, 0, 1]], 1)
    w = 0.5 * torch.stack([W[:, 2, 1] - W[:, 1, 2], W[:, 0, 2] - W[:, 2, 0], W[:, 1, 0] - W[:, 0, 1]], 1)
    tr = Vn.diagonal(dim1=1, dim2=2).sum(1)[:, None, None]
    o = w + (_inverse(tr * eye - Vn) @ z[:, :, None])[:, :, 0]
    zero = torch.zeros_like(o[:, 0])
    om = torch.stack([zero, -o[:, 2], o[:, 1], o[:, 2], zero, -o[:, 0], -o[:, 1], o[:, 0], zero], 1).reshape(-1, 3, 3)
    sq = (o * o).sum(1)
    mag = torch.sqrt(sq).clamp_min(1e-300)
    big = (sq > 1e-30)[:, None, None]
    q = eye + torch.where(big, (torch.sin(dt * mag) / mag)[:, None, None] * om
                          + (2.0 * torch.sin(0.5 * dt * mag) ** 2 / sq.clamp_min(1e-300))[:, None, None] * (om @ om),
                          torch.zeros_like(om))
    R = q @ Rn
    V = Vn + dt * (L @ Vn - Vn @ om)
    return R.mT @ D @ R, dt * (R.mT @ (W - om) @ R), R, V


def _voigt(t):
    return torch.stack([t[:, 0, 0], t[:, 1, 1], t[:, 2, 2], 0.5 * (t[:, 1, 2] + t[:, 2, 1]),
                        0.5 * (t[:, 0, 2] + t[:, 2, 0]), 0.5 * (t[:, 0, 1] + t[:, 1, 0])], 1)


def _full(v):
    return torch.stack([v[:, 0], v[:, 5], v[:, 4], v[:, 5], v[:, 1], v[:, 3], v[:, 4], v[:, 3], v[:, 2]], 1).reshape(-1, 3, 3)


def _jc_bisect(inc, sig, st, dt):
    """The trial state and the bracketed bisection of the Johnson-Cook update, all points at once."""
    E, nu, A, B, C, hard, m, r0, tref, tmelt = PROPS[:10]
    mu, lam, tol = E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu)), E * 1e-9
    iso = torch.tensor([1.0, 1.0, 1.0, 0.0, 0.0, 0.0], dtype=torch.float64, device=inc.device)
    trial = sig + 2 * mu * inc + lam * inc[:, :3].sum(1, keepdim=True) * iso
    p = trial[:, :3].sum(1) / 3.0
    dev = trial - p[:, None] * iso
    q = torch.sqrt(1.5 * ((dev[:, :3] ** 2).sum(1) + 2.0 * (dev[:, 3:] ** 2).sum(1)))
    ep0, temp, oldy, warm = st[:, 1], st[:, 2], st[:, 3], st[:, 4]
    thermal = 1.0 - ((temp - tref) / (tmelt - tref)).clamp(0.0, 1.0) ** m
    x, lo, hi = torch.zeros_like(q), torch.zeros_like(q), q / (2 * mu)
    y, it, go = oldy.clone(), torch.zeros_like(q), torch.ones_like(q, dtype=torch.bool)
    for k in range(50):
        rate = x / dt
        term = torch.where(rate == 0, torch.ones_like(rate), 1.0 + C * torch.log(torch.where(rate == 0, torch.ones_like(rate), rate) / r0))
        yn = torch.maximum((A + B * (ep0 + x) ** hard) * thermal * term, oldy)
        res = (q - 3 * mu * x).clamp_min(0.0) - yn
        y, it = torch.where(go, yn, y), it + go
        go = go & ~((res.abs() < tol) | ((x == 0) & (res < 0)))
        if not bool(go.any()):
            break
        lo = torch.where(go & (res >= 0), torch.maximum(lo, x), lo)
        hi = torch.where(go & (res < 0), torch.minimum(hi, x), hi)
        nx = torch.minimum(torch.maximum(warm, lo), hi) if k == 0 else 0.5 * (lo + hi)
        x = torch.where(go, nx, x)
    return trial, dev, p, q, x, y, it, iso, mu


def _jc(inc, sig, st, eI, eP, dt):
    rho, beta, cp, wth = PROPS[10:14]
    trial, dev, p, q, x, y, it, iso, mu = _jc_bisect(inc, sig, st, dt)
    first = st[:, 0] == 0
    scale = torch.where(q > 0, (1.0 - 3 * mu * x / q.clamp_min(1e-300)).clamp_min(0.0), torch.ones_like(q))
    new = torch.where(first[:, None] | (q == 0)[:, None], trial, p[:, None] * iso + scale[:, None] * dev)
    pw = 0.5 * x * (q - 3 * mu * x).clamp_min(0.0)
    work = 0.5 * ((sig + new) * inc).sum(1)
    zero = torch.zeros_like(q)
    out = torch.stack([zero + 1, st[:, 1] + x, st[:, 2] + wth * beta * pw / (rho * cp), y, x, st[:, 5] + it], 1)
    out1 = torch.stack([zero + 1, zero, zero + PROPS[8], zero, zero, zero + 1], 1)
    return (new, torch.where(first[:, None], out1, out), torch.where(first, eI, eI + work / rho),
            torch.where(first, eP, eP + pw / rho))


def _material(m, F, dt):
    """One material update of the state dict (tensors [n,3,3], Voigt stress), in place; the spatial stress."""
    dbar, _, m["R"], m["V"] = _corotational(m["F"], F, m["V"], m["R"], dt)
    m["F"] = F
    m["sig"], m["st"], m["eI"], m["eP"] = _jc(_voigt(dbar) * dt, m["sig"], m["st"], m["eI"], m["eP"], dt)
    return m["R"] @ _full(m["sig"]) @ m["R"].mT


def _new_material(n):
    eye = torch.eye(3, dtype=torch.float64, device=DEV).expand(n, 3, 3).clone()
    z = torch.zeros(n, dtype=torch.float64, device=DEV)
    return dict(F=eye, V=eye.clone(), R=eye.clone(), sig=torch.zeros((n, 6), dtype=torch.float64, device=DEV),
                st=torch.zeros((n, 6), dtype=torch.float64, device=DEV), eI=z, eP=z.clone())


class _Bonds:
    def __init__(self, c, pos, vol, scale=1.0):
        self.idx, self.mask = _neighbours(pos, c, scale)
        self.xi = pos[self.idx] - pos[:, None]
        self.w = vol[self.idx] * self.mask
        K = torch.einsum("ns,nsa,nsb->nab", self.w, self.xi, self.xi)
        self.kinv = _inverse(K)
        self.length = self.xi.norm(dim=2)
        self.broken = torch.zeros_like(self.mask)

    def F(self, u):
        G = torch.einsum("ns,nsa,nsb->nab", self.w, u[self.idx] - u[:, None], self.xi)
        return torch.eye(3, dtype=torch.float64, device=DEV) + G @ self.kinv

    def damage(self, u, initiation):
        y = (self.xi + u[self.idx] - u[:, None]).norm(dim=2)
        self.broken |= self.mask & ((y - self.length) / self.length.clamp_min(1e-300) > initiation)

    def force(self, F, spatial):
        M = torch.linalg.det(F)[:, None, None] * spatial @ _inverse(F).mT @ self.kinv
        w = self.w * ~self.broken
        both = torch.einsum("ns,nsa->na", w, self.xi)
        f = (M @ both[:, :, None])[:, :, 0]
        for s0 in range(0, self.idx.shape[1], 32):  # [n, 32, 3, 3] at a time
            part = slice(s0, s0 + 32)
            f = f + torch.einsum("ns,nsab,nsb->na", w[:, part], M[self.idx[:, part]], self.xi[:, part])
        return f


def _bar_exact(c, seed):
    case = _bar_case(c, seed)
    pos, vol = _body(c, seed)
    n = pos.shape[0]
    bonds, m = _Bonds(c, pos, vol), _new_material(n)
    i = torch.arange(n, device=DEV)
    ix, iy, iz = i // (c["ny"] * c["nz"]), (i // c["nz"]) % c["ny"], i % c["nz"]
    support, loaded = ix < 3, ix >= c["nx"] - 3
    # the anchor: the support point nearest the centroid, and the pin above it
    dist = (2 * ix[support] - (c["nx"] - 1)) ** 2 + (2 * iy[support] - (c["ny"] - 1)) ** 2 + (2 * iz[support] - (c["nz"] - 1)) ** 2
    anchor = i[support][torch.argmin(dist)]
    if int((dist == dist.min()).sum()) > 1:  # a tie is settled by the rounding of the centroid, as the host sums it
        nominal = [[a * SPACING, b * SPACING - 0.5 * (c["ny"] - 1) * SPACING, d * SPACING - 0.5 * (c["nz"] - 1) * SPACING]
                   for a in range(c["nx"]) for b in range(c["ny"]) for d in range(c["nz"])]
        centre = [0.0, 0.0, 0.0]
        for p in nominal:
            for d in range(3):
                centre[d] += p[d]
        best = math.inf
        for k in range(3 * c["ny"] * c["nz"]):
            dd = 0.0
            for d in range(3):
                delta = nominal[k][d] - centre[d] / n
                dd += delta * delta
            if dd < best:
                best, anchor = dd, torch.tensor(k, device=DEV)
    ax, az = ix[anchor], iz[anchor]
    pin = (ax * c["ny"] + c["ny"] - 1) * c["nz"] + az

    def prescribe(t, u, v, a):
        if case.bc_mode == vcase.BC_SMOOTH_DISPLACEMENT:
            ph = math.pi * t / case.rise_time
            r = ([case.amplitude, 0.0, 0.0] if t >= case.rise_time else
                 [0.5 * case.amplitude * (1 - math.cos(ph)), 0.5 * case.amplitude * math.pi / case.rise_time * math.sin(ph),
                  0.5 * case.amplitude * (math.pi / case.rise_time) ** 2 * math.cos(ph)])
            s = [0.0, 0.0, 0.0]
        else:
            vh, T = 0.5 * case.grip_velocity, case.ramp_time
            r = [vh * t * t / (2 * T), vh * t / T, vh / T] if t < T else [vh * (t - 0.5 * T), vh, 0.0]
            s = [-q for q in r]
        for x, up, low in zip((u, v, a), r, s):
            x[support, 0] = low
            x[loaded, 0] = up
            x[anchor, 1] = 0.0
            x[anchor, 2] = 0.0
            x[pin, 2] = 0.0

    u, v, a = (torch.zeros((n, 3), dtype=torch.float64, device=DEV) for _ in range(3))
    prescribe(0.0, u, v, a)
    dt = case.dt
    for step in range(1, c["preload"] + c["steps"] + 1):
        u = u + dt * v + 0.5 * dt * dt * a
        prescribe(step * dt, u, v.clone(), a.clone())
        F = bonds.F(u)
        spatial = _material(m, F, dt)
        if c["damage"]:
            bonds.damage(u, case.damage_initiation)
        an = bonds.force(F, spatial) / case.density
        v = v + 0.5 * dt * (a + an)
        a = an
        prescribe(step * dt, u, v, a)
    out = dict(displacement=u, velocity=v, stress_corotational=_full(m["sig"]).reshape(n, 9), state=m["st"],
               energy_inelastic=m["eP"][:, None])
    return dict(rows=None, **{k: out[k] for k, _ in _bar_fields(c)})


def exact(case, seed):
    kind = case["kind"]
    if kind == "bar":
        slots = 4.19 * case["ratio"] ** 3
        if case["precision"] != "fp64" or _count(case) * slots * (case["preload"] + case["steps"]) > 6e9:
            return None  # many seconds of 64-bit torch
        return _bar_exact(case, seed)
    if kind == "setup":
        pos, vol = _body(case, seed)
        return dict(row_ptr=None, col=None, kinv=_Bonds(case, pos, vol, _scale(case, seed)).kinv.reshape(-1, 9))
    if kind == "modules":
        pos, vol = _body(case, seed)
        bonds, m, path = _Bonds(case, pos, vol, _scale(case, seed)), _new_material(pos.shape[0]), _load_path(pos, seed)
        for k in range(3):
            u = path[_path_index(k)]
            F = bonds.F(u)
            spatial = _material(m, F, POINT_DT)
            bonds.damage(u, MODULE_INITIATION)
        index = (bonds.w * bonds.broken).sum(1) / bonds.w.sum(1)
        return dict(F=F.reshape(-1, 9), spatial=spatial.reshape(-1, 9), index=index,
                    force=bonds.force(F, spatial), state=m["st"], bond_damage=None)
    if kind == "points":
        if case["op"] == "return_map":
            inc, sig, st = _return_map_inputs(case["n"], seed)
            *_, x, y, _, _, _ = _jc_bisect(inc, sig, st, POINT_DT)
            return dict(ep=x, y=y, it=None)
        path = [f.reshape(-1, 3, 3) for f in _point_fields(case["n"], seed)]
        eye = torch.eye(3, dtype=torch.float64, device=DEV)
        if case["op"] == "corotational":
            m = _new_material(case["n"])
            dbar, spin, R, V = _corotational(path[0], path[1], m["V"], m["R"], POINT_DT)
            e = 0.5 * (path[1].mT @ path[1] - eye)
            return {k: t.reshape(-1, 9) for k, t in dict(rate_of_deformation=dbar, relative_spin=spin, rotation=R,
                                                         left_stretch=V, strain=e).items()}
        m = _new_material(case["n"])
        for k in range(4):
            spatial = _material(m, path[_path_index(k)], POINT_DT)
        flat = lambda t: t.reshape(-1, 9)  # noqa: E731
        return dict(spatial=flat(spatial), defgrad_old=flat(m["F"]), left_stretch=flat(m["V"]), rotation=flat(m["R"]),
                    strain=flat(0.5 * (m["F"].mT @ m["F"] - eye)), stress_corotational=flat(_full(m["sig"])),
                    state=m["st"], temperature=m["st"][:, 2], energy_internal=m["eI"], energy_inelastic=m["eP"])
    if kind == "network":
        w, b, x, go = _network_inputs(case, seed)
        wd = w.view(torch.bfloat16).double()
        mats = [wd[:2048].view(128, 16), wd[2048:18432].view(128, 128), wd[18432:34816].view(128, 128), wd[34816:].view(16, 128)]
        bias = [b[:128].double(), b[128:256].double(), b[256:384].double(), b[384:].double()]
        if case["op"] == "forward":
            h = x.double()
            for k in range(3):
                h = torch.nn.functional.silu(h @ mats[k].T + bias[k])
            return h @ mats[3].T + bias[3]
        params = [t.clone().requires_grad_() for t in mats + bias]
        h = x.double()
        for k in range(3):
            h = torch.nn.functional.silu(h @ params[k].T + params[4 + k])
        out = h @ params[3].T + params[7]
        grads = torch.autograd.grad((out * go.double()).sum(), params)
        return torch.cat([t.reshape(-1) for t in grads])
    return None


# ------------------------------------------------------------------ work
def _bonds_per_point(c):
    """Mean neighbours per point of the lattice: interior offsets less the faces' missing ones."""
    r = int(c["ratio"])
    total = 0.0
    for dx in range(-r, r + 1):
        for dy in range(-r, r + 1):
            for dz in range(-r, r + 1):
                if 0 < dx * dx + dy * dy + dz * dz <= c["ratio"] ** 2:
                    total += (max(0, c["nx"] - abs(dx)) / c["nx"]) * (max(0, c["ny"] - abs(dy)) / c["ny"]) * \
                             (max(0, c["nz"] - abs(dz)) / c["nz"])
    return total


MLP_MACS = 16 * 128 + 2 * 128 * 128 + 128 * 16


def work(case):
    kind = case["kind"]
    if kind == "bar":
        n, nb, steps = _count(case), _bonds_per_point(case), case["steps"]
        # the state an increment reads and writes once (displacements, velocities, accelerations, the
        # material history, K^-1, the bond masks), and the two bond sums' operations plus the material's
        per_point = 32 + 6 * 32 + 72 + 2 * (3 * 72 + 3 * 48 + 16) + nb / 8 * (3 if case["damage"] else 2)
        return {"bytes": steps * n * per_point, "flops": steps * n * (75 * nb + 900)}
    if kind == "setup":
        n, nb = _count(case), _bonds_per_point(case)
        return {"bytes": n * (24 + 8 + 8 + 72) + n * nb * 4, "flops": n * nb * (9 + 30)}
    if kind == "modules":
        n, nb = _count(case), _bonds_per_point(case)
        # the index row is needed by three bond sums, the bond damage read and written once and read again
        per_point = 24 * 3 + 8 + 72 * 2 + 2 * (9 * 8 * 5 + 6 * 8 + 24) + 72 + 8 + 24
        return {"bytes": n * per_point + n * nb * (4 + 16), "flops": n * nb * (27 + 30 + 33) + 900 * n}
    if kind == "points":
        n = case["n"]
        if case["op"] == "return_map":
            return {"bytes": n * 8 * (6 + 6 + 6 + 2.5), "flops": 300 * n}
        if case["op"] == "corotational":
            return {"bytes": n * 72 * 9, "flops": 500 * n}
        return {"bytes": n * 8 * (9 + 2 * (9 * 4 + 6 + 2) + 1 + 9 + 9), "flops": 1500 * n}
    if kind == "network":
        B = case["batch"]
        if case["op"] == "forward":
            return {"bytes": B * 128 + 75328, "flops": 2 * MLP_MACS * B}
        return {"bytes": B * 128 + 75328 + 149056, "flops": 6 * MLP_MACS * B}
    steps = int(case["samples"] * 0.95) // case["batch"] * case["epochs"]
    return {"bytes": case["samples"] * 128 + steps * case["batch"] * 128,
            "flops": steps * case["batch"] * 6 * MLP_MACS + case["samples"] * 2000}
