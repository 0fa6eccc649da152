"""Performance cases of the liquid-step library, each through its public entry points.

The listed cases are what a program built on the library runs: whole substeps (with host
buffers, and as the chain of device operators that a scheduler drives), the transfers alone,
the reference-shaped operators on host records, and the learned preconditioner's training and
inference. Scenes are the ones of ``fluidity_b200.scenes`` (dam break, sparse splash, column
drop) seen some steps into a run: eight jittered particles per cell, a smooth velocity field
with its APIC slopes and a little noise, positions advected by one step, so that the particles
arrive almost, but not quite, in cell order.

``listed`` names the cases, ``draw`` takes another one from the same ranges, ``prepare`` makes
what a program holds before the call, ``run`` is one pass, ``work`` what the pass cannot do
without, ``exact`` the same results in 64 bits from plain torch.
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch
import torch.nn.functional as F

import fluidity_b200 as fb
from fluidity_b200 import scenes

DT, RHO, GRAVITY = scenes.DT, scenes.DENSITY, scenes.GRAVITY
OFFSETS = [(i, j, k) for k in range(3) for j in range(3) for i in range(3)]


def listed():
    return [
        # The smallest simulation in use (the 32^3 dam break that the CPU path also runs): one
        # substep from and to pinned host memory, where launches and latency are the cost.
        {"name": "step_host_dam_32", "kind": "step_host", "scene": "dam_break", "nx": 32, "ny": 32, "nz": 32, "precision": 0},
        # A preview-size splash through the same call with the BF16 V-cycle.
        {"name": "step_host_splash_64", "kind": "step_host", "scene": "splash", "nx": 64, "ny": 64, "nz": 64, "precision": 1},
        # The 128^3 dam break (2.1M particles) as the chain of device operators, FP32 V-cycle.
        {"name": "substep_dam_128", "kind": "substep", "scene": "dam_break", "nx": 128, "ny": 128, "nz": 128, "precision": 0},
        # The 256^3 sparse splash (29.6M particles), the production size, BF16 V-cycle.
        {"name": "substep_splash_256", "kind": "substep", "scene": "splash", "nx": 256, "ny": 256, "nz": 256, "precision": 1},
        # A box that is no cube and no power of two: ragged hierarchy levels and sparse blocks.
        {"name": "substep_column_ragged", "kind": "substep", "scene": "column_drop", "nx": 104, "ny": 184, "nz": 136, "precision": 1},
        # The transfers alone with a mass per particle: raw deposits and the full gather, as a
        # caller with its own pressure solver uses them.
        {"name": "transfers_mass_ragged", "kind": "transfers", "scene": "splash", "nx": 120, "ny": 104, "nz": 88},
        # The learned block preconditioner applied to a residual of the 128^3 splash.
        {"name": "learned_apply_128", "kind": "learned", "scene": "splash", "nx": 128, "ny": 128, "nz": 128},
        # One training step of that network at the configured batch, convolutions on the tensor cores.
        {"name": "train_bf16_64", "kind": "train", "batch": 64, "tensor_cores": True},
        # The same step in FP32, the exact path, on a batch that fills no multiple of anything.
        {"name": "train_fp32_45", "kind": "train", "batch": 45, "tensor_cores": False},
        # The reference-shaped pressure projection of host records: a dam break's 3375 cells,
        # to the reference's own gate.
        {"name": "mac_pressure_3375", "kind": "mac_pressure", "nx": 15, "ny": 15, "nz": 15},
        # The reference-shaped deposit and gather on host records of 20k particles.
        {"name": "operators_host_20k", "kind": "operators", "blocks": 8, "particles": 20000},
        # The quantized deposit, whole numbers out.
        {"name": "quanta_host_3k", "kind": "quanta", "blocks": 4, "particles": 3000},
    ]


def draw(rng):
    kind = rng.choice(["step_host", "substep", "substep", "transfers", "learned", "train", "train", "mac_pressure",
                       "operators", "quanta"])
    scene = rng.choice(["dam_break", "splash", "column_drop"])

    def cells(lo, hi):  # a multiple of the 8-cell block, log-uniform
        return 8 * max(lo // 8, min(hi // 8, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 8)))

    if kind == "step_host":
        return {"kind": kind, "scene": scene, "nx": cells(24, 72), "ny": cells(24, 72), "nz": cells(24, 72),
                "precision": rng.randrange(2)}
    if kind == "substep":
        return {"kind": kind, "scene": scene, "nx": cells(48, 224), "ny": cells(48, 224), "nz": cells(48, 224),
                "precision": rng.randrange(2)}
    if kind in ("transfers", "learned"):
        return {"kind": kind, "scene": scene, "nx": cells(40, 152), "ny": cells(40, 152), "nz": cells(40, 152)}
    if kind == "train":
        tc = rng.random() < 0.5
        return {"kind": kind, "batch": round(math.exp(rng.uniform(math.log(8), math.log(256 if tc else 100)))),
                "tensor_cores": tc}
    if kind == "mac_pressure":
        return {"kind": kind, "nx": rng.randint(3, 16), "ny": rng.randint(3, 16), "nz": rng.randint(3, 16)}
    if kind == "operators":
        return {"kind": kind, "blocks": rng.randint(4, 10), "particles": round(math.exp(rng.uniform(math.log(500), math.log(60000))))}
    return {"kind": kind, "blocks": rng.randint(3, 8), "particles": round(math.exp(rng.uniform(math.log(100), math.log(20000))))}


# ----------------------------------------------------------------------------- inputs


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _region(scene, X, Y, Z):
    if scene == "dam_break":
        return (X <= 0.5) & (Y <= 0.5) & (Z <= 0.5)
    if scene == "column_drop":
        return (Y <= 0.15) | ((X >= 0.1) & (X <= 0.3) & (Y <= 0.8) & (Z >= 0.1) & (Z <= 0.3))
    ball = lambda cx: (X - cx) ** 2 + (Y - 0.6) ** 2 + (Z - 0.5) ** 2 <= 0.15 ** 2  # noqa: E731
    return (Y <= 0.2) | ball(0.35) | ball(0.65)


def _liquid_cells(case):
    """Liquid cells (m, 3) as x, y, z in (block, cell) order, and their centres in box units."""
    nx, ny, nz = _dims(case)
    axes = [torch.arange(1, n - 1, device="cuda") for n in (nx, ny, nz)]
    K, J, I = torch.meshgrid(axes[2], axes[1], axes[0], indexing="ij")
    inside = _region(case["scene"], (I + 0.5) / nx, (J + 0.5) / ny, (K + 0.5) / nz)
    c = torch.stack([I[inside], J[inside], K[inside]], 1)
    return c[torch.argsort(_cell_key(c, (nx, ny, nz)))]


def _cell_key(c, n):
    x, y, z = c[:, 0], c[:, 1], c[:, 2]
    return ((((z >> 3) * (n[1] // 8) + (y >> 3)) * (n[0] // 8) + (x >> 3)) * 512 + (z & 7) * 64 + (y & 7) * 8 + (x & 7))


def _particles(case, seed):
    """FP32 SoA (15, count) of a scene in motion and the cell width."""
    n, gen = _dims(case), _generator(seed)
    h = 1.0 / n[0]
    cells = _liquid_cells(case)
    strata = torch.tensor([[s & 1, s >> 1 & 1, s >> 2] for s in range(8)], device="cuda")
    m = cells.shape[0]
    soa = torch.empty((15, 8 * m), device="cuda")
    for d in range(3):
        u = torch.rand((m, 8), generator=gen, device="cuda")
        soa[d] = ((cells[:, d, None] + (strata[None, :, d] + u) * 0.5) * h).reshape(-1)
    # a seeded divergence-free flow of about a metre per second, with its exact slopes
    amp = 0.5 + torch.rand((3, 2), generator=gen, device="cuda")
    ph = 6.28 * torch.rand((3, 2), generator=gen, device="cuda")
    for a in range(3):
        soa[3 + a] = 0.01 * torch.randn(8 * m, generator=gen, device="cuda")
        for t in range(2):  # component a varies along the two other axes
            d, w = (a + 1 + t) % 3, 6.28 * (1 + t)
            arg = w * soa[d] + ph[a, t]
            soa[3 + a] += amp[a, t] * torch.sin(arg)
            soa[6 + 3 * a + d] = amp[a, t] * w * torch.cos(arg)
        soa[6 + 3 * a + a] = 0.5 * torch.randn(8 * m, generator=gen, device="cuda")
    if case["scene"] == "splash":  # the two balls approach each other
        up = soa[1] > 0.3 * n[1] * h
        soa[3] += torch.where(up, torch.where(soa[0] < 0.5, 2.0, -2.0), 0.0)
    for d in range(3):
        soa[d] += DT * soa[3 + d]
        soa[d].clamp_(1.001 * h, (n[d] - 1.001) * h)
    return soa, h


def _view(soa, count, mass=None):
    p = fb.Particles()
    at = lambda r: soa.data_ptr() + 4 * r * soa.shape[1]  # noqa: E731
    p.x[:] = [at(d) for d in range(3)]
    p.v[:] = [at(3 + d) for d in range(3)]
    p.c[:] = [at(6 + d) for d in range(9)]
    p.mass = mass.data_ptr() if mass is not None else None
    p.count = count
    return p


def _pointers(tensors):
    return (ctypes.c_void_p * 3)(*[t.data_ptr() for t in tensors])


def _ok(code, *allowed):
    if code != fb.OK and code not in allowed:
        raise fb.FluidityError(code, "performance case")


def _windows(batch, seed):
    """Training windows (batch, 2, 10, 10, 10): smooth residuals scaled to 1 and cell masks with
    a free surface or a wall through part of them."""
    gen = _generator(seed)
    r = torch.randn((batch, 1, 12, 12, 12), generator=gen, device="cuda")
    r = F.avg_pool3d(r, 3, 1) + 0.1 * torch.randn((batch, 1, 10, 10, 10), generator=gen, device="cuda")
    level = torch.randint(4, 14, (batch, 1, 1, 1, 1), generator=gen, device="cuda")
    wall = torch.randint(-4, 3, (batch, 1, 1, 1, 1), generator=gen, device="cuda")
    i = torch.arange(10, device="cuda")
    mask = torch.where(i.view(1, 1, 1, 10, 1) < level, 1.0, 0.0) * torch.ones_like(r)
    mask = torch.where(i.view(1, 1, 1, 1, 10) < wall, -1.0, mask)
    r = torch.where(mask == 1.0, r, 0.0)
    r = r / r.abs().amax(dim=(1, 2, 3, 4), keepdim=True)
    return torch.cat([r, mask], 1).contiguous()


LAYERS = [(2, 16, 27), (16, 16, 27), (16, 32, 27), (32, 32, 27), (32, 64, 27), (64, 32, 1), (32, 32, 27), (32, 16, 1),
          (16, 16, 27), (16, 1, 1)]


def _weights(seed):
    gen, parts = _generator(seed + 7), []
    for cin, cout, taps in LAYERS:
        w = 2 * torch.rand(cin * cout * taps, generator=gen, device="cuda") - 1
        parts += [w * math.sqrt(6.0 / (cin * taps)), 0.05 * torch.randn(cout, generator=gen, device="cuda")]
    return torch.cat(parts)


def _records(case, seed):
    """MacTransferParticle3D records (n, 19) of one cloud in the middle of blocks^3 4^3-cell blocks."""
    rng = np.random.default_rng(seed)
    k, n = case["blocks"], case["particles"]
    h = 1.0 / 32
    x = rng.uniform(1.5, 4 * k - 1.5, (n, 3)) * h
    out = np.zeros((n, 19))
    out[:, 0:3] = x + np.clip(rng.normal(0.0, 0.05 * h, (n, 3)), -0.4 * h, 0.4 * h)
    out[:, 3:6] = x
    out[:, 6] = rng.uniform(0.5, 2.0, n) * h ** 3 * RHO / 8
    out[:, 7:10] = rng.normal(size=(n, 3))
    out[:, 10:19] = 5.0 * rng.normal(size=(n, 9))
    blocks = np.array([[i, j, l] for l in range(k) for j in range(k) for i in range(k)], np.int32)
    return out, blocks, h


def _pressure_system(case, seed):
    """A liquid brick of nx x ny x nz cells in a corner of a tank: sealed walls on the low sides,
    air (Dirichlet) on the high ones; predicted velocities of a falling, moving liquid."""
    rng = np.random.default_rng(seed)
    n, h = _dims(case), 1.0 / 32
    z, y, x = np.meshgrid(*[np.arange(1, v + 1) for v in n[::-1]], indexing="ij")
    cells = np.stack([x.ravel(), y.ravel(), z.ravel()], 1).astype(np.int32)
    values = np.zeros((len(cells), 5))
    values[:, 0] = h ** 3
    faces = []
    for a in range(3):
        size = [v + (d == a) for d, v in enumerate(n)]
        fz, fy, fx = np.meshgrid(*[np.arange(1, v + 1) for v in size[::-1]], indexing="ij")
        faces.append(np.stack([np.full(fx.size, a), fx.ravel(), fy.ravel(), fz.ravel()], 1))
    faces = np.concatenate(faces).astype(np.int32)
    a, fx, fy, fz = (faces[:, k].astype(np.int64) for k in range(4))
    faces = faces[np.lexsort((fx % 4, fy % 4, fz % 4, a, fx // 4, fy // 4, fz // 4))]
    along = faces[np.arange(len(faces)), 1 + faces[:, 0]]
    last = np.array(n)[faces[:, 0]] + 1
    kind = np.where(along == 1, 0, np.where(along == last, 2, 1)).astype(np.int32)
    fv = np.zeros((len(faces), 6))
    open_ = kind != 0
    fv[open_, 0], fv[open_, 1], fv[open_, 2] = h * h, 1.0 / RHO, h
    fv[open_, 3] = 0.3 * rng.normal(size=open_.sum()) + np.where(faces[open_, 0] == 1, DT * GRAVITY[1], 0.0)
    return cells, values, faces, kind, fv, h


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("step_host", "substep", "transfers", "learned"):
        soa, h = _particles(case, seed)
        count = soa.shape[1]
        s["ctx"] = fb.LiquidContext(_dims(case), h=h, capacity=count)
        s["params"] = fb.transfer_params(DT, RHO * h ** 3 / 8)
        s["options"] = fb.default_pressure_options(precision=case.get("precision", 0))
        s["count"] = count
        nx, ny, nz = _dims(case)
        if kind == "step_host":
            s["in"] = soa.cpu().pin_memory()
            s["out"] = torch.empty_like(s["in"]).pin_memory()
            return s
        s["soa"], s["sorted"] = soa, torch.empty_like(soa)
        s["faces"] = [torch.zeros(nx * ny * nz, device="cuda") for _ in range(6)]
        if kind == "substep":
            s["p"] = torch.zeros(nx * ny * nz, dtype=torch.float64, device="cuda")
        elif kind == "transfers":
            g = _generator(seed + 1)
            s["mass"] = RHO * h ** 3 / 8 * (0.5 + torch.rand(count, generator=g, device="cuda"))
            s["mass_sorted"] = torch.empty_like(s["mass"])
            s["u"] = [torch.randn(nx * ny * nz, generator=g, device="cuda") for _ in range(6)]
            s["full"] = torch.zeros((count, 24), device="cuda")
        else:
            A, B = _view(soa, count), _view(s["sorted"], count)
            _ok(fb.library().fl_topology_from_particles(s["ctx"].handle, A, None, fb.Report()))
            _ok(fb.library().fl_sort_particles_by_block(s["ctx"].handle, A, B, None, fb.Report()))
            n = 512 * len(s["ctx"].active_blocks())
            # a residual on the liquid cells alone, smooth along the cell order
            r = torch.randn(nx * ny * nz, generator=_generator(seed + 2), device="cuda")
            s["r"] = F.avg_pool1d(r.view(1, 1, -1), 5, 1, 2).view(-1)
            starts = fb.copy_to_host(s["ctx"].fields()["cell_start"], n + 1, np.int32)
            s["r"][:n] *= torch.from_numpy((starts[1:] > starts[:-1]).astype(np.float32)).cuda()
            s["r"][n:] = 0.0
            s["z"] = torch.zeros_like(r)
            s["weights"] = _weights(seed)
            s["ctx"].set_learned_preconditioner(s["weights"])
            # the solver classifies the cells that the network's mask is made of
            ups = _pointers(s["faces"][:3])
            _ok(fb.library().fl_pressure_project(s["ctx"].handle, ups, _pointers(s["faces"][3:]), s["params"], s["options"],
                                                 None, None, None), fb.ABORTED)
        return s
    if kind == "train":
        b = case["batch"]
        s["net"] = fb.UNet(b, tensor_cores=case["tensor_cores"])
        s["x"], s["P"] = _windows(b, seed), _weights(seed)
        s["G"], s["M"], s["V"] = (torch.zeros_like(s["P"]) for _ in range(3))
        s["y"], s["gy"] = torch.zeros((b, 512), device="cuda"), torch.zeros((b, 512), device="cuda")
        s["loss"], s["step"] = torch.zeros(1, device="cuda"), 0
        return s
    if kind == "mac_pressure":
        s["system"] = _pressure_system(case, seed)
        return s
    s["records"], s["blocks"], s["h"] = _records(case, seed)
    rng = np.random.default_rng(seed + 3)
    s["old"], s["new"] = rng.normal(size=(2, 192 * len(s["blocks"])))
    return s


# ----------------------------------------------------------------------------- one pass


def run(s):
    kind, lib = s["case"]["kind"], fb.library()
    if kind == "step_host":
        _, diag = s["ctx"].step_host(s["in"].numpy(), s["out"].numpy(), s["params"], s["options"])
        return [s["out"][r] for r in range(15)]
    if kind in ("substep", "transfers"):
        ctx, n, mass = s["ctx"].handle, s["count"], s.get("mass")
        A, B = _view(s["soa"], n, mass), _view(s["sorted"], n, s.get("mass_sorted"))
        _ok(lib.fl_topology_from_particles(ctx, A, None, fb.Report()))
        _ok(lib.fl_sort_particles_by_block(ctx, A, B, None, None))
        out = list(s["faces"])  # sized for the whole lattice, active blocks first
        f0, f1 = _pointers(s["faces"][:3]), _pointers(s["faces"][3:])
        if kind == "transfers":
            _ok(lib.fl_p2g(ctx, B, s["params"], 0, f0, f1, None, None))
            _ok(lib.fl_g2p(ctx, B, _pointers(s["u"][:3]), _pointers(s["u"][3:]), DT, s["full"].data_ptr(), None, None))
            return out + [s["full"][:, 0:3], s["full"][:, 3:6], s["full"][:, 6:15], s["full"][:, 15:24], s["mass_sorted"]]
        _ok(lib.fl_p2g(ctx, B, s["params"], 1, f0, (ctypes.c_void_p * 3)(), None, None))
        _ok(lib.fl_pressure_project(ctx, f0, f1, s["params"], s["options"], fb.PressureDiagnostics(), s["p"].data_ptr(), None))
        _ok(lib.fl_g2p(ctx, B, f1, (ctypes.c_void_p * 3)(), DT, None, None, None))
        return out + [s["p"]] + [s["sorted"][r] for r in range(15)]
    if kind == "learned":
        s["ctx"].apply_learned(s["r"], s["z"])
        return s["z"]
    if kind == "train":
        s["step"] += 1
        s["net"].forward(s["P"], s["x"], s["y"])
        fb.UNet.block_residual_loss(s["y"], s["x"], s["loss"], s["gy"])
        s["net"].backward(s["P"], s["gy"], s["G"])
        fb.UNet.adam_step(s["P"], s["G"], s["M"], s["V"], s["step"])
        return {"y": s["y"], "loss": s["loss"], "grads": s["G"], "params": s["P"], "m": s["M"], "v": s["V"]}
    if kind == "mac_pressure":
        ci, cv, fi, fk, fv, h = s["system"]
        o = fb.project_mac_pressure_3d(ci, cv, fi, fk, fv, h, DT)
        return {k: o[k] for k in ("pressure", "rhs", "residual", "defect", "corrected_u")}
    origin = (0.0, 0.0, 0.0)
    if kind == "operators":
        m, q, _ = fb.deposit_mac_3d(origin, s["h"], s["blocks"], s["records"])
        g, _ = fb.gather_mac_3d(origin, s["h"], s["blocks"], s["records"], s["old"], s["new"])
        return [m, q, g[:, 0:3], g[:, 3:6], g[:, 6:15], g[:, 15:24]]
    m, q, _ = fb.deposit_mac_quanta_3d(origin, s["h"], s["blocks"], s["records"], 2.0 ** -40, 2.0 ** -34, len(s["records"]))
    return [m, q]


# ----------------------------------------------------------------------------- the least work


def _scene_size(case):
    """Particles, active blocks and liquid cells of a scene, from its region alone."""
    nx, ny, nz = _dims(case)
    z, y, x = np.meshgrid(*[np.arange(1, v - 1) for v in (nz, ny, nx)], indexing="ij")
    inside = _region(case["scene"], (x + 0.5) / nx, (y + 0.5) / ny, (z + 0.5) / nz)
    occ = np.zeros((nz // 8 + 2, ny // 8 + 2, nx // 8 + 2), bool)
    occ[z[inside] // 8 + 1, y[inside] // 8 + 1, x[inside] // 8 + 1] = True
    act = np.zeros_like(occ)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                act |= np.roll(occ, (dz, dy, dx), (0, 1, 2))
    return 8 * int(inside.sum()), int(act[1:-1, 1:-1, 1:-1].sum()), int(inside.sum())


def work(case):
    kind = case["kind"]
    if kind in ("step_host", "substep", "transfers", "learned"):
        n, blocks, liquid = _scene_size(case)
        faces = 3 * 512 * blocks
        p2g, g2p = n * 27 * 3 * 6, n * 27 * 3 * 8  # multiply-adds of the B-spline sums
        if kind == "step_host":  # the state in and out
            return {"bytes": 120 * n, "flops": p2g + g2p}
        if kind == "substep":  # the state in and out, predicted and corrected faces, the pressure
            return {"bytes": 120 * n + 8 * faces + 8 * 512 * blocks, "flops": p2g + g2p}
        if kind == "transfers":  # the state, masses and two face fields in; two face fields and 24 values out
            return {"bytes": 64 * n + 16 * faces + 96 * n, "flops": p2g + 2 * g2p}
        return {"bytes": 8 * 512 * blocks + 2 * 141937, "flops": 25.6e6 * liquid / 512}
    if kind == "train":  # windows and parameters in, parameters, moments, gradients and outputs out
        b = case["batch"]
        return {"bytes": 4 * (2000 + 1024) * b + 4 * 7 * 141937, "flops": 3 * 25.6e6 * b}
    if kind == "mac_pressure":
        c = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 8 * (5 + 4) * c + 3 * c * (8 * 7 + 20) + 12 * c, "flops": 40.0 * 20 * c}
    n, faces = case["particles"], 192 * case["blocks"] ** 3
    if kind == "operators":
        return {"bytes": 8 * (2 * 19 * n + 24 * n + 4 * faces), "flops": n * 27 * 3 * 22}
    return {"bytes": 8 * (19 * n + 2 * faces), "flops": n * 27 * 3 * 8}


def tolerance(case):
    kind = case["kind"]
    if kind == "quanta":
        return "exact"
    # Each about four times what was seen against `exact`, or between two V-cycles, orders of the
    # batch or parameters 1e-7 apart where a projection's stop or a ReLU's edge decides.
    if kind in ("transfers", "operators"):  # FP32 sums of some 200 terms in another order: 4e-6
        return {"rel": 1.5e-5, "max": 2e-4}
    if kind in ("substep", "step_host"):  # and a projection that stops at a 1e-6 residual: 1.2e-6
        return {"rel": 5e-6, "max": 1e-4}
    if kind == "learned":  # BF16 weights and activations: 4.6e-3
        return {"rel": 1e-2, "max": 0.25}
    if kind == "train" and case["tensor_cores"]:  # BF16 operands, masks that flip: 1e-3
        return {"rel": 4e-3, "max": 0.15}
    if kind == "train":  # squared FP32 gradients: 1.3e-5
        return {"rel": 5e-5, "max": 1e-3}
    return {"rel": 1e-6, "max": 1e-4}  # FP64 CG stopped at the reference's gate, dot products in another order


# ----------------------------------------------------------------------------- 64-bit results


def _axis(X, a, axis):
    """First node, the three weights, their derivatives and the node offsets of one axis (cell units)."""
    shift = 0.0 if axis == a else 0.5
    first = torch.floor(X - shift - 0.5)
    lo = first + shift
    c = X - (lo + 1)
    w = torch.stack([0.5 * (0.5 - c) ** 2, 0.75 - c * c, 0.5 * (0.5 + c) ** 2])
    dw = torch.stack([c - 0.5, -2 * c, c + 0.5])
    r = torch.stack([lo - X, lo + 1 - X, lo + 2 - X])
    return first.long(), w, dw, r


class _Grid:
    """Dense FP64 faces of a box of cells: low faces, one layer of nodes beyond every side."""

    def __init__(self, n):
        self.n, self.pad = n, tuple(v + 6 for v in n)

    def index(self, f, o):
        i = [f[d] + o[d] + 3 for d in range(3)]
        return (i[2] * self.pad[1] + i[1]) * self.pad[0] + i[0]

    def deposit(self, X, v, C, mass, h):
        out = []
        for a in range(3):
            ax = [_axis(X[d], a, d) for d in range(3)]
            first = [t[0] for t in ax]
            W, Q = (torch.zeros(math.prod(self.pad), dtype=torch.float64, device=X[0].device) for _ in range(2))
            for o in OFFSETS:
                w = ax[0][1][o[0]] * ax[1][1][o[1]] * ax[2][1][o[2]] * mass
                u = v[a] + h * sum(C[3 * a + d] * ax[d][3][o[d]] for d in range(3))
                at = self.index(first, o)
                W.index_add_(0, at, w)
                Q.index_add_(0, at, w * u)
            out.append((W, Q))
        return out

    def gather(self, X, faces, h):
        v, fit, grad = [], [], []
        for a in range(3):
            ax = [_axis(X[d], a, d) for d in range(3)]
            first = [t[0] for t in ax]
            s = [torch.zeros_like(X[0]) for _ in range(7)]
            for o in OFFSETS:
                u = faces[a][self.index(first, o)]
                w = [ax[d][1][o[d]] for d in range(3)]
                full = w[0] * w[1] * w[2] * u
                s[0] += full
                for d in range(3):
                    s[1 + d] += full * ax[d][3][o[d]]
                    s[4 + d] += ax[d][2][o[d]] * w[(d + 1) % 3] * w[(d + 2) % 3] * u
            v.append(s[0])
            fit += [4 * t / h for t in s[1:4]]
            grad += [t / h for t in s[4:7]]
        return v, fit, grad

    def inner(self, f):
        nx, ny, nz = self.n
        return f.view(self.pad[2], self.pad[1], self.pad[0])[3:3 + nz, 3:3 + ny, 3:3 + nx]


def _to_blocks(f, act):
    """Dense (nz, ny, nx) values as the 8^3 blocks of `act` in order, zeros after them."""
    nz, ny, nx = f.shape
    f = f.reshape(nz // 8, 8, ny // 8, 8, nx // 8, 8).permute(0, 2, 4, 1, 3, 5).reshape(-1, 512)[act.reshape(-1)].reshape(-1)
    return F.pad(f, (0, nz * ny * nx - f.numel()))


def _sorted_state(case, soa, h):
    n = _dims(case)
    cell = torch.stack([torch.floor(soa[d] * np.float32(1.0 / h)).long() for d in range(3)], 1)
    order = torch.sort(_cell_key(cell, n), stable=True).indices
    cell = cell[order]
    count = torch.zeros(n[2], n[1], n[0], device="cuda")
    count.index_put_((cell[:, 2], cell[:, 1], cell[:, 0]), torch.ones((), device="cuda"), accumulate=True)
    occ = (F.max_pool3d(count[None, None], 8)[0, 0] > 0).float()
    act = F.max_pool3d(occ[None, None], 3, 1, 1)[0, 0] > 0
    return order, count > 0, act


def _solve(fluid, solid, u, h):
    """Pressure and corrected faces of the box by FP64 Jacobi CG on dense arrays."""
    pad = lambda t, v: F.pad(t[None, None], (1, 1, 1, 1, 1, 1), value=v)[0, 0]  # noqa: E731
    fl, so = pad(fluid.double(), 0.0), pad(solid.double(), 1.0)
    core = (slice(1, -1),) * 3

    def shift(t, axis, by):  # value at the neighbour along x, y or z
        return torch.roll(t, -by, 2 - axis)

    both = [(fl * shift(fl, a, -1)) for a in range(3)]  # fluid on both sides of the low face
    diag = sum((1 - shift(so, a, b)) for a in range(3) for b in (-1, 1))[core] * fluid
    diag = torch.where(diag > 0, diag, torch.ones_like(diag))

    def apply(p):
        q = pad(p * fluid, 0.0)
        s = sum(shift(q, a, b) for a in range(3) for b in (-1, 1))[core]
        return (diag * p - s) * fluid

    high = [torch.cat([u[a].narrow(2 - a, 1, u[a].shape[2 - a] - 1), torch.zeros_like(u[a].narrow(2 - a, 0, 1))], 2 - a) for a in range(3)]
    b = -(RHO * h / DT) * sum(high[a] - u[a] for a in range(3)) * fluid
    p, r = torch.zeros_like(b), b.clone()
    z = r / diag
    d, rz = z.clone(), (r * z).sum()
    stop = 1e-13 * b.norm()
    for it in range(6000):
        q = apply(d)
        alpha = rz / (d * q).sum()
        p += alpha * d
        r -= alpha * q
        if it % 16 == 15 and r.norm() <= stop:
            break
        z = r / diag
        rz_new = (r * z).sum()
        d = z + (rz_new / rz) * d
        rz = rz_new
    del both
    pp, out = pad(p * fluid, 0.0), []
    for a in range(3):
        open_ = ((1 - so) * (1 - shift(so, a, -1)) * ((fl + shift(fl, a, -1)) > 0))[core]
        out.append(u[a] + open_ * (DT / (RHO * h)) * (shift(pp, a, -1) - pp)[core])
    return p, out


def _exact_scene(case, seed):
    kind = case["kind"]
    soa, h = _particles(case, seed)
    if soa.shape[1] > 4_000_000:  # the scattered FP64 sums of more particles take too long
        return None
    n, g = _dims(case), _Grid(_dims(case))
    count = soa.shape[1]
    order, fluid, act = _sorted_state(case, soa, h)
    st = soa[:, order].double()
    X = [st[d] / h for d in range(3)]
    idx = [torch.arange(v, device="cuda") for v in n]
    K, J, I = torch.meshgrid(idx[2], idx[1], idx[0], indexing="ij")
    at = (I, J, K)
    if kind == "transfers":
        gen = _generator(seed + 1)
        mass = RHO * h ** 3 / 8 * (0.5 + torch.rand(count, generator=gen, device="cuda"))
        u = [torch.randn(math.prod(n), generator=gen, device="cuda") for _ in range(6)]
        ms = mass[order]
        dep = g.deposit(X, st[3:6], st[6:15], ms.double(), h)
        blocks = int(act.sum())
        dense = []
        for a in range(6):
            full = torch.zeros(act.numel(), 512, dtype=torch.float64, device="cuda")
            full[act.reshape(-1)] = u[a][:512 * blocks].double().view(-1, 512)
            bz, by, bx = act.shape
            f = full.view(bz, by, bx, 8, 8, 8).permute(0, 3, 1, 4, 2, 5).reshape(n[2], n[1], n[0])
            dense.append(F.pad(f[None, None], (3,) * 6)[0, 0].reshape(-1))
        v, fit, grad = g.gather(X, dense[:3], h)
        old, _, _ = g.gather(X, dense[3:], h)
        out = [_to_blocks(g.inner(dep[a][k]), act) for k in range(2) for a in range(3)]
        return out + [torch.stack(v, 1), torch.stack([v[a] - old[a] for a in range(3)], 1), torch.stack(fit, 1), torch.stack(grad, 1), ms]
    mass = torch.full((count,), RHO * h ** 3 / 8, dtype=torch.float64, device="cuda")
    dep = g.deposit(X, st[3:6], st[6:15], mass, h)
    solid = torch.zeros_like(fluid)
    for d in range(3):
        solid |= (at[d] < 1) | (at[d] > n[d] - 2)
    fluid &= ~solid
    up = []
    for a in range(3):
        W, Q = (g.inner(t) for t in dep[a])
        u = torch.where(W > 0, Q / torch.where(W > 0, W, torch.ones_like(W)), torch.zeros_like(W)) + DT * GRAVITY[a]
        wall = solid | torch.roll(solid, 1, 2 - a) | (at[a] == 0)
        up.append(torch.where(wall, torch.zeros_like(u), u))
    p, un = _solve(fluid, solid, up, h)
    v, fit, _ = g.gather(X, [F.pad(f[None, None], (3,) * 6)[0, 0].reshape(-1) for f in un], h)
    x = [(st[d] + DT * v[d]).clamp((1 + 1e-3) * h, (n[d] - 1 - 1e-3) * h) for d in range(3)]
    if kind == "step_host":
        return x + v + fit
    return [_to_blocks(f, act) for f in up + un + [p]] + x + v + fit


def _network(P, x):
    """The U-Net on (batch, 2, 10, 10, 10) windows."""
    at, params = 0, []
    for cin, cout, taps in LAYERS:
        k = 3 if taps == 27 else 1
        w = P[at:at + cin * cout * taps].view(cout, cin, k, k, k)
        at += w.numel()
        params.append((w, P[at:at + cout]))
        at += cout
    conv = lambda i, t, pad: F.conv3d(t, *params[i], padding=pad)  # noqa: E731
    up = lambda t: F.interpolate(t, scale_factor=2, mode="nearest")  # noqa: E731
    s1 = F.relu(conv(1, F.relu(conv(0, x, 0)), 1))
    s2 = F.relu(conv(3, F.relu(conv(2, F.avg_pool3d(s1, 2), 1)), 1))
    bt = F.relu(conv(4, F.avg_pool3d(s2, 2), 1))
    d2 = F.relu(conv(6, F.relu(conv(5, up(bt), 0) + s2), 1))
    d1 = F.relu(conv(8, F.relu(conv(7, up(d2), 0) + s1), 1))
    return conv(9, d1, 0).reshape(x.shape[0], 512)


def _block_loss(y, x):
    mask = x[:, 1]
    fluid = (mask == 1).double()
    inner = fluid[:, 1:9, 1:9, 1:9]
    sides = [(z, y_, x_) for z, y_, x_ in ((0, 1, 1), (2, 1, 1), (1, 0, 1), (1, 2, 1), (1, 1, 0), (1, 1, 2))]
    at = lambda t, o: t[:, o[0]:o[0] + 8, o[1]:o[1] + 8, o[2]:o[2] + 8]  # noqa: E731
    diag = sum((at(mask, o) >= 0).double() for o in sides)
    yc = y.view(-1, 8, 8, 8) * inner
    yp = F.pad(yc, (1,) * 6)
    r = x[:, 0, 1:9, 1:9, 1:9] * inner
    rho = (r - (diag * yc - sum(at(yp, o) for o in sides))) * inner
    den = (r ** 2).sum(dim=(1, 2, 3))
    valid = (den > 0).double()
    return ((rho ** 2).sum(dim=(1, 2, 3)) / den.clamp(min=1.0) * valid).sum() / valid.sum()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step_host", "substep", "transfers"):
        return _exact_scene(case, seed)
    if kind == "learned":
        s = prepare(case, seed)
        blocks = s["ctx"].active_blocks()
        n = _dims(case)
        _, fluid, act = _sorted_state(case, s["soa"], 1.0 / n[0])
        # windows of residual and mask over the whole box: 1 liquid, 0 air, -1 solid (and outside)
        dense = torch.zeros((2, n[2], n[1], n[0]), dtype=torch.float64, device="cuda")
        b = torch.from_numpy(blocks).cuda().long()
        l = torch.arange(512, device="cuda")
        z, y, x = (8 * b[:, k, None] + o for k, o in ((2, l >> 6), (1, l >> 3 & 7), (0, l & 7)))
        dense[0, z, y, x] = s["r"][:512 * len(b)].double().view(-1, 512)
        dense[1] = fluid.double()
        for d in range(3):
            i = torch.arange(n[d], device="cuda").view([-1 if k == 2 - d else 1 for k in range(3)])
            dense[1] = torch.where((i < 1) | (i > n[d] - 2), -1.0, dense[1])
        pad = torch.stack([F.pad(dense[0], (1,) * 6), F.pad(dense[1], (1,) * 6, value=-1.0)])
        w = torch.arange(10, device="cuda")
        out = []
        for part in b.split(256):
            at = [(8 * part[:, k, None] + w) for k in (2, 1, 0)]
            win = pad[:, at[0][:, :, None, None], at[1][:, None, :, None], at[2][:, None, None, :]].permute(1, 0, 2, 3, 4).contiguous()
            win[:, 0] *= win[:, 1] == 1
            scale = win[:, 0].abs().amax(dim=(1, 2, 3))
            win[:, 0] /= torch.where(scale > 0, scale, 1.0).view(-1, 1, 1, 1)
            yv = _network(s["weights"].double(), win) * scale[:, None]
            out.append(yv * (win[:, 1, 1:9, 1:9, 1:9] == 1).reshape(-1, 512))
        z = torch.cat(out).reshape(-1)
        return F.pad(z, (0, n[0] * n[1] * n[2] - z.numel()))
    if kind == "train":
        x = _windows(case["batch"], seed).double()
        P = _weights(seed).double().requires_grad_()
        y = _network(P, x)
        loss = _block_loss(y, x)
        loss.backward()
        if case["tensor_cores"]:  # masks that BF16 flips near zero move the gradients themselves
            return {"y": y.detach(), "loss": None, "grads": None, "params": None, "m": None, "v": None}
        g = P.grad
        m, v = 0.1 * g, 0.001 * g * g
        step = 1e-3 * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8)
        return {"y": y.detach(), "loss": loss.detach().reshape(1), "grads": g, "params": P.detach() - step, "m": m, "v": v}
    if kind == "mac_pressure":
        cells, values, faces, kinds, fv, h = _pressure_system(case, seed)
        order = {tuple(c): i for i, c in enumerate(cells.tolist())}
        A, b = np.zeros((len(cells),) * 2), np.zeros(len(cells))
        ends = []
        for f, (a, *head) in enumerate(faces.tolist()):
            tail = list(head)
            tail[a] -= 1
            t, hd = order.get(tuple(tail)), order.get(tuple(head))
            ends.append((t, hd))
            c = fv[f, 0] * DT * fv[f, 1] / fv[f, 2] if fv[f, 0] > 0 else 0.0
            flux = fv[f, 0] * fv[f, 3]
            for i, other, sign in ((t, hd, -1.0), (hd, t, 1.0)):
                if i is not None:
                    b[i] += sign * flux
                    A[i, i] += c
                    if other is not None:
                        A[i, other] -= c
        p = torch.linalg.solve(torch.from_numpy(A).cuda(), torch.from_numpy(b).cuda()).cpu().numpy()
        u = fv[:, 3].copy()
        for f, (t, hd) in enumerate(ends):
            if fv[f, 0] > 0:
                u[f] += DT * fv[f, 1] / fv[f, 2] * ((p[t] if t is not None else 0.0) - (p[hd] if hd is not None else 0.0))
        return {"pressure": p, "rhs": b, "residual": None, "defect": None, "corrected_u": u}
    if kind == "quanta":
        return None  # whole numbers
    rec, blocks, h = _records(case, seed)
    k = case["blocks"]
    g = _Grid((4 * k,) * 3)
    t = torch.from_numpy(rec).cuda()
    X = [t[:, 3 + d] / h for d in range(3)]
    dep = g.deposit(X, [t[:, 7 + d] for d in range(3)], [t[:, 10 + d] for d in range(9)], t[:, 6], h)
    slots = lambda fs: torch.stack([g.inner(f).reshape(k, 4, k, 4, k, 4).permute(0, 2, 4, 1, 3, 5).reshape(-1, 64)  # noqa: E731
                                    for f in fs], 1).reshape(-1)
    rng = np.random.default_rng(seed + 3)
    old, new = rng.normal(size=(2, 192 * len(blocks)))

    def dense(u):
        per = torch.from_numpy(u).cuda().view(-1, 3, 64)
        return [F.pad(per[:, a].reshape(k, k, k, 4, 4, 4).permute(0, 3, 1, 4, 2, 5).reshape(1, 1, 4 * k, 4 * k, 4 * k),
                      (3,) * 6).reshape(-1) for a in range(3)]

    v, fit, grad = g.gather(X, dense(new), h)
    vo, _, _ = g.gather(X, dense(old), h)
    return [slots([d[0] for d in dep]), slots([d[1] for d in dep]), torch.stack(v, 1),
            torch.stack([v[a] - vo[a] for a in range(3)], 1), torch.stack(fit, 1), torch.stack(grad, 1)]
