"""Workloads that programs run through this package, for timing and for comparing results.

``listed()`` names twelve of them, ``draw(rng)`` gives more of the same ranges; ``prepare``
builds what a program holds before its time loop (inputs made on the GPU from a seed),
``run`` makes one pass of the loop's body through the public entry points, ``work`` counts the
bytes and operations of a pass and ``exact`` computes its results in 64 bits with plain torch.

Paths (the ``"path"`` of a case):
  flow       Domain, config mode: a box stepped ``steps`` times, its fields exported to device
             tensors, its force history read where forces are on.  ``kind`` "porous": fully
             periodic box with random spheres and a body force; "channel": inlet, outlet,
             walls and one fixed sphere; "moving": the channel with an oscillating sphere whose
             pose the host passes in before every step.
  sweep      Batch: many small channels of uneven sizes stepped together by a captured graph.
  reference  Domain, reference mode: the loop of main_simulation (pose, step, force of the
             step) on a z-periodic box with a heaving cylinder.
  conv       one 3x3x3 convolution layer of the warm-start network, forward and backward.
  forward    the warm-start network's forward pass.
  train      one training step of the warm-start network.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from lbm3d_bb_b200 import Domain, abi
from lbm3d_bb_b200 import unet as unet_mod
from lbm3d_bb_b200.batch import Batch

PERIODIC = ("periodic",) * 6
CX = (1, -1, 0, 0, 0, 0, 1, -1, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0, 0)
CY = (0, 0, 1, -1, 0, 0, 1, -1, 0, 0, 1, -1, -1, 1, 0, 0, 1, -1, 0)
CZ = (0, 0, 0, 0, 1, -1, 0, 0, 1, -1, 1, -1, 0, 0, -1, 1, -1, 1, 0)
OPP = tuple(d ^ 1 for d in range(18)) + (18,)
WGT = tuple([1 / 18] * 6 + [1 / 36] * 12 + [1 / 3])
STORE_BYTES = {"fp32": 4, "fp64": 8, "fp16dev": 2}
TRT_LAMBDA = 3.0 / 16.0
LAYERS = (("e1a", 16, 16, True, 1), ("e1b", 16, 16, True, 1), ("e2a", 16, 32, True, 2), ("e2b", 32, 32, True, 2),
          ("e3a", 32, 64, True, 4), ("e3b", 64, 64, True, 4), ("d2a", 96, 32, True, 2), ("d2b", 32, 32, True, 2),
          ("d1a", 48, 16, True, 1), ("d1b", 16, 16, True, 1), ("head", 16, 16, False, 1))  # name, cin, cout, relu, coarsening


def _flow(kind, nx, ny, nz, storage, coll, tau, steps, outlet="pressure", force=True, accel="x"):
    return {"path": "flow", "kind": kind, "nx": nx, "ny": ny, "nz": nz, "storage": storage, "coll": coll, "tau": tau,
            "steps": steps, "outlet": outlet, "force": force, "accel": accel}


def listed():
    return [
        # a design loop around one body: a short run on a box that fits in L2, its drag read back
        dict(name="channel_small", **_flow("channel", 96, 48, 48, "fp32", "BGK", 0.8, 8, outlet="outflow")),
        # external flow at an ordinary size
        dict(name="channel_large", **_flow("channel", 384, 192, 192, "fp32", "BGK", 0.6, 4)),
        # a body whose motion law lives on the host
        dict(name="moving_sphere", **_flow("moving", 192, 96, 96, "fp32", "TRT", 0.56, 8, outlet="outflow")),
        # porous media in the three storage forms; the FP32 box is the benchmark's
        dict(name="porous_fp32", **_flow("porous", 512, 512, 512, "fp32", "BGK", 0.6, 4, force=False)),
        dict(name="porous_fp16dev", **_flow("porous", 512, 256, 256, "fp16dev", "BGK", 0.6, 4, force=False)),
        dict(name="porous_fp64", **_flow("porous", 256, 256, 256, "fp64", "BGK", 0.6, 4, force=False)),
        # a periodic box of no convenient size, forced along a diagonal
        dict(name="porous_ragged", **_flow("porous", 210, 187, 171, "fp32", "TRT", 0.7, 4, accel="xyz")),
        # a parameter sweep over small channels
        {"name": "sweep", "path": "sweep", "count": 64, "storage": "fp32", "steps": 20},
        # the reference's own driver loop on a thin cylinder box
        {"name": "reference_cylinder", "path": "reference", "nx": 480, "ny": 240, "nz": 4, "radius": 16.5, "coll": "TRT",
         "q": 19, "reynolds": 150.0, "steps": 8},
        # the warm-start network: a wide layer in both directions, a prediction, a training step
        {"name": "conv_layer", "path": "conv", "n": 4, "d": 32, "h": 32, "w": 64, "cin": 96, "cout": 32},
        {"name": "network_forward", "path": "forward", "n": 4, "d": 64, "h": 64, "w": 128},
        {"name": "network_train", "path": "train", "n": 4, "d": 64, "h": 64, "w": 128},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["porous", "porous", "porous", "channel", "channel", "channel", "moving", "moving", "sweep",
                       "reference", "conv", "conv", "forward", "train"])
    if path in ("porous", "channel", "moving"):
        cells = _log_int(rng, 1.5e5, 2e7)
        storage = rng.choice(["fp32", "fp32", "fp16dev", "fp64"])
        coll = rng.choice(["BGK", "TRT"])
        n = round(cells ** (1 / 3))
        nx = max(24, round(n * rng.uniform(0.8, 2.0)))
        if rng.random() < 0.5:
            nx = max(32, (nx + 16) // 32 * 32)
        if rng.random() < 0.3:
            nx = max(128, (nx + 64) // 128 * 128)
        ny = max(20, round(math.sqrt(cells / nx) * rng.uniform(0.8, 1.25)))
        nz = max(20, round(cells / (nx * ny)))
        if path == "porous":
            tau = rng.uniform(0.55, 1.0)
            return _flow("porous", nx, ny, nz, storage, coll, round(tau, 3), rng.randint(2, 8),
                         force=rng.random() < 0.5, accel=rng.choice(["x", "xyz"]))
        tau = rng.uniform(0.55, 0.9) if coll == "TRT" else rng.uniform(0.58, 0.9)
        return _flow(path, nx, ny, nz, storage, coll, round(tau, 3), rng.randint(2, 8),
                     outlet=rng.choice(["pressure", "outflow"]))
    if path == "sweep":
        return {"path": "sweep", "count": rng.randint(8, 80), "storage": rng.choice(["fp32", "fp32", "fp16dev", "fp64"]),
                "steps": rng.randint(6, 24)}
    if path == "reference":
        nx = _log_int(rng, 120, 700)
        ny = max(60, round(nx * rng.uniform(0.4, 0.7)))
        return {"path": "reference", "nx": nx, "ny": ny, "nz": rng.randint(2, 12), "radius": round(ny * rng.uniform(0.05, 0.1) + 0.16, 2),
                "coll": rng.choice(["BGK", "TRT"]), "q": rng.choice([19, 19, 27]),
                "reynolds": round(rng.uniform(60, 180), 1), "steps": rng.randint(2, 8)}
    vox = _log_int(rng, 3e4, 2e6)
    w = rng.choice([64, 128, 192])
    n = rng.randint(1, 5)
    dh = max(4.0, math.sqrt(vox / (n * w)))
    if path == "conv":
        cin, cout = rng.choice([(c[1], c[2]) for c in LAYERS])
        w = rng.choice([16, 32, 48, 64, 96, 128, 144])
        dh = max(3.0, math.sqrt(vox / 4 / (n * w)))
        d = max(2, round(dh * rng.uniform(0.7, 1.4)))
        return {"path": "conv", "n": n, "d": d, "h": max(2, round(dh * dh / d)), "w": w, "cin": cin, "cout": cout}
    d = max(4, round(dh * rng.uniform(0.7, 1.4) / 4) * 4)
    return {"path": path, "n": n, "d": d, "h": max(4, round(dh * dh / d / 4) * 4), "w": w}


# ---- work -------------------------------------------------------------------------------
def _macs(case):
    vox = case["n"] * case["d"] * case["h"] * case["w"]
    return sum(27 * ci * co * vox / s ** 3 for _, ci, co, _, s in LAYERS)


def work(case):
    p = case["path"]
    if p == "flow":
        cells = case["nx"] * case["ny"] * case["nz"]
        b = STORE_BYTES[case["storage"]]
        out = 8 if case["storage"] == "fp64" else 4
        # per step every population is read and written once, and each cell's flag is read
        return {"bytes": cells * (case["steps"] * (38 * b + 1) + 19 * b + 4 * out), "flops": 250.0 * cells * case["steps"]}
    if p == "sweep":
        cells = sum(q["nx"] * q["ny"] * q["nz"] for q in _sweep_params(case, 0))
        b = STORE_BYTES[case["storage"]]
        out = 8 if case["storage"] == "fp64" else 4
        return {"bytes": cells * (case["steps"] * (38 * b + 1) + 19 * b + 4 * out), "flops": 250.0 * cells * case["steps"]}
    if p == "reference":
        cells, q = case["nx"] * case["ny"] * case["nz"], case["q"]
        return {"bytes": cells * (case["steps"] * (8 * q + 1) + 16), "flops": 14.0 * q * cells * case["steps"]}
    vox = case["n"] * case["d"] * case["h"] * case["w"]
    if p == "conv":
        ci, co = case["cin"], case["cout"]
        # x, dy in; y, dx out; weights in, their gradient out
        return {"bytes": vox * 2.0 * (2 * ci + 2 * co) + 27 * ci * co * 6.0, "flops": 6.0 * 27 * ci * co * vox}
    weights = sum(27 * ci * co + co for _, ci, co, _, _ in LAYERS)
    if p == "forward":
        return {"bytes": vox * 64.0 + 2.0 * weights, "flops": 2 * _macs(case)}
    # the first layer needs no gradient with respect to its input
    return {"bytes": vox * (64.0 + 16 + 1) + 36.0 * weights, "flops": 6 * _macs(case) - 2.0 * 27 * 256 * vox}


# ---- inputs -----------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _smooth_velocity(case, seed, mean):
    """Velocity (3, nz, ny, nx), FP32: `mean` plus a few long waves of amplitude about 0.03."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed)
    ax = [torch.arange(n, device="cuda", dtype=torch.float32) * (2 * math.pi / n) for n in (nx, ny, nz)]
    u = torch.empty((3, nz, ny, nx), device="cuda")
    for c in range(3):
        u[c] = mean[c]
        for _ in range(2):
            k, ph, a = rng.integers(1, 4, 3), rng.uniform(0, 2 * math.pi, 3), rng.uniform(0.01, 0.02)
            w = [torch.sin(float(k[i]) * ax[i] + float(ph[i])) for i in range(3)]
            u[c] += float(a) * w[2][:, None, None] * w[1][None, :, None] * w[0][None, None, :]
    return u


def _equilibrium(d, rho, u, v, w):
    """feq of direction d."""
    cu = CX[d] * u + CY[d] * v + CZ[d] * w
    return WGT[d] * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * (u * u + v * v + w * w))


def _flow_inputs(case, seed):
    """Initial populations (19, nz, ny, nx) and the parameters of a flow case."""
    rng = np.random.default_rng(seed + 1)
    porous = case["kind"] == "porous"
    n = np.array([case["nx"], case["ny"], case["nz"]], np.float64)
    q = {"u_in": 0.04, "accel": (0.0, 0.0, 0.0)}
    if porous:
        q["accel"] = (1e-6, 0.0, 0.0) if case["accel"] == "x" else (8e-7, -5e-7, 3e-7)
        count = max(3, round(200 * float(np.prod(n)) / 512 ** 3))
        r = rng.uniform(6.0, 16.0, (count, 1)) * min(1.0, float(n.min()) / 64)
        q["spheres"] = np.concatenate([rng.uniform(0, 1, (count, 3)) * n, r], axis=1)
    else:
        q["radius"] = float(n[1:].min() * rng.uniform(0.1, 0.13))
        q["center"] = (float(n[0] * rng.uniform(0.25, 0.35)), float(n[1] * rng.uniform(0.45, 0.55)), float(n[2] * rng.uniform(0.45, 0.55)))
        q["amp"], q["omega"] = 0.8 * q["radius"], 2 * math.pi / 2000.0
    u = _smooth_velocity(case, seed, (0.0, 0.0, 0.0) if porous else (q["u_in"], 0.0, 0.0))
    f = torch.empty((19, *u.shape[1:]), device="cuda", dtype=torch.float64 if case["storage"] == "fp64" else torch.float32)
    for d in range(19):
        f[d] = _equilibrium(d, 1.0, u[0], u[1], u[2])
    q["f"] = f
    return q


def _rates(case):
    tau = case["tau"]
    return 1.0 / tau, 1.0 / (0.5 + TRT_LAMBDA / (tau - 0.5)) if case["coll"] == "TRT" else 1.0 / tau


def _fields(n, storage):
    dt = torch.float64 if storage == "fp64" else torch.float32
    return torch.empty(n, dtype=dt, device="cuda"), torch.empty((3, n), dtype=dt, device="cuda")


def _prepare_flow(case, seed):
    q = _flow_inputs(case, seed)
    om_p, om_m = _rates(case)
    channel = case["kind"] != "porous"
    faces = ("inlet", case["outlet"], "wall", "wall", "wall", "wall") if channel else PERIODIC
    face_u = [(q["u_in"], 0.0, 0.0)] + [(0.0, 0.0, 0.0)] * 5 if channel else None
    d = Domain(case["nx"], case["ny"], case["nz"], collision=case["coll"], storage=case["storage"], faces=faces,
               omega_p=om_p, omega_m=om_m, face_u=face_u, accel=q["accel"], compute_force=case["force"])
    if channel:
        d.add_sphere(q["center"], q["radius"], moving=case["kind"] == "moving")
    else:
        d.add_spheres(q["spheres"])
    d.init_equilibrium()
    d.set_populations(q.pop("f"))
    rho, vel = _fields(d.N, case["storage"])
    return {"case": case, "d": d, "rho": rho, "vel": vel, "q": q}


def _sphere_pose(q, t):
    cx, cy, cz = q["center"]
    return abi.make_pose(center=(cx, cy + q["amp"] * math.sin(q["omega"] * t), cz),
                         vel=(0.0, q["amp"] * q["omega"] * math.cos(q["omega"] * t), 0.0))


def _run_flow(s):
    case, d, q = s["case"], s["d"], s["q"]
    first = d.step_count + 1
    if case["kind"] == "moving":
        for n in range(first, first + case["steps"]):
            d.update_body(_sphere_pose(q, n - 1.0), _sphere_pose(q, n - 0.5))
            d.step(1)
    else:
        d.step(case["steps"])
    d.macros_into(s["rho"], s["vel"][0], s["vel"][1], s["vel"][2])
    out = {"rho": s["rho"], "vel": s["vel"]}
    if case["force"]:  # the record a run keeps, in the precision of its populations
        h = d.force_history(first, case["steps"])
        out["force"] = h if case["storage"] == "fp64" else h.astype(np.float32)
    return out


def _sweep_params(case, seed):
    """Sizes are the case's own (a sweep is laid out once), bodies and rates the seed's."""
    sizes, rng = np.random.default_rng(case["count"]), np.random.default_rng(seed + 7)
    out = []
    for _ in range(case["count"]):
        nx, n = int(sizes.choice((48, 64, 96))), int(sizes.choice((32, 48)))
        r = float(rng.uniform(3.0, 8.0))
        c = (float(rng.uniform(nx / 4, 3 * nx / 4)), float(rng.uniform(n / 4, 3 * n / 4)), float(rng.uniform(n / 4, 3 * n / 4)))
        re = math.exp(rng.uniform(math.log(5.0), math.log(80.0)))
        out.append({"nx": nx, "ny": n, "nz": n, "r": r, "center": c, "tau": 0.5 + 3.0 * 0.05 * 2.0 * r / re,
                    "seed": int(rng.integers(1 << 30))})
    return out


def _sweep_populations(p, storage):
    u = _smooth_velocity(p, p["seed"], (0.05, 0.0, 0.0))
    f = torch.empty((19, *u.shape[1:]), device="cuda", dtype=torch.float64 if storage == "fp64" else torch.float32)
    for d in range(19):
        f[d] = _equilibrium(d, 1.0, u[0], u[1], u[2])
    return f


def _prepare_sweep(case, seed):
    doms = []
    for p in _sweep_params(case, seed):
        d = Domain(p["nx"], p["ny"], p["nz"], collision="BGK", storage=case["storage"],
                   faces=("inlet", "pressure", "wall", "wall", "wall", "wall"), omega_p=1.0 / p["tau"],
                   face_u=[(0.05, 0.0, 0.0)] + [(0.0, 0.0, 0.0)] * 5, force_history=64)
        d.add_sphere(p["center"], p["r"])
        d.init_equilibrium()
        d.set_populations(_sweep_populations(p, case["storage"]))
        doms.append(d)
    b = Batch(doms)
    b.capture(case["steps"])
    rho, vel = _fields(sum(d.N for d in doms), case["storage"])
    return {"case": case, "batch": b, "doms": doms, "rho": rho, "vel": vel}


def _run_sweep(s):
    s["batch"].replay(1)
    at = 0
    for d in s["doms"]:
        v = s["vel"][:, at:at + d.N]
        d.macros_into(s["rho"][at:at + d.N], v[0], v[1], v[2])
        at += d.N
    return {"rho": s["rho"], "vel": s["vel"]}


def _reference_inputs(case, seed):
    f32 = np.float32
    R, U = f32(case["radius"]), f32(0.05)
    nu = U * (f32(2) * R) / f32(case["reynolds"])
    tau_p = f32(0.5) + f32(3) * nu
    tau_m = f32(0.5) + f32(TRT_LAMBDA) / (tau_p - f32(0.5))
    n = case["nx"] * case["ny"] * case["nz"]
    u = (U * (f32(1) + f32(0.2) * (f32(2) * np.random.default_rng(seed).random(n, dtype=f32) - f32(1)))).astype(f32)
    fe = 0.154 * float(U) / (2 * case["radius"])
    return {"om_p": float(f32(1) / tau_p), "om_m": float(f32(1) / tau_m), "U": float(U), "u": u, "n": n,
            "xc": 0.25 * case["nx"] + 0.25, "yc": 0.5 * case["ny"] + 0.25, "amp": 0.4 * case["radius"], "w": 2 * math.pi * fe}


def _cylinder_pose(q, t):
    f32 = np.float32
    y, vy = q["yc"] - q["amp"] * math.sin(q["w"] * t), -q["amp"] * q["w"] * math.cos(q["w"] * t)
    return abi.make_pose(center=(q["xc"], float(f32(y)), 0.0), vel=(0.0, float(f32(vy)), 0.0))


def _prepare_reference(case, seed):
    q = _reference_inputs(case, seed)
    d = Domain(case["nx"], case["ny"], case["nz"], mode="reference", collision=case["coll"], omega_p=q["om_p"],
               omega_m=q["om_m"], u_inf=(q["U"], 0.0, 0.0), q=case["q"])
    d.add_body(abi.make_body(abi.BODY_CYLINDER_Z, (q["xc"], q["yc"], 0.0), radius=case["radius"], moving=True))
    d.init_equilibrium(rho=np.ones(q["n"]), u=q.pop("u").astype(np.float64), v=np.zeros(q["n"]), w=np.zeros(q["n"]))
    rho, vel = _fields(d.N, "fp32")
    return {"case": case, "d": d, "q": q, "rho": rho, "vel": vel}


def _run_reference(s):
    d, q = s["d"], s["q"]
    first = d.step_count + 1
    aero = np.zeros((s["case"]["steps"], 6), np.float32)
    for k in range(s["case"]["steps"]):
        t = first + k - 1.0
        d.update_body(_cylinder_pose(q, t), _cylinder_pose(q, t + 0.5))
        d.step(1)
        aero[k] = d.force(first + k)
    d.macros_into(s["rho"], s["vel"][0], s["vel"][1], s["vel"][2])
    return {"rho": s["rho"], "vel": s["vel"], "force": aero}


# ---- the warm-start network ---------------------------------------------------------------
def _conv_inputs(case, seed):
    g = _gen(seed)
    shape = (case["n"], case["d"], case["h"], case["w"])
    ci, co = case["cin"], case["cout"]
    return {"x": torch.relu(torch.randn((*shape, ci), device="cuda", generator=g)).bfloat16(),
            "w": (torch.randn((27, co, ci), device="cuda", generator=g) * math.sqrt(2.0 / (27 * ci))).bfloat16(),
            "b": 0.1 * torch.randn(co, device="cuda", generator=g),
            # the gradient as it leaves this layer's own ReLU: about half of it zero
            "dy": torch.relu(1e-3 * torch.randn((*shape, co), device="cuda", generator=g)).bfloat16()
            * torch.randn((*shape, co), device="cuda", generator=g).sign().bfloat16()}


def _prepare_conv(case, seed):
    q = _conv_inputs(case, seed)
    ci, co = case["cin"], case["cout"]
    dy = q["dy"]
    return {"case": case, **q, "ops": unet_mod.Ops(), "y": torch.empty_like(dy), "dx": torch.empty_like(q["x"]),
            "wt": torch.empty((27, ci, co), dtype=torch.bfloat16, device="cuda"),
            "dw": torch.zeros((27, co, ci), device="cuda"), "db": torch.zeros(co, device="cuda")}


def _run_conv(s):
    c, o = s["case"], s["ops"]
    shape, ci, co = (c["n"], c["d"], c["h"], c["w"]), c["cin"], c["cout"]
    o.conv(s["x"], s["w"], s["b"], s["y"], shape, ci, co, True)
    s["dw"].zero_()
    s["db"].zero_()
    o.bwd_weight(s["x"], s["dy"], s["dw"], shape, ci, co)
    o.bias_grad(s["dy"], s["db"], shape[0] * shape[1] * shape[2] * shape[3], co)
    o.flip(s["w"], s["wt"], ci, co)
    o.conv(s["dy"], s["wt"], None, s["dx"], shape, co, ci, False)
    o.relu_bwd(s["dx"], s["x"])  # through the ReLU that made x
    return {"y": s["y"], "dx": s["dx"], "dw": s["dw"], "db": s["db"]}


def _net_inputs(case, seed):
    """Features of ellipsoid channels (mask, distance, Reynolds number, position), normalised
    target fields, fluid mask, He-normal weights with small biases."""
    n, d, h, w = case["n"], case["d"], case["h"], case["w"]
    rng = np.random.default_rng(seed + 3)
    ax = [(torch.arange(k, device="cuda", dtype=torch.float32) + 0.5) / k for k in (d, h, w)]
    x = torch.zeros((n, d, h, w, 16), device="cuda")
    for i in range(n):
        c, s = rng.uniform(0.3, 0.7, 3), rng.uniform(0.1, 0.25, 3)
        r = torch.sqrt(sum(((a - float(c[k])) / float(s[k])).square().reshape([-1 if j == k else 1 for j in range(3)])
                           for k, a in enumerate(ax)))
        x[i, ..., 0] = (r <= 1).float()
        x[i, ..., 1] = torch.clamp((r - 1) * 0.4, -1, 4)
        x[i, ..., 2] = float(rng.uniform(-1, 1))
        x[i, ..., 3], x[i, ..., 4], x[i, ..., 5] = ax[2][None, None, :], ax[1][None, :, None], ax[0][:, None, None]
    mask = (x[..., 0] == 0).to(torch.uint8)
    g = _gen(seed)
    target = torch.stack([0.2 * x[..., 1], 1 - x[..., 0], 0.1 * x[..., 4], 0.1 * x[..., 5]], dim=-1)
    target = target + 0.05 * torch.randn(target.shape, device="cuda", generator=g)
    params = {}
    for name, ci, co, relu, _ in LAYERS:
        used = 6 if name == "e1a" else ci
        wt = rng.standard_normal((27, co, ci)) * math.sqrt((2.0 if relu else 1.0) / (27 * used))
        if name == "e1a":
            wt[:, :, 6:] = 0
        if name == "head":
            wt[:, 4:] = 0
        params[name + ".w"] = wt.astype(np.float32)
        params[name + ".b"] = (0.05 * rng.standard_normal(co) * (np.arange(co) < 4 if name == "head" else 1)).astype(np.float32)
    cw = torch.ones(4, device="cuda")
    return {"x": x.bfloat16(), "mask": mask, "target": target, "params": params, "cw": cw}


def _prepare_net(case, seed):
    q = _net_inputs(case, seed)
    net = unet_mod.UNet3D(16, params=q.pop("params"))
    return {"case": case, "net": net, **q, "count": float(q["mask"].sum())}


def _run_forward(s):
    return s["net"].forward(s["x"])


def _run_train(s):
    net = s["net"]
    out = net.forward(s["x"])
    net.loss_and_grad(s["target"], s["mask"], s["cw"], s["count"])
    net.zero_grad()
    net.backward(net.D["out"])
    net.adam_step(lr=1e-3)
    return {"out": out, "weights": net.Wb}


PREPARE = {"flow": _prepare_flow, "sweep": _prepare_sweep, "reference": _prepare_reference, "conv": _prepare_conv,
           "forward": _prepare_net, "train": _prepare_net}
RUN = {"flow": _run_flow, "sweep": _run_sweep, "reference": _run_reference, "conv": _run_conv, "forward": _run_forward,
       "train": _run_train}


def prepare(case, seed):
    return PREPARE[case["path"]](case, seed)


def run(state):
    return RUN[state["case"]["path"]](state)


# ---- results in 64 bits -------------------------------------------------------------------
def _moments(f, accel=(0.0, 0.0, 0.0), cs=(CX, CY, CZ)):
    rho = f.sum(0)
    u = []
    for c, a in zip(cs, accel):
        j = torch.zeros_like(rho)
        for d, k in enumerate(c):
            if k:
                j += k * f[d]
        u.append(j / rho + 0.5 * a)
    return rho, u


def _collided(f, rho, u, om_p, om_m, trt, accel):
    p = torch.empty_like(f)
    usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    force = any(accel)
    F = [rho * a for a in accel]
    uF = sum(a * b for a, b in zip(u, F)) if force else 0.0
    for d in range(0, 18, 2):
        w = WGT[d]
        cu = CX[d] * u[0] + CY[d] * u[1] + CZ[d] * u[2]
        ev, od = w * rho * (1 + 4.5 * cu * cu - 1.5 * usq), 3 * w * rho * cu
        se = so = 0.0
        if force:
            cF = CX[d] * F[0] + CY[d] * F[1] + CZ[d] * F[2]
            se, so = w * (9 * cu * cF - 3 * uF), 3 * w * cF
        fp, fm = 0.5 * (f[d] + f[d + 1]), 0.5 * (f[d] - f[d + 1])
        om = om_m if trt else om_p
        a = fp - om_p * (fp - ev) + (1 - 0.5 * om_p) * se
        b = fm - om * (fm - od) + (1 - 0.5 * om) * so
        p[d], p[d + 1] = a + b, a - b
    p[18] = f[18] - om_p * (f[18] - WGT[18] * rho * (1 - 1.5 * usq))
    if force:
        p[18] += (1 - 0.5 * om_p) * WGT[18] * (-3 * uF)
    return p


def _coords(shape):
    return [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5).reshape([-1 if j == k else 1 for j in range(3)])
            for k, n in enumerate(shape)][::-1]  # x, y, z


def _inside_sphere(shape, center, r, periodic):
    nz, ny, nx = shape
    d2 = 0.0
    for a, c, n in zip(_coords(shape), center, (nx, ny, nz)):
        e = a - c
        if periodic:
            e = torch.where(e > 0.5 * n, e - n, torch.where(e < -0.5 * n, e + n, e))
        d2 = d2 + e * e
    return d2 <= r * r


def _wall_speed(pose):
    """The rigid translation of a body (its angular velocity is zero here)."""
    return tuple(float(v) for v in pose.vel)


def _exact_flow_steps(f, steps, solid, faces, u_in, om_p, om_m, trt, accel, lever, pose=None, solid_at=None, first=1):
    """Config-mode steps in plain torch; returns populations, solid mask, forces (steps, 6)."""
    shape = f.shape[1:]
    X = _coords(shape)
    f[:, solid] = torch.tensor(WGT, dtype=torch.float64, device="cuda")[:, None]
    forces = []
    for n in range(first, first + steps):
        uw = (0.0, 0.0, 0.0)
        if pose is not None:
            was, solid = solid, solid_at(n)
            half = pose(n - 0.5)
            uw, lever = _wall_speed(half), [float(c) for c in half.center]
            fresh = was & ~solid
            for d in range(19):
                f[d, fresh] = _equilibrium(d, 1.0, *uw)
                f[d, solid] = WGT[d]
        rho, u = _moments(f, accel)
        p = _collided(f, rho, u, om_p, om_m, trt, accel)
        usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
        F = torch.zeros(6, dtype=torch.float64, device="cuda")
        for d in range(19):
            c, o = (CX[d], CY[d], CZ[d]), OPP[d]
            if d == 18:
                f[d] = p[d]
                continue
            sh = dict(shifts=(c[2], c[1], c[0]), dims=(0, 1, 2))
            link = torch.roll(solid, **sh)
            wall = p[o] - 6 * WGT[o] * rho * sum(-a * b for a, b in zip(c, uw))
            v = torch.where(link, wall, torch.roll(p[d], **sh))
            link &= ~solid
            for axis in (2, 1, 0):  # z, y, x: the x face's rule stands at edges and corners
                if c[axis] == 0 or faces[2 * axis] == "periodic":
                    continue
                kind = faces[2 * axis + (0 if c[axis] > 0 else 1)]
                at = [slice(None)] * 3
                at[2 - axis] = 0 if c[axis] > 0 else -1
                at = tuple(at)
                link[at] = False
                if kind == "inlet":
                    val = rho[at] * _equilibrium(d, 1.0, u_in, 0.0, 0.0)
                elif kind == "outflow":
                    val = p[d][at]
                elif kind == "pressure":
                    cu = (c[0] * u[0] + c[1] * u[1] + c[2] * u[2])[at]
                    val = -p[o][at] + 2 * WGT[d] * (1 + 4.5 * cu * cu - 1.5 * usq[at])
                else:
                    val = p[o][at]
                v[at] = val
            f[d] = v
            if lever is not None:
                t = torch.where(link, p[o] + v, torch.zeros((), dtype=torch.float64, device="cuda"))
                fx = [-t * k for k in c]
                r = [X[k] - 0.5 * c[k] - lever[k] for k in range(3)]
                F += torch.stack([fx[0].sum(), fx[1].sum(), fx[2].sum(), (r[1] * fx[2] - r[2] * fx[1]).sum(),
                                  (r[2] * fx[0] - r[0] * fx[2]).sum(), (r[0] * fx[1] - r[1] * fx[0]).sum()])
        del p
        forces.append(F)
    return f, solid, torch.stack(forces)


def _field_values(f, solid, accel):
    f[:, solid] = torch.tensor(WGT, dtype=torch.float64, device="cuda")[:, None]
    rho, u = _moments(f, accel)
    rho[solid] = 0
    for c in u:
        c[solid] = 0
    return rho.reshape(-1), torch.stack([c.reshape(-1) for c in u])


def _exact_flow(case, seed):
    q = _flow_inputs(case, seed)
    om_p, om_m = _rates(case)
    f = q.pop("f").double()
    shape = f.shape[1:]
    channel = case["kind"] != "porous"
    solid_at = None
    if channel:
        faces = ("inlet", case["outlet"], "wall", "wall", "wall", "wall")
        solid = _inside_sphere(shape, q["center"], q["radius"], False)
        lever = list(q["center"])
        if case["kind"] == "moving":
            def solid_at(n):
                return _inside_sphere(shape, list(_sphere_pose(q, n - 1.0).center), q["radius"], False)
    else:
        faces = PERIODIC
        solid = torch.zeros(tuple(shape), dtype=torch.bool, device="cuda")
        for x, y, z, r in q["spheres"]:
            solid |= _inside_sphere(shape, (x, y, z), r, True)
        lever = list(q["spheres"][0][:3])
    pose = (lambda t: _sphere_pose(q, t)) if case["kind"] == "moving" else None
    f, solid, F = _exact_flow_steps(f, case["steps"], solid, faces, q["u_in"], om_p, om_m, case["coll"] == "TRT",
                                    q["accel"], lever if case["force"] else None, pose, solid_at)
    rho, vel = _field_values(f, solid, q["accel"])
    out = {"rho": rho, "vel": vel}
    if case["force"]:
        out["force"] = F
    return out


def _exact_sweep(case, seed):
    rhos, vels = [], []
    for p in _sweep_params(case, seed):
        f = _sweep_populations(p, case["storage"]).double()
        solid = _inside_sphere(f.shape[1:], p["center"], p["r"], False)
        om = 1.0 / p["tau"]
        f, solid, _ = _exact_flow_steps(f, case["steps"], solid, ("inlet", "pressure", "wall", "wall", "wall", "wall"), 0.05,
                                        om, om, False, (0.0, 0.0, 0.0), None)
        rho, vel = _field_values(f, solid, (0.0, 0.0, 0.0))
        rhos.append(rho)
        vels.append(vel)
    return {"rho": torch.cat(rhos), "vel": torch.cat(vels, dim=1)}


def _lattice(q):
    if q == 19:
        return CX, CY, CZ, WGT
    corners = ((1, 1, 1), (-1, -1, -1), (1, 1, -1), (-1, -1, 1), (1, -1, 1), (-1, 1, -1), (-1, 1, 1), (1, -1, -1))
    return (CX[:18] + tuple(c[0] for c in corners) + (0,), CY[:18] + tuple(c[1] for c in corners) + (0,),
            CZ[:18] + tuple(c[2] for c in corners) + (0,), tuple([2 / 27] * 6 + [1 / 54] * 12 + [1 / 216] * 8 + [8 / 27]))


def _exact_reference(case, seed):
    """The reference's step: every node collides, z wraps, bounce-back at the links with the
    wall speed of the half-step pose, moving-wall inlet and y walls, anti-bounce-back outlet."""
    q = _reference_inputs(case, seed)
    nx, ny, nz, nq = case["nx"], case["ny"], case["nz"], case["q"]
    cx, cy, cz, wgt = _lattice(nq)
    w = [float(np.float32(v)) for v in wgt]
    opp = [d ^ 1 for d in range(nq - 1)] + [nq - 1]
    om_p, om_m, U = q["om_p"], q["om_m"], q["U"]
    u0 = torch.from_numpy(q["u"].astype(np.float64)).cuda().reshape(nz, ny, nx)

    def feq(d, rho, u):
        cu = cx[d] * u[0] + cy[d] * u[1] + cz[d] * u[2]
        return w[d] * rho * (1 + 3 * cu + 4.5 * cu * cu - 1.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]))

    zero = torch.zeros_like(u0)
    f = torch.stack([feq(d, 1.0, (u0, zero, zero)) for d in range(nq)])
    X = _coords((nz, ny, nx))
    x32 = [torch.from_numpy((np.arange(n, dtype=np.float32) + np.float32(0.5))).cuda() for n in (nx, ny)]
    R2 = np.float32(case["radius"])
    forces = []
    for k in range(case["steps"]):
        pn, ph = _cylinder_pose(q, float(k)), _cylinder_pose(q, k + 0.5)
        dx = x32[0] - torch.tensor(pn.center[0], dtype=torch.float32, device="cuda")
        dy = x32[1] - torch.tensor(pn.center[1], dtype=torch.float32, device="cuda")
        plane = (dx * dx)[None, :] + (dy * dy)[:, None] <= torch.tensor(R2 * R2, device="cuda")
        solid = plane[None].expand(nz, ny, nx)
        rho, u = _moments(f, cs=(cx, cy, cz))
        p = torch.empty_like(f)
        for d in range(nq):
            o = opp[d]
            e, eo = feq(d, rho, u), feq(o, rho, u)
            if case["coll"] == "TRT":
                p[d] = f[d] - om_p * 0.5 * (f[d] + f[o] - e - eo) - om_m * 0.5 * (f[d] - f[o] - e + eo)
            else:
                p[d] = f[d] - om_p * (f[d] - e)
        usq = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
        F = torch.zeros(6, dtype=torch.float64, device="cuda")
        links = {}
        for d in range(nq):
            sh = dict(shifts=(cz[d], cy[d], cx[d]), dims=(0, 1, 2))
            v = torch.roll(p[d], **sh)
            for axis, c in ((2, cx[d]), (1, cy[d])):  # outside in x or y: the node's own value
                if c:
                    at = [slice(None)] * 3
                    at[axis] = 0 if c > 0 else -1
                    v[tuple(at)] = p[d][tuple(at)]
            o = opp[d]
            if d != nq - 1:  # links (x, o) with a solid at x + c_o = x - c_d; never across the z ends
                link = torch.roll(solid, **sh) & ~solid
                if cz[d]:
                    link = link.clone()
                    link[0 if cz[d] > 0 else -1] = False
                uy = float(ph.vel[1])
                v = torch.where(link, p[o] - 6 * w[o] * rho * (cy[o] * uy), v)
                links[o] = link
            f[d] = v
        for d in range(nq):
            o = opp[d]
            for at, on in (((slice(None), slice(None), 0), cx[d] > 0), ((slice(None), 0), cy[d] > 0), ((slice(None), -1), cy[d] < 0)):
                if on:
                    f[d][at] = p[o][at] + 6 * w[d] * rho[at] * (cx[d] * U)
            if cx[d] < 0:
                at = (slice(None), slice(None), -1)
                cu = (cx[d] * u[0] + cy[d] * u[1] + cz[d] * u[2])[at]
                f[d][at] = -p[o][at] + 2 * w[d] * rho[at] * (1 + 4.5 * cu * cu - 1.5 * usq[at])
        r = [X[0] - ph.center[0], X[1] - ph.center[1], X[2] - ph.center[2]]
        for d, link in links.items():
            t = torch.where(link, p[d] + f[opp[d]], zero)
            fx = [t * cx[d], t * cy[d], t * cz[d]]
            F += torch.stack([fx[0].sum(), fx[1].sum(), fx[2].sum(), (r[1] * fx[2] - r[2] * fx[1]).sum(),
                              (r[2] * fx[0] - r[0] * fx[2]).sum(), (r[0] * fx[1] - r[1] * fx[0]).sum()])
        forces.append(F)
    rho, u = _moments(f, cs=(cx, cy, cz))
    return {"rho": rho.reshape(-1), "vel": torch.stack([c.reshape(-1) for c in u]), "force": torch.stack(forces)}


def _shifted(xp, tap, shape):
    """The padded activations read at one of the 27 taps."""
    n, d, h, w = shape
    z, y, x = tap // 9, (tap // 3) % 3, tap % 3
    return xp[:, z:z + d, y:y + h, x:x + w]


def _conv64(x, w):
    """3x3x3 convolution, zero padding, channels last; w (27, cout, cin)."""
    shape = x.shape[:4]
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    y = torch.zeros((*shape, w.shape[1]), dtype=torch.float64, device="cuda")
    for t in range(27):
        y += _shifted(xp, t, shape) @ w[t].T
    return y


def _conv64_backward(x, w, dy, need_dx=True):
    shape = x.shape[:4]
    xp = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1, 1, 1))
    g = dy.reshape(-1, dy.shape[-1])
    dw = torch.stack([g.T @ _shifted(xp, t, shape).reshape(-1, x.shape[-1]) for t in range(27)])
    dx = _conv64(dy, w.flip(0).transpose(1, 2)) if need_dx else None
    return dx, dw, g.sum(0)


def _exact_conv(case, seed):
    q = {k: v.double() for k, v in _conv_inputs(case, seed).items()}
    y = torch.relu(_conv64(q["x"], q["w"]) + q["b"])
    dx, dw, db = _conv64_backward(q["x"], q["w"], q["dy"])
    return {"y": y, "dx": dx * (q["x"] > 0), "dw": dw, "db": db}


def _pool(x):
    n, d, h, w, c = x.shape
    return x.reshape(n, d // 2, 2, h // 2, 2, w // 2, 2, c).mean(dim=(2, 4, 6))


def _up(x):
    return x.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)


class _Net64:
    """The network's forward and backward pass in 64 bits (BF16 working weights as given)."""

    def __init__(self, params):
        self.w = {k[:-2]: torch.from_numpy(v).cuda().bfloat16().double() for k, v in params.items() if k.endswith(".w")}
        self.b = {k[:-2]: torch.from_numpy(v).cuda().double() for k, v in params.items() if k.endswith(".b")}
        self.saved, self.grads = {}, {}

    def layer(self, name, x):
        y = _conv64(x, self.w[name]) + self.b[name]
        y = y if name == "head" else torch.relu(y)
        self.saved[name] = (x, y)
        return y

    def forward(self, x):
        f = self.layer
        s1 = f("e1b", f("e1a", x))
        s2 = f("e2b", f("e2a", _pool(s1)))
        b3 = f("e3b", f("e3a", _pool(s2)))
        a5 = f("d2b", f("d2a", torch.cat([_up(b3), s2], -1)))
        return f("head", f("d1b", f("d1a", torch.cat([_up(a5), s1], -1))))

    def back(self, name, g):
        x, y = self.saved.pop(name)
        g = g if name == "head" else g * (y > 0)
        dx, self.grads[name + ".w"], self.grads[name + ".b"] = _conv64_backward(x, self.w[name], g, name != "e1a")
        return dx

    def backward(self, g):
        b = self.back
        g = b("d1a", b("d1b", b("head", g)))
        g5, s1 = 8 * _pool(g[..., :32]), g[..., 32:]
        g = b("d2a", b("d2b", g5))
        g3, s2 = 8 * _pool(g[..., :64]), g[..., 64:]
        s2 = s2 + _up(b("e3a", b("e3b", g3))) / 8
        s1 = s1 + _up(b("e2a", b("e2b", s2))) / 8
        b("e1a", b("e1b", s1))


def _exact_forward(case, seed):
    q = _net_inputs(case, seed)
    return _Net64(q["params"]).forward(q["x"].double())


def _exact_train(case, seed):
    q = _net_inputs(case, seed)
    net = _Net64(q["params"])
    out = net.forward(q["x"].double())
    g = torch.zeros_like(out)
    g[..., :4] = 2 * (out[..., :4] - q["target"].double()) * q["mask"].double()[..., None] / float(q["mask"].sum())
    net.backward(g)
    weights = {}
    for name in net.w:
        w, dw = torch.from_numpy(q["params"][name + ".w"]).cuda().double(), net.grads[name + ".w"]
        weights[name] = w - 1e-3 * dw / (dw.abs() + 1e-8)  # the first step of Adam
    return {"out": out, "weights": weights}


EXACT = {"flow": _exact_flow, "sweep": _exact_sweep, "reference": _exact_reference, "conv": _exact_conv,
         "forward": _exact_forward, "train": _exact_train}


def exact(case, seed):
    return EXACT[case["path"]](case, seed)
