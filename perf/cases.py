"""What a user of the solver has it do, as cases that can be timed and compared.

Each case is one call sequence through the public Python interface (``pism_b200.ssa``,
``pism_b200.learned``): the SSA solve in the set-ups it is run in, the consumers of its velocity,
the finite-element solve, and the training and the forward pass of the warm-start network.
``listed()`` gives fixed cases, ``draw(rng)`` one more of the same ranges, ``prepare(case, seed)``
what a program holds before the call, ``run(state)`` one pass, ``work(case)`` the bytes and
operations of a pass (each input read once and each output written once; for the iterative
solves that counts their fields alone, because the number of iterations follows from the data),
and ``exact(case, seed)`` the outputs in 64 bits where they are a closed computation.  A
solve stops at its tolerance, and the network's Adam step changes its parameters, so those have
no such value beyond what is returned here.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pismv0.7.3_b200")


def _package():
    """the package under its import name (its folder's name is no identifier)"""
    if "pism_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("pism_b200", os.path.join(_PKG, "__init__.py"),
                                                      submodule_search_locations=[_PKG])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["pism_b200"] = mod
        spec.loader.exec_module(mod)
    from pism_b200 import learned, ssa, synthetic, verification
    return ssa, learned, synthetic, verification


F64 = torch.float64
SECPERA = 31556925.9747
INPUTS = ("thickness", "surface", "bed", "mask", "tauc", "melange")
# input and output channels and level of the network's ten 3 x 3 convolutions
LAYERS = ((16, 32, 0), (32, 32, 0), (32, 64, 1), (64, 64, 1), (64, 96, 2), (96, 96, 2), (96, 128, 3), (224, 96, 2),
          (160, 64, 1), (96, 32, 0))


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest solve: the reference's plastic-till stream at its default tolerances, where
        # an iteration is a few kernels on a thousand cells
        {"name": "stream_5x201", "kind": "stream", "Mx": 5, "My": 201},
        # the benchmark sheet's set-up on a coarse grid (40 km): a quick look, a spin-up's early steps
        {"name": "fast_101", "kind": "fast", "M": 101, "learned": False},
        # the headline: 801^2 sheet, network warm start, inexact Picard, FP32 inner solves refined in FP64
        {"name": "fast_801", "kind": "fast", "M": 801, "learned": True},
        # the FP64 path that generates training data and judges the fast one
        {"name": "fp64_401", "kind": "fp64", "M": 401},
        # an ensemble's members on one handle, each with its own hardness and yield stress
        {"name": "ensemble_8x401", "kind": "ensemble", "M": 401, "members": 8},
        # StressBalance's 3-D fields after a solve, polythermal ice, as every full update takes them
        {"name": "columns_801x41", "kind": "columns", "Mx": 801, "My": 801, "Mz": 41, "law": "gpbld"},
        # the explicit mass transport step with the velocity
        {"name": "mass_801", "kind": "mass", "Mx": 801, "My": 801},
        # the calving front: strain rates, stresses, the calving step and its time step
        {"name": "front_801", "kind": "front", "Mx": 801, "My": 801},
        # the finite-element solve on the reference's stream (many short CG iterations) ...
        {"name": "fem_stream_5x481", "kind": "fem_stream", "Mx": 5, "My": 481},
        # ... and on its periodic shelf (few iterations on a larger grid)
        {"name": "fem_shelf_241", "kind": "fem_shelf", "Mx": 241, "My": 241},
        # one training step of the warm-start network on the batch it is trained with
        {"name": "train_16x128", "kind": "train", "B": 16, "H": 128, "W": 128},
        # the network's prediction for the 801^2 sheet (its 10 km image)
        {"name": "predict_408", "kind": "predict", "B": 1, "H": 408, "W": 408},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("stream", "fast", "fast", "fp64", "ensemble", "columns", "mass", "front", "fem_stream",
                       "fem_shelf", "train", "predict"))
    if kind == "stream":
        return {"kind": kind, "Mx": rng.randint(3, 9), "My": _log_int(rng, 41, 401)}
    if kind == "fast":
        M = _log_int(rng, 61, 780)
        return {"kind": kind, "M": M, "learned": M >= 301}
    if kind == "fp64":
        return {"kind": kind, "M": _log_int(rng, 61, 401)}
    if kind == "ensemble":
        return {"kind": kind, "M": _log_int(rng, 101, 401), "members": rng.randint(2, 6)}
    if kind == "columns":
        return {"kind": kind, "Mx": _log_int(rng, 31, 801), "My": _log_int(rng, 31, 801), "Mz": rng.randint(5, 41),
                "law": rng.choice(("gpbld", "pb", "isothermal_glen"))}
    if kind in ("mass", "front"):
        return {"kind": kind, "Mx": _log_int(rng, 31, 1201), "My": _log_int(rng, 31, 1201)}
    if kind == "fem_stream":
        return {"kind": kind, "Mx": rng.randint(3, 9), "My": _log_int(rng, 41, 401)}
    if kind == "fem_shelf":
        return {"kind": kind, "Mx": _log_int(rng, 31, 301), "My": _log_int(rng, 31, 301)}
    if kind == "train":
        return {"kind": kind, "B": rng.randint(1, 16), "H": 8 * rng.randint(4, 16), "W": 8 * rng.randint(4, 16)}
    return {"kind": kind, "B": 1, "H": 8 * _log_int(rng, 8, 64), "W": 8 * _log_int(rng, 8, 64)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dev(fields):
    """the fields as a program that keeps its model on the GPU holds them"""
    return {k: torch.tensor(np.asarray(fields[k]), dtype=F64, device="cuda") for k in INPUTS}


def _fast(c):
    """the fast set-up: multigrid, FP32 inner solves, each linear solve as accurate as the last
    relative nu*H change, the whole Picard loop in one graph"""
    return c.copy(pc_type="mg", precision="mixed", ksp_rtol=1e-6, ksp_rtol_adaptive=True, ksp_rtol_factor=1.0,
                  ksp_rtol_max=1e-1, graphs=3, max_iterations_ssafd=5000)


def _stream(case, seed, V):
    """verification test I with a yield stress that varies by some percent along the flow"""
    rng = np.random.Generator(np.random.PCG64(seed))
    g, c, f = V.build_test_i(My=case["My"], Mx=case["Mx"])
    a, b = rng.uniform(0.0, 0.05), rng.uniform(0.0, 2.0 * math.pi)
    i = np.arange(g.Mx)[:, None] / max(1, g.Mx - 1)
    f["tauc"] = f["tauc"] * (1.0 + a * np.cos(2.0 * math.pi * i + b))
    return g, c, f


def _shelf(case, seed, V):
    """verification test J with a thickness that varies by some percent"""
    rng = np.random.Generator(np.random.PCG64(seed))
    g, c, f = V.build_test_j(case["Mx"], case["My"])
    a, b, d = rng.uniform(0.0, 0.03), rng.uniform(0.0, 2.0 * math.pi), rng.uniform(0.0, 2.0 * math.pi)
    x = 2.0 * math.pi * np.arange(g.Mx)[:, None] / g.Mx
    y = 2.0 * math.pi * np.arange(g.My)[None, :] / g.My
    f["thickness"] = f["thickness"] * (1.0 + a * np.cos(x + b) * np.cos(y + d))
    f["surface"] = (1.0 - c.ice_density / c.sea_water_density) * f["thickness"]
    return g, c, f


def _noise(gen, Mx, My, n):
    """a smooth random field of about n x n bumps, standard deviation about one"""
    t = torch.randn((1, 1, n + 3, n + 3), dtype=F64, device="cuda", generator=gen)
    t = torch.nn.functional.interpolate(t, size=(Mx, My), mode="bicubic", align_corners=True)[0, 0]
    return (t - t.mean()) / t.std()


def _geometry(case, seed):
    """an ice sheet with shelves and a calving front on a rough bed, its velocity and its mass
    balance: what the consumers of the velocity read"""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    Mx, My = case["Mx"], case["My"]
    rho, rho_sw = 910.0, 1028.0
    alpha = 1.0 - rho / rho_sw
    bed = -300.0 + 800.0 * _noise(gen, Mx, My, 24)
    i = torch.linspace(-1.0, 1.0, Mx, dtype=F64, device="cuda")[:, None]
    j = torch.linspace(-1.0, 1.0, My, dtype=F64, device="cuda")[None, :]
    s = (1800.0 * (0.75 - i * i - j * j) + 300.0 * _noise(gen, Mx, My, 12)).clamp(min=0.0)
    H = torch.minimum(s - bed, s / alpha).clamp(0.0, 4000.0)
    floating = alpha * H > bed + H + 1.0
    free = H < 0.01
    two, three, four, zero = (torch.full_like(H, v) for v in (2.0, 3.0, 4.0, 0.0))
    mask = torch.where(floating, torch.where(free, four, three), torch.where(free, zero, two))
    surface = torch.where(floating, alpha * H, bed + H)
    speed = 400.0 / SECPERA * (0.2 + i.abs() + j.abs())
    vel = torch.stack([speed * (i + 0.3 * _noise(gen, Mx, My, 16)), speed * (j + 0.3 * _noise(gen, Mx, My, 16))], dim=-1)
    vel = torch.where((free & (mask != 2.0))[..., None], torch.zeros_like(vel), vel).contiguous()
    cmb = 910.0 / SECPERA * (0.3 + 0.5 * _noise(gen, Mx, My, 10))
    bmr = 1.0 / SECPERA * (0.01 + 0.02 * _noise(gen, Mx, My, 10).abs())
    fields = {"thickness": H, "surface": surface, "bed": bed, "mask": mask, "tauc": torch.full_like(H, 5.0e4),
              "melange": torch.zeros_like(H)}
    return fields, vel, cmb, bmr, gen


def _grid(case, Mz=None):
    from pism_b200.config import GridDesc
    L = 2000.0e3
    d = 2.0 * L / max(case["Mx"] - 1, case["My"] - 1)
    z = None if Mz is None else np.linspace(0.0, 4000.0, Mz)
    return GridDesc(case["Mx"], case["My"], 0.5 * d * (case["Mx"] - 1), 0.5 * d * (case["My"] - 1), z=z)


def _enthalpy(fields, Mz, gen):
    """columns that warm towards the bed, some of them temperate there (J/kg)"""
    H = fields["thickness"]
    z = torch.linspace(0.0, 4000.0, Mz, dtype=F64, device="cuda")
    depth = (H[..., None] - z).clamp(min=0.0)
    Ts = 245.0 + 8.0 * _noise(gen, *H.shape, 10)
    T = Ts[..., None] + 0.016 * depth + 2.0 * _noise(gen, *H.shape, 20)[..., None]
    return (2009.0 * (T - 223.15)).contiguous()


def _image(case, seed):
    """a batch of network images with the channels' ranges (thickness, bed, yield stress, hardness,
    grounded, floating, driving stress), targets and weights"""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    B, H, W = case["B"], case["H"], case["W"]
    x = torch.empty((B, H, W, 8), dtype=F64, device="cuda")
    t = torch.empty((B, H, W, 2), dtype=F64, device="cuda")
    for b in range(B):
        thick = (1.2 + 1.0 * _noise(gen, H, W, 6)).clamp(0.0, 4.0)
        icy = (thick > 0).to(F64)
        grounded = icy * (_noise(gen, H, W, 5) > -0.4).to(F64)
        chans = (thick, -0.3 + 0.8 * _noise(gen, H, W, 10), _noise(gen, H, W, 12), 1.9 * icy, grounded, icy - grounded,
                 0.4 * icy * _noise(gen, H, W, 8), 0.4 * icy * _noise(gen, H, W, 8))
        for q, v in enumerate(chans):
            x[b, :, :, q] = v
        t[b, :, :, 0] = 2.5 * icy * _noise(gen, H, W, 6)
        t[b, :, :, 1] = 2.5 * icy * _noise(gen, H, W, 6)
    w = torch.where(x[..., 4] + x[..., 5] > 0, 1.0, 0.2)
    return x.float().contiguous(), t.float().contiguous(), w.float().contiguous()


# ---------------------------------------------------------------------------
# what a program holds, and one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    ssa, learned, synthetic, V = _package()
    kind = case["kind"]
    if kind == "stream":
        g, c, f = _stream(case, seed, V)
        fields = dict(_dev(f), bc_mask=torch.tensor(f["bc_mask"], device="cuda"),
                      bc_values=torch.tensor(f["bc_values"], device="cuda"))
        out = torch.zeros((g.Mx, g.My, 2), dtype=F64, device="cuda")
        return {"kind": "solve", "ssa": ssa.SSAFD(g, c), "fields": fields, "out": out,
                "guess": torch.zeros_like(out), "net": None}
    if kind in ("fast", "fp64"):
        M = case["M"]
        g, c, f, _ = synthetic.build_synthetic(M, 4000.0e3 / (M - 1), seed=300_000 + seed % 1_000_000)
        c = _fast(c) if kind == "fast" else learned.solve_config(c).copy(max_iterations_ssafd=5000)
        s, net, stride = ssa.SSAFD(g, c), None, 2 if M >= 600 else 1
        if case.get("learned"):
            net = learned.UNet.load(max_batch=1, max_h=learned.image_shape(M, M, stride)[0],
                                    max_w=learned.image_shape(M, M, stride)[1])
        out = torch.zeros((M, M, 2), dtype=F64, device="cuda")
        return {"kind": "solve", "ssa": s, "fields": _dev(f), "out": out, "guess": torch.zeros_like(out), "net": net,
                "stride": stride}
    if kind == "ensemble":
        M, members = case["M"], []
        for q in range(case["members"]):
            rng = np.random.Generator(np.random.PCG64([seed, q]))
            g, c, f, _ = synthetic.build_synthetic(M, 4000.0e3 / (M - 1), seed=500_000 + (16 * seed + q) % 1_000_000,
                                                   temperature_c=rng.uniform(-20.0, -2.0),
                                                   tauc_median=rng.uniform(20e3, 200e3))
            members.append(dict(_dev(f), ice_softness=c.ice_softness,
                                velocity=torch.zeros((M, M, 2), dtype=F64, device="cuda")))
        hh, ww = learned.image_shape(M, M, 1)
        return {"kind": kind, "ssa": ssa.SSAFD(g, _fast(c)), "members": members,
                "net": learned.UNet.load(max_batch=1, max_h=hh, max_w=ww)}
    if kind in ("columns", "mass", "front"):
        fields, vel, cmb, bmr, gen = _geometry(case, seed)
        from pism_b200.config import SSAConfig
        st = {"kind": kind, "bmr": bmr.contiguous(), "cmb": cmb.contiguous()}
        if kind == "columns":
            Mz = case["Mz"]
            if case["law"] != "isothermal_glen":
                fields["enthalpy"] = _enthalpy(fields, Mz, gen)
            s = ssa.SSAFD(_grid(case, Mz), SSAConfig(flow_law=case["law"]))
            st["out"] = {k: torch.empty((case["Mx"], case["My"], Mz), dtype=F64, device="cuda")
                         for k in ("u", "v", "w", "strain_heating")}
        else:
            s = ssa.SSAFD(_grid(case), SSAConfig(flow_law="isothermal_glen"))
            st["mask"], st["H"] = fields["mask"], fields["thickness"]
            st["href"] = torch.where(fields["mask"] == 4.0, 20.0, 0.0).to(F64)
        torch.cuda.synchronize()
        s.set_inputs(**fields)
        s.set_initial_guess(vel)
        st["ssa"] = s
        return st
    if kind in ("fem_stream", "fem_shelf"):
        g, c, f = (_stream if kind == "fem_stream" else _shelf)(case, seed, V)
        s = ssa.SSAFEM(g, c)
        d = {k: torch.tensor(f[k], dtype=F64, device="cuda")
             for k in ("thickness", "surface", "bed", "mask", "tauc", "bc_mask", "bc_values")}
        s.set_inputs(**d)
        out = torch.zeros((g.Mx, g.My, 2), dtype=F64, device="cuda")
        return {"kind": "fem", "ssa": s, "out": out, "guess": torch.zeros_like(out)}
    x, t, w = _image(case, seed)
    if kind == "train":
        net = learned.UNet(case["B"], case["H"], case["W"], seed=seed)
        return {"kind": kind, "net": net, "x": x, "t": t, "w": w,
                "grad": torch.empty(net.param_count(), dtype=torch.float32, device="cuda")}
    return {"kind": kind, "net": learned.UNet.load(max_batch=case["B"], max_h=case["H"], max_w=case["W"]), "x": x}


def run(state):
    kind = state["kind"]
    if kind == "solve":
        s = state["ssa"]
        s.set_inputs(**state["fields"])
        if state["net"] is not None:
            sys.modules["pism_b200.learned"].learned_guess(s, state["net"], state["stride"])
        else:
            s.set_initial_guess(state["guess"])
        return s.solve(out=state["out"])
    if kind == "ensemble":
        return state["ssa"].solve_batch(state["members"], net=state["net"], stride=1)[0]
    if kind == "columns":
        return state["ssa"].stress_balance_3d(state["bmr"], out=state["out"])
    if kind == "mass":
        return state["ssa"].mass_continuity_step(0.1 * SECPERA, state["cmb"], state["bmr"])
    if kind == "front":
        s = state["ssa"]
        out = s.strain_rates(state["mask"], device=True)
        out["calving"] = s.eigen_calving(0.1 * SECPERA, 1e17, state["mask"], state["href"], state["H"])
        out["time_step"] = s.eigen_calving_max_timestep(1e17, state["mask"])
        return out
    if kind == "fem":
        state["ssa"].set_initial_guess(state["guess"])
        return state["ssa"].solve(out=state["out"])
    if kind == "train":
        net = state["net"]
        y = net.forward(state["x"])
        loss = net.backward(state["t"], state["w"], grad_out=state["grad"])
        net.adam(1e-3)
        return {"y": y, "loss": loss, "grad": state["grad"]}
    return state["net"].forward(state["x"])


# ---------------------------------------------------------------------------
# the least a pass moves and computes
# ---------------------------------------------------------------------------
def _net_flops(case):
    """multiply-adds of the ten convolutions and the head, as operations, of a forward pass"""
    pix = case["B"] * case["H"] * case["W"]
    return 2.0 * sum(9 * ci * co * pix / 4 ** lev for ci, co, lev in LAYERS) + 2.0 * 64 * pix


def work(case):
    kind = case["kind"]
    if kind in ("fast", "fp64"):     # six fields and the velocity in, the velocity out
        return {"bytes": case["M"] ** 2 * (6 * 8 + 16 + 16), "flops": 0.0}
    if kind == "ensemble":
        return {"bytes": case["members"] * case["M"] ** 2 * (6 * 8 + 16), "flops": 0.0}
    if kind in ("train", "predict"):
        pix, n = case["B"] * case["H"] * case["W"], 9 * sum(ci * co for ci, co, _ in LAYERS)
        if kind == "train":          # input, target, weight, output; parameters, moments and gradient
            return {"bytes": pix * 4 * (8 + 2 + 1 + 2) + n * 4 * 8, "flops": 3.0 * _net_flops(case)}
        return {"bytes": pix * 4 * (8 + 2) + n * 4, "flops": _net_flops(case)}
    N = case["Mx"] * case["My"]
    if kind == "stream":
        return {"bytes": N * (6 * 8 + 8 + 16 + 16 + 16), "flops": 0.0}
    if kind in ("fem_stream", "fem_shelf"):
        return {"bytes": N * (5 * 8 + 8 + 16 + 16 + 16), "flops": 0.0}
    if kind == "columns":            # four fields out; the enthalpy, velocity, mask, thickness, melt rate in
        enth = 0 if case["law"] == "isothermal_glen" else 8 * case["Mz"]
        return {"bytes": N * (4 * 8 * case["Mz"] + enth + 16 + 1 + 8 + 8), "flops": 0.0}
    if kind == "mass":               # velocity, mask, thickness, bed, two mass balances in; four fields out
        return {"bytes": N * (16 + 1 + 8 + 8 + 8 + 8 + 4 * 8), "flops": 0.0}
    # front: velocity and mask in, strain rates and stresses out; mask, Href, thickness in and out
    return {"bytes": N * (16 + 8 + 16 + 24 + 6 * 8), "flops": 0.0}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
def _nb(a, di, dj):
    return torch.roll(a, shifts=(-di, -dj), dims=(0, 1))


def _gradient(case, vel, keep_e, keep_w, keep_n, keep_s):
    """u_x, u_y, v_x, v_y with one-sided differences where a side is dropped"""
    d = 4000.0e3 / max(case["Mx"] - 1, case["My"] - 1)
    nx, ny = keep_e + keep_w, keep_n + keep_s
    dx = torch.where(nx > 0, 1.0 / (d * nx.clamp(min=1.0)), 0.0)
    dy = torch.where(ny > 0, 1.0 / (d * ny.clamp(min=1.0)), 0.0)
    out = []
    for q in (0, 1):
        a = vel[..., q]
        out.append(dx * (keep_w * (a - _nb(a, -1, 0)) + keep_e * (_nb(a, 1, 0) - a)))
        out.append(dy * (keep_s * (a - _nb(a, 0, -1)) + keep_n * (_nb(a, 0, 1) - a)))
    return out


def _sides(flag):
    """1.0 where the flag holds at the east, west, north, south neighbour"""
    return [_nb(flag, di, dj).to(F64) for di, dj in ((1, 0), (-1, 0), (0, 1), (0, -1))]


def _hardness(law, E, depth):
    if law == "isothermal_glen":
        return 3.1689e-24 ** (-1.0 / 3.0)
    p = 910.0 * 9.81 * depth.clamp(min=0.0)
    Tm = 273.15 - 7.9e-8 * p
    Es = 2009.0 * (Tm - 223.15)
    Tpa = torch.where(E < Es, E / 2009.0 + 223.15, Tm) - Tm + 273.15

    def paterson_budd(T):
        return torch.where(T < 263.15, 3.61e-13 * torch.exp(-6.0e4 / (8.31441 * T)),
                           1.73e3 * torch.exp(-13.9e4 / (8.31441 * T)))

    A = paterson_budd(Tpa)
    if law == "gpbld":
        omega = ((E - Es) / 3.34e5).clamp(0.0, 0.01)
        A = torch.where(E < Es, A, paterson_budd(torch.full_like(Tm, 273.15)) * (1.0 + 181.25 * omega))
    return A ** (-1.0 / 3.0)


def _exact_columns(case, seed):
    fields, vel, _, bmr, gen = _geometry(case, seed)
    Mz, H = case["Mz"], fields["thickness"]
    icy = (fields["mask"] == 2.0) | (fields["mask"] == 3.0)
    same = [1.0 - (_nb(icy, di, dj) != icy).to(F64) for di, dj in ((1, 0), (-1, 0), (0, 1), (0, -1))]
    u_x, u_y, v_x, v_y = _gradient(case, vel, *same)
    z = torch.tensor(np.linspace(0.0, 4000.0, Mz), dtype=F64, device="cuda")
    w = -bmr[..., None] - (u_x + v_y)[..., None] * (z - z[0])
    D2 = 0.5 * ((u_x + v_y) ** 2 + u_x ** 2 + v_y ** 2 + 0.5 * (u_y + v_x) ** 2)
    heat = 2.0 * D2[..., None] ** (2.0 / 3.0)
    if case["law"] == "isothermal_glen":
        heat = heat * _hardness(case["law"], None, None)
    else:
        heat = heat * _hardness(case["law"], _enthalpy(fields, Mz, gen), H[..., None] - z)
    top = torch.searchsorted(z, H, right=True).clamp(1, Mz - 1) - 1
    heat = torch.where(torch.arange(Mz, device="cuda") <= top[..., None], heat, 0.0)
    return {"u": vel[..., 0, None].expand(-1, -1, Mz), "v": vel[..., 1, None].expand(-1, -1, Mz), "w": w,
            "strain_heating": heat}


def _exact_mass(case, seed):
    fields, vel, cmb, bmr, _ = _geometry(case, seed)
    H, bed, mask, dt = fields["thickness"], fields["bed"], fields["mask"], 0.1 * SECPERA
    d = 4000.0e3 / max(case["Mx"] - 1, case["My"] - 1)
    icy = (mask == 2.0) | (mask == 3.0)

    def face(q, di, dj):
        a, b = vel[..., q], _nb(vel[..., q], di, dj)
        there = _nb(icy, di, dj)
        return torch.where(icy & there, 0.5 * (a + b), torch.where(icy, a, torch.where(there, b, 0.0)))

    e, w, n, s = face(0, 1, 0), face(0, -1, 0), face(1, 0, 1), face(1, 0, -1)
    div = (e * torch.where(e > 0, H, _nb(H, 1, 0)) - w * torch.where(w > 0, _nb(H, -1, 0), H)) / d
    div = div + (n * torch.where(n > 0, H, _nb(H, 0, 1)) - s * torch.where(s > 0, _nb(H, 0, -1), H)) / d
    ocean = mask == 4.0
    smb, melt = torch.where(ocean, 0.0, cmb / 910.0), torch.where(ocean, 0.0, bmr)
    new = H + dt * (smb - melt - div)
    lost = (-new).clamp(min=0.0)
    new = new.clamp(min=0.0)
    alpha = 1.0 - 910.0 / 1028.0
    floating, free = alpha * new > bed + new + 1.0, new < 0.01
    kg = 910.0 * d * d
    grounded = mask < 3.0
    totals = {"grounded_basal_ice_flux": -(melt * grounded).sum() * kg * dt, "nonneg_rule_flux": lost.sum() * kg,
              "sub_shelf_ice_flux": -(melt * ~grounded).sum() * kg * dt, "surface_ice_flux": smb.sum() * kg * dt,
              "sum_divQ_SIA": torch.zeros((), dtype=F64), "sum_divQ_SSA": None, "Href_to_H_flux": 0.0,
              "H_to_Href_flux": 0.0}   # the divergence's sum cancels: no digits of it are the inputs'
    return {"thickness": new,
            "mask": torch.where(floating, torch.where(free, 4.0, 3.0), torch.where(free, 0.0, 2.0)).to(F64),
            "surface": torch.where(floating, alpha * new, bed + new), "flux_divergence": div,
            "totals": {k: None if v is None else float(v) for k, v in totals.items()}}


def _exact_front(case, seed):
    fields, vel, _, _, _ = _geometry(case, seed)
    icy = (fields["mask"] == 2.0) | (fields["mask"] == 3.0)
    u_x, u_y, v_x, v_y = _gradient(case, vel, *_sides(icy))
    a, b, c = 0.5 * (u_x + v_y), 0.5 * (u_x - v_y), 0.5 * (v_x + u_y)
    q = torch.sqrt(b * b + c * c)
    gamma = 0.5 * (u_x ** 2 + v_y ** 2 + (u_x + v_y) ** 2 + 0.5 * (u_y + v_x) ** 2)
    reg = (1.0 / SECPERA / 1000.0e3) ** 2
    nu = 0.5 * 3.1689e-24 ** (-1.0 / 3.0) * (reg + gamma) ** (-1.0 / 3.0)
    ice = icy[..., None].to(F64)
    # the calving step cuts cells by thresholds: its fields are compared as they come
    return {"edot": torch.stack([a + q, a - q], dim=-1) * ice,
            "stresses": torch.stack([nu * u_x, nu * v_y, 0.5 * nu * (u_y + v_x)], dim=-1) * ice,
            "calving": None, "time_step": None}


def _exact_net(case, seed):
    import torch.nn.functional as Fn
    _, learned, _, _ = _package()
    x, t, w = _image(case, seed)
    train = case["kind"] == "train"
    p = learned.init_params(seed) if train else np.load(learned.DEFAULT_WEIGHTS)["params"]
    p = torch.tensor(p, dtype=F64, device="cuda", requires_grad=train)
    at, weights = 0, []
    for ci, co, _ in LAYERS:
        k = p[at:at + 9 * co * ci].reshape(3, 3, co, ci).permute(2, 3, 0, 1)
        weights.append((k, p[at + 9 * co * ci:at + 9 * co * ci + co]))
        at += 9 * co * ci + co
    head, bias = p[at:at + 64].reshape(2, 32, 1, 1), p[at + 64:at + 66]

    def conv(l, a):
        return Fn.relu(Fn.conv2d(a, weights[l][0], weights[l][1], padding=1))

    def up(a):
        return a.repeat_interleave(2, 2).repeat_interleave(2, 3)

    a = x.double().permute(0, 3, 1, 2)
    e1 = conv(1, conv(0, torch.cat([a, torch.zeros_like(a)], 1)))
    e2 = conv(3, conv(2, Fn.avg_pool2d(e1, 2)))
    e3 = conv(5, conv(4, Fn.avg_pool2d(e2, 2)))
    b = conv(6, Fn.avg_pool2d(e3, 2))
    d3 = conv(7, torch.cat([up(b), e3], 1))
    d2 = conv(8, torch.cat([up(d3), e2], 1))
    d1 = conv(9, torch.cat([up(d2), e1], 1))
    y = Fn.conv2d(d1, head, bias).permute(0, 2, 3, 1)
    if not train:
        return y.detach().contiguous()
    w = w.double()
    loss = (w * ((y - t.double()) ** 2).sum(-1)).sum() / (2.0 * w.sum())
    loss.backward()
    return {"y": y.detach().contiguous(), "loss": float(loss.detach()), "grad": p.grad}


def exact(case, seed):
    _package()
    kind = case["kind"]
    if kind == "columns":
        return _exact_columns(case, seed)
    if kind == "mass":
        return _exact_mass(case, seed)
    if kind == "front":
        return _exact_front(case, seed)
    if kind in ("train", "predict"):
        return _exact_net(case, seed)
    return None
