"""The work that is timed: the calls a program using this package makes, over the sizes it makes them at.

    listed()             the fixed cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program has in hand before the call (inputs from the seed, on the GPU)
    run(state)           one pass through the public entry points, and its outputs
    work(case)           bytes and operations a pass cannot do without
    exact(case, seed)    the outputs in 64 bits by plain torch, where they have such a value

Kinds of case (key "kind"):
    thermal   GpuThermalContext.advance: one epoch of explicit bioheat substeps
    ablation  GpuAblationContext.advance_substeps: fused bioheat / plateau / damage / char substeps,
              with "plume" also the plume's transport steps in the void domain
    mc_host   run_voxel_mc3d: photon transport from a layer table to numpy maps, the whole host call
    mc_map    denoise.mc_map: an absorbed map on a crater geometry that stays on the device
    denoise   Denoiser.__call__: a low-photon map through the trained network
    train     UNet.forward_backward + adam: one training step of the denoiser
    epoch     CoupledAblationEngine.step_epoch: a whole coupled epoch, laser on or off
"""
import math

import numpy as np
import torch

SUB = 5e-5             # s, thermal substep of every workload
LAYERS = [(9, 16, 16), (27, 16, 16), (27, 16, 32), (27, 32, 32), (27, 32, 64), (27, 64, 64),
          (27, 64, 32), (27, 32, 32), (27, 32, 16), (27, 16, 16)]   # (taps, cin, cout) of the denoiser
LEVEL = [0, 0, 1, 1, 2, 2, 2, 1, 1, 0]                              # resolution level of each
SCALE = 1e4            # the denoiser's map scale


def listed():
    return [
        # the single-epoch stack's grid: the smallest solver call, one epoch of 20 substeps
        dict(name="thermal-64x64x128", kind="thermal", nx=64, ny=64, nz=128, voxel_mm=0.015, substeps=20),
        # the full-resolution grid's epoch of fused substeps, damage and char kinetics on, no plume
        dict(name="ablation-200x200x192", kind="ablation", nx=200, ny=200, nz=192, voxel_mm=0.015, substeps=20,
             damage=True, char=True, plume=False, d_xy=0.0, d_z=0.0, drift=0.0, tau=0.0),
        # the interactive simulator's 'standard' preset (20 um voxels: 138 slices, not a multiple of 4)
        dict(name="plume-150x150x138", kind="ablation", nx=150, ny=150, nz=138, voxel_mm=0.020, substeps=20,
             damage=False, char=True, plume=True, d_xy=1.0, d_z=2.0, drift=0.0, tau=0.0),
        # the full-resolution coupled run's plume: 34 diffusion steps in each of the 20 substeps
        dict(name="plume-200x200x192", kind="ablation", nx=200, ny=200, nz=192, voxel_mm=0.015, substeps=20,
             damage=False, char=True, plume=True, d_xy=22.875, d_z=22.875, drift=0.0, tau=0.0),
        # run_voxel_mc3d at its default-sized grid: a planar stack, fluence tallied, numpy out
        dict(name="mc-host-40x40x50", kind="mc_host", nx=40, ny=40, nz=50, photons=100_000, tilt_deg=22.0),
        # one laser epoch's photons on the full-resolution stack
        dict(name="mc-150k", kind="mc_map", nx=200, ny=200, nz=128, photons=150_000),
        # the denoiser's training targets
        dict(name="mc-1500k", kind="mc_map", nx=200, ny=200, nz=128, photons=1_500_000),
        # a denoised optical epoch at full resolution
        dict(name="denoise-200x200x128", kind="denoise", nx=200, ny=200, nz=128),
        # a step of the denoiser's training at its default grid
        dict(name="train-200x200x128", kind="train", nx=200, ny=200, nz=128),
        # a small coupled run's laser epoch: latency and host work count
        dict(name="epoch-on-48x48x144", kind="epoch", nx=48, ny=48, nz=128, air=16, photons=20_000, laser=True),
        # the full-resolution run: 200 of its 1000 epochs have the laser on, 800 have it off
        dict(name="epoch-on-200x200x192", kind="epoch", nx=200, ny=200, nz=128, air=64, photons=150_000, laser=True),
        dict(name="epoch-off-200x200x192", kind="epoch", nx=200, ny=200, nz=128, air=64, photons=150_000,
             laser=False),
    ]


def draw(rng):
    def size(lo, hi, mult=1):
        v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        return max(mult, int(round(v / mult)) * mult)

    kind = rng.choice(["thermal", "ablation", "ablation", "plume", "plume", "mc_host", "mc_map", "denoise", "train",
                       "epoch", "epoch"])
    if kind == "thermal":
        return dict(kind=kind, nx=size(24, 200), ny=size(24, 200), nz=size(32, 192), voxel_mm=0.015,
                    substeps=rng.choice([1, 7, 20, 20, 40]))
    if kind in ("ablation", "plume"):
        plume = kind == "plume"
        d = math.exp(rng.uniform(math.log(0.5), math.log(25.0)))
        return dict(kind="ablation", nx=size(24, 200), ny=size(24, 200), nz=size(32, 192), voxel_mm=0.015,
                    substeps=rng.choice([1, 5, 20, 20]), damage=rng.random() < 0.5, char=rng.random() < 0.7,
                    plume=plume, d_xy=round(d, 3) if plume else 0.0,
                    d_z=round(d * rng.choice([1.0, 1.0, 2.0]) * 0.5, 3) if plume else 0.0,
                    drift=rng.choice([0.0, 0.0, 15.0]) if plume else 0.0,
                    tau=rng.choice([0.0, 0.0, 0.00875]) if plume else 0.0)
    if kind == "mc_host":
        return dict(kind=kind, nx=size(20, 80), ny=size(20, 80), nz=size(24, 100), photons=size(10_000, 400_000),
                    tilt_deg=rng.choice([0.0, 22.0]))
    if kind == "mc_map":
        return dict(kind=kind, nx=size(64, 200), ny=size(64, 200), nz=128, photons=size(15_000, 1_500_000))
    if kind in ("denoise", "train"):
        return dict(kind=kind, nx=size(32, 200, 4), ny=size(32, 200, 4), nz=size(32, 128, 4))
    return dict(kind=kind, nx=size(40, 200), ny=size(40, 200), nz=128, air=rng.choice([16, 31, 64]),
                photons=size(15_000, 150_000), laser=rng.random() < 0.5)


# ---- inputs ------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _rand(gen, shape, lo=0.0, hi=1.0):
    return torch.rand(shape, generator=gen, device="cuda", dtype=torch.float32) * (hi - lo) + lo


def _body(nx, ny, nz, gen):
    """A layered body as the workloads have it (air on top, dry cuticle, air gap, wet tissue) with a
    crater through the cuticle into the gap: masks, and per-layer draws expanded to grids."""
    dev = "cuda"
    frac = (torch.arange(nz, device=dev, dtype=torch.float32) + 0.5) / nz
    x = (torch.arange(nx, device=dev, dtype=torch.float32) + 0.5) / nx - 0.5
    y = (torch.arange(ny, device=dev, dtype=torch.float32) + 0.5) / ny - 0.5
    c = _rand(gen, (2,), -0.05, 0.05)
    depth = float(_rand(gen, (1,), 0.10, 0.22))
    r2 = ((x[:, None] - c[0]) ** 2 + (y[None, :] - c[1]) ** 2)[:, :, None]
    z = frac[None, None, :]
    top, gap0, gap1 = 0.365, 0.43, 0.53
    crater = (z >= top) & (z < top + depth * torch.clamp(1.0 - r2 / 0.02, min=0.0))
    air = (z < top).expand(nx, ny, nz)
    gap = ((z >= gap0) & (z < gap1)).expand(nx, ny, nz)
    ablated = air | crater
    void = ablated | gap
    dry = ((z >= top) & (z < gap0)).expand(nx, ny, nz) & ~crater
    dry = dry | ((z >= 0.95).expand(nx, ny, nz))
    return dict(r2=r2, z=z, ablated=ablated, void=void, dry=dry, gap=gap, top=top)


def _thermal_fields(case, gen, b):
    """Conduction, heat capacity (raised where the explicit step needs it), source and temperature."""
    nx, ny, nz, h = case["nx"], case["ny"], case["nz"], case["voxel_mm"]
    shape = (nx, ny, nz)
    band = (torch.arange(nz, device="cuda") * 7) // nz
    k = _rand(gen, (7,), 0.2e-3, 0.6e-3)[band].expand(shape)
    rho = _rand(gen, (7,), 1.7e-3, 4.9e-3)[band].expand(shape)
    hollow = b["void"]
    k = torch.where(hollow, torch.full((), 0.026e-3, device="cuda"), k).contiguous()
    rho = torch.where(hollow, torch.full((), 1.206e-6, device="cuda"), rho)
    alpha = 0.35 / (SUB * 3.0 / (h * h))
    rho = torch.maximum(rho, k * (1.0 / alpha)).contiguous()
    glow = torch.exp(-b["r2"] / 0.01) * torch.exp(-torch.clamp(b["z"] - b["top"], min=0.0) / 0.1) * (b["z"] >= b["top"])
    q = (glow * _rand(gen, shape, 20.0, 80.0)).contiguous()
    t0 = (25.0 + 80.0 * glow + _rand(gen, shape, 0.0, 2.0)).contiguous()
    return dict(k=k, rho=rho, q=q, t0=t0)


def _ablation_fields(case, seed):
    gen = _gen(seed)
    shape = (case["nx"], case["ny"], case["nz"])
    b = _body(*shape, gen)
    f = _thermal_fields(case, gen, b)
    wet = ~b["dry"] & ~b["ablated"]
    f["h0"] = torch.where(wet & (f["t0"] > 95.0), _rand(gen, shape, 0.0, 0.5), torch.zeros((), device="cuda"))
    f["chi0"] = torch.where(b["dry"], _rand(gen, shape, 0.0, 0.4), torch.zeros((), device="cuda"))
    f["c0"] = _rand(gen, shape, 0.0, 2.0) * b["void"] * torch.exp(-b["r2"] / 0.05)
    f["dry"], f["ablated"], f["void"] = b["dry"], b["ablated"], b["void"]
    return f


H_EFF, T_AMB, T_ABL, T_VOID = 15e-6, 25.0, 100.0, 350.0
ARR, CHAR = (1.0e4, 5000.0 / 8.314), (1.0e11, 1.75e5 / 8.314)


def _layer_table(seed):
    """Optics of a planar stack, drawn within the ranges of the benchmark's layers."""
    r = np.random.default_rng(int(seed))
    rows = [(0.06, 5, 30, 10, 40, 0.88, 1.56), (0.18, 5, 30, 10, 40, 0.88, 1.56), (0.58, 0.05, 0.5, 10, 20, 0.90, 1.46),
            (0.78, 0.1, 1.0, 1, 5, 0.90, 1.35), (1.00, 0.2, 2.0, 5, 15, 0.93, 1.40)]
    return [dict(z_end=z, mu_a=float(r.uniform(a0, a1)), mu_s=float(r.uniform(s0, s1)), g=g, n=n)
            for z, a0, a1, s0, s1, g, n in rows]


def _network_inputs(case, seed):
    """A noisy absorbed map, its optics, flags and a smoother target map, as a training pair has them."""
    gen = _gen(seed)
    shape = (case["nx"], case["ny"], case["nz"])
    b = _body(*shape, gen)
    band = (torch.arange(case["nz"], device="cuda") * 7) // case["nz"]
    mu_a = _rand(gen, (7,), 0.1, 20.0)[band].expand(shape)
    mu_s = _rand(gen, (7,), 2.0, 40.0)[band].expand(shape)
    zero = torch.zeros((), device="cuda")
    mu_a, mu_s = torch.where(b["void"], zero, mu_a).contiguous(), torch.where(b["void"], zero, mu_s).contiguous()
    flags = (b["ablated"].to(torch.uint8) | (b["dry"].to(torch.uint8) << 1) | (b["void"].to(torch.uint8) << 2))
    glow = torch.exp(-b["r2"] / 0.02) * torch.exp(-torch.clamp(b["z"] - b["top"], min=0.0) / 0.15)
    target = (glow * 2e-4 * (mu_a > 0)).contiguous()
    counts = torch.poisson((target * 15_000.0 * 4.0).contiguous(), generator=gen)
    noisy = (counts / (15_000.0 * 4.0)).contiguous()
    return dict(mu_a=mu_a, mu_s=mu_s, flags=flags.contiguous(), target=target, noisy=noisy)


def _network_params(seed):
    r = np.random.default_rng(1000 + int(seed))
    parts = []
    for t, ci, co in LAYERS:
        w = r.normal(0.0, math.sqrt(2.0 / (t * ci if t == 27 else 108)), size=(t, co, ci))
        if t == 9:
            w[:, :, 12:] = 0.0
        parts += [w.ravel(), r.normal(0.0, 0.02, co)]
    parts += [r.normal(0.0, 0.1, 16), np.zeros(1)]
    return np.concatenate(parts).astype(np.float32)


# ---- prepare / run -----------------------------------------------------------------------------

def prepare(case, seed):
    import bug_defense_b200 as bd
    from bug_defense_b200 import denoise, voxel_mc, workloads
    kind = case["kind"]
    s = dict(case=case, seed=int(seed))
    if kind == "thermal":
        gen = _gen(seed)
        nx, ny, nz, h = case["nx"], case["ny"], case["nz"], case["voxel_mm"]
        f = _thermal_fields(case, gen, _body(nx, ny, nz, gen))
        ctx = bd.GpuThermalContext(nx, ny, nz, h, h, h, SUB, f["k"], f["rho"], H_EFF, T_AMB)
        ctx.set_T(f["t0"])
        ctx.set_Q(f["q"])
        s["ctx"] = ctx
    elif kind == "ablation":
        nx, ny, nz, h = case["nx"], case["ny"], case["nz"], case["voxel_mm"]
        f = _ablation_fields(case, seed)
        pl = dict(D_xy=case["d_xy"], D_z=case["d_z"], vz=case["drift"], tau_linger=case["tau"]) if case["plume"] else None
        ctx = bd.GpuAblationContext(nx, ny, nz, h, h, h, SUB, H_EFF, T_AMB, T_ABL, T_VOID,
                                    arrhenius=ARR if case["damage"] else None, char_params=CHAR if case["char"] else None,
                                    plume_params=pl, plume_dt_policy="subcycle")
        ctx.set_state(f["t0"], f["h0"], torch.zeros_like(f["t0"]), f["chi0"], f["dry"], f["ablated"], f["q"], f["k"],
                      f["rho"], plume=f["c0"] if pl else None, plume_void=f["void"])
        s["ctx"] = ctx
    elif kind == "mc_host":
        s["layers"] = _layer_table(seed)
    elif kind == "mc_map":
        s["sample"] = workloads.crater_sample(int(seed), case["nx"], case["ny"], case["nz"])
        v = s["sample"]
        s["props"] = voxel_mc.pack_props(v["mu_a"], v["mu_s"], v["g"], v["n"], v["mu_a"].device)
    elif kind in ("denoise", "train"):
        v = _network_inputs(case, seed)
        ones = torch.ones_like(v["mu_a"])
        s["props"] = voxel_mc.pack_props(v["mu_a"], v["mu_s"], 0.9 * ones, 1.4 * ones, v["mu_a"].device)
        s.update(noisy=v["noisy"], target=v["target"], flags=v["flags"])
        params = _network_params(seed)
        shape = (case["nx"], case["ny"], case["nz"])
        if kind == "denoise":
            s["den"] = denoise.Denoiser(params)
            s["den"].net(shape, v["noisy"].device)          # a program keeps its network for all its maps
        else:
            s["net"] = denoise.UNet(shape, training=True, params=params)
            s["pred"] = torch.empty(shape, dtype=torch.float32, device="cuda")
    else:
        geo = workloads.full_coupled_run(int(seed) % 1000, nx=case["nx"], ny=case["ny"], nz=case["nz"],
                                         n_plume_air=case["air"], device="cuda")
        kw = workloads.engine_kwargs(geo)
        kw.update(n_photons=case["photons"], seed=int(seed) + 1, tally_fluence=False)
        # one plume for all seeds, so that a pass is the same number of plume steps
        kw["plume_closure"] = dict(kw["plume_closure"], D_xy=22.875, D_z=22.875)
        eng = bd.CoupledAblationEngine(**kw)
        eng.step_epochs(3)                                   # a run under way: plume in the air, a first crater
        if not case["laser"]:
            eng.power = 0.0
        s["eng"] = eng
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "thermal":
        s["ctx"].advance(case["substeps"], 1)
        return dict(T=s["ctx"].get_T_view())
    if kind == "ablation":
        c = s["ctx"]
        c.advance_substeps(case["substeps"], 1)
        out = dict(T=c.T_a, H=c.H_acc)
        if case["damage"]:
            out["Omega"] = c.Omega
        if case["char"]:
            out["chi"] = c.chi
        if case["plume"]:
            out["C"] = c.P_a
        return out
    if kind == "mc_host":
        import bug_defense_b200 as bd
        r = bd.run_voxel_mc3d(power=40.0, n_photons=case["photons"], spot_dia=0.5, theta_inc_deg=case["tilt_deg"],
                              Lx=2.0, Ly=2.0, Lz=1.0, Nx=case["nx"], Ny=case["ny"], Nz=case["nz"],
                              layers_config=s["layers"], base_seed=s["seed"])
        return {key: r[key] for key in ("A_3d", "Q_3d", "Phi_3d", "lateral_escape_z", "ledger")}
    if kind == "mc_map":
        from bug_defense_b200 import denoise
        A, _, ledger = denoise.mc_map(s["sample"], case["photons"], s["seed"], props=s["props"])
        return dict(A=A, ledger=ledger)
    if kind == "denoise":
        return dict(pred=s["den"](s["noisy"], s["props"], s["flags"]))
    if kind == "train":
        net = s["net"]
        net.forward_backward(s["noisy"], s["props"], s["flags"], s["target"], scale=SCALE, pred=s["pred"])
        net.adam(1e-6)                                       # the end of the schedule
        return dict(pred=s["pred"], grads=net.grads(), params=net.params())
    eng = s["eng"]
    d = eng.step_epoch()
    # the device fields behind engine.T, .H_acc, .chi, .Q and the plume, and the epoch's diagnostics
    return dict(T=eng._T, H=eng._H, chi=eng._chi, A=eng._A, C=eng.plume.raw, mu_ext=eng.plume.mu_ext, props=eng._props,
                flags=eng._flags, diag=[d["n_new"], d["n_void"], d["absorbed_frac"], d["plume_tau"],
                                        d["plume_mean_mu_a"]])


# ---- work --------------------------------------------------------------------------------------

def _plume_steps(case):
    """Diffusion steps in each substep: the fewest whose coefficients are all >= 0, with a tenth to spare."""
    h = float(np.float32(case["voxel_mm"]))
    dxy, dz, v = (float(np.float32(case[key])) for key in ("d_xy", "d_z", "drift"))
    rate = 2.0 * (2.0 * dxy + dz) / (h * h) + max(0.0, v) / h
    return max(1, math.ceil(float(np.float32(SUB)) * rate / 0.9 - 1e-9))


def work(case):
    """Every input field once, every output field once; operations of all the steps."""
    n = case["nx"] * case["ny"] * case["nz"]
    kind = case["kind"]
    if kind == "thermal":
        return dict(bytes=n * 20.0, flops=n * 40.0 * case["substeps"])
    if kind == "ablation":
        b, f = 4.0 * 7 + 1.0, 45.0                            # T, H in and out, q, k, rho; flags
        if case["damage"]:
            b, f = b + 8.0, f + 8.0
        if case["char"]:
            b, f = b + 8.0 * 0.11, f + 12.0 * 0.11            # the dry tenth of the body
        total = dict(bytes=n * b, flops=n * f * case["substeps"])
        if case["plume"]:
            void = 0.47 * n
            total["bytes"] += void * 8.0
            total["flops"] += void * 13.0 * case["substeps"] * _plume_steps(case)
        return total
    if kind == "mc_host":
        return dict(bytes=n * (16.0 + 3 * 8.0), flops=case["photons"] * 120 * 60.0)
    if kind == "mc_map":
        return dict(bytes=n * (16.0 + 1.0 + 4.0), flops=case["photons"] * 300 * 60.0)
    if kind in ("denoise", "train"):
        f = sum(2.0 * t * (12 if t == 9 else ci) * co * n / 8 ** lv for (t, ci, co), lv in zip(LAYERS, LEVEL))
        if kind == "denoise":
            return dict(bytes=n * (4.0 + 16.0 + 1.0 + 4.0), flops=f)
        return dict(bytes=n * (4.0 + 16.0 + 1.0 + 4.0 + 4.0), flops=3.0 * f)
    n = case["nx"] * case["ny"] * (case["nz"] + case["air"])
    steps = 20 * 34
    photons = case["photons"] if case["laser"] else 0
    return dict(bytes=n * (37.0 + 90.0), flops=n * 45.0 * 20 + 0.45 * n * 13.0 * steps + photons * 300 * 60.0)


# ---- exact -------------------------------------------------------------------------------------

def _bioheat(T, k, rho, q, h, dt, h_eff, t_amb):
    """One explicit step in float64: harmonic face conductances, insulated sides, convective z faces."""
    div = torch.zeros_like(T)
    for ax in range(3):
        n = T.shape[ax]
        if n == 1:
            continue
        a, b = [slice(None)] * 3, [slice(None)] * 3
        a[ax], b[ax] = slice(0, n - 1), slice(1, n)
        a, b = tuple(a), tuple(b)
        f = 2.0 * k[a] * k[b] / (k[a] + k[b] + 1e-12) * (T[b] - T[a]) / (h * h)
        div[a] += f
        div[b] -= f
    for kk in (0, T.shape[2] - 1):
        Tc, kc = T[:, :, kk], k[:, :, kk]
        div[:, :, kk] += (t_amb - Tc) / (h * (0.5 * h / kc + 1.0 / h_eff))
    return T + dt * (div + q) / rho


def _exact_ablation(case, seed):
    f = {key: v.double() if v.dtype == torch.float32 else v for key, v in _ablation_fields(case, seed).items()}
    h, dt = float(np.float32(case["voxel_mm"])), float(np.float32(SUB))
    he, ta = float(np.float32(H_EFF)), T_AMB
    arr, chp = [tuple(float(np.float32(v)) for v in p) for p in (ARR, CHAR)]
    T, H, chi = f["t0"], f["h0"], f["chi0"]
    om = torch.zeros_like(T)
    abl, dry = f["ablated"], f["dry"]
    wet = ~abl & ~dry
    for _ in range(case["substeps"]):
        Tt = _bioheat(T, f["k"], f["rho"], f["q"], h, dt, he, ta)
        over = wet & (Tt > T_ABL)
        back = wet & ~(Tt > T_ABL) & (H > 0)
        rel = torch.minimum(H, (T_ABL - Tt) * f["rho"])
        H = torch.where(over, H + (Tt - T_ABL) * f["rho"], torch.where(back, H - rel, H))
        Tt = torch.where(over, torch.full_like(Tt, T_ABL), torch.where(back, Tt + rel / f["rho"], Tt))
        Tt = torch.where(abl & (Tt > T_VOID), torch.full_like(Tt, T_VOID), Tt)
        if case["damage"]:
            om = torch.where(abl, om, om + dt * arr[0] * torch.exp(-arr[1] / (Tt + 273.15)))
        if case["char"]:
            new = 1.0 - (1.0 - chi) * torch.exp(-chp[0] * torch.exp(-chp[1] / (Tt + 273.15)) * dt)
            chi = torch.where(dry & ~abl, new, chi)
        T = Tt
    out = dict(T=T, H=H)
    if case["damage"]:
        out["Omega"] = om
    if case["char"]:
        out["chi"] = chi
    if case["plume"]:
        C, V = f["c0"], f["void"]
        n = _plume_steps(case)
        dtp = dt / n
        dxy, dz, v, tau = (float(np.float32(case[key])) for key in ("d_xy", "d_z", "drift", "tau"))
        wx = wy = dtp * dxy / (h * h)
        wb = dtp * dz / (h * h)
        wt = wb + dtp * max(0.0, v) / h
        decay = math.exp(-dtp / tau) if tau > 0.0 else 1.0
        inside = torch.zeros_like(V)
        inside[1:-1, 1:-1, 1:-1] = V[1:-1, 1:-1, 1:-1]
        solid = (~V).double()
        sides = [((slice(0, -2), slice(1, -1), slice(1, -1)), wx), ((slice(2, None), slice(1, -1), slice(1, -1)), wx),
                 ((slice(1, -1), slice(0, -2), slice(1, -1)), wy), ((slice(1, -1), slice(2, None), slice(1, -1)), wy),
                 ((slice(1, -1), slice(1, -1), slice(0, -2)), wb), ((slice(1, -1), slice(1, -1), slice(2, None)), wt)]
        mid = (slice(1, -1),) * 3
        w0 = torch.full_like(C, 1.0 - 2.0 * wx - 2.0 * wy - wb - wt)
        for sl, w in sides:
            w0[mid] += w * solid[sl]
        keep = inside.double() * decay
        for _ in range(n * case["substeps"]):
            N = w0 * C
            m = N[mid]
            for sl, w in sides:
                m.add_(C[sl], alpha=w)
            C = (N * keep).clamp_(min=0.0)
        out["C"] = C
    return out


def _taps(t, taps):
    return (t // 9, (t // 3) % 3, t % 3) if taps == 27 else (t // 3, t % 3, 1)


def _conv(x, w, sign=1):
    """3x3x3 (or 3x3, z packed) convolution of (c, nx, ny, nz) with w[taps][cout][cin], float64."""
    taps, shape = w.shape[0], x.shape[1:]
    xp = torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1))
    out = torch.zeros((w.shape[1], x[0].numel()), dtype=x.dtype, device=x.device)
    for t in range(taps):
        i, j, k = (d if sign > 0 else 2 - d for d in _taps(t, taps))
        out += w[t] @ xp[:, i:i + shape[0], j:j + shape[1], k:k + shape[2]].reshape(x.shape[0], -1)
    return out.view((w.shape[1],) + tuple(shape))


def _wgrad(g, x, taps):
    shape = x.shape[1:]
    xp = torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1))
    gf = g.reshape(g.shape[0], -1)
    out = []
    for t in range(taps):
        i, j, k = _taps(t, taps)
        out.append(gf @ xp[:, i:i + shape[0], j:j + shape[1], k:k + shape[2]].reshape(x.shape[0], -1).T)
    return torch.stack(out)


def _pool(x):
    c, nx, ny, nz = x.shape
    return x.view(c, nx // 2, 2, ny // 2, 2, nz // 2, 2).sum(dim=(2, 4, 6))


def _up(x):
    return x.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)


def _exact_network(case, seed, train):
    v = _network_inputs(case, seed)
    p = torch.from_numpy(_network_params(seed)).cuda().double()
    L, o = [], 0
    for t, ci, co in LAYERS:
        w = p[o:o + t * ci * co].view(t, co, ci)
        o += t * ci * co
        L.append((w, p[o:o + co].view(co, 1, 1, 1)))
        o += co
    hw, hb = p[o:o + 16], p[o + 16]
    fl = v["flags"]
    one = torch.ones((), dtype=torch.float64, device="cuda")
    state = torch.where((fl & 5) != 0, 0.0 * one, torch.where((fl & 2) != 0, 0.5 * one, one))
    noisy, mask = v["noisy"].double() * SCALE, (v["mu_a"] > 0).double()
    f4 = torch.stack([noisy, torch.log1p(v["mu_a"].double()), 0.25 * torch.log1p(v["mu_s"].double()), state])
    fp = torch.nn.functional.pad(f4, (1, 1))
    nz = case["nz"]
    x16 = torch.cat([fp[..., 0:nz], fp[..., 1:nz + 1], fp[..., 2:nz + 2], torch.zeros_like(f4)])
    layer = lambda i, x: torch.relu(_conv(x, L[i][0]) + L[i][1])   # noqa: E731
    a1 = layer(0, x16)
    s0 = layer(1, a1)
    p0 = _pool(s0) / 8
    a3 = layer(2, p0)
    s1 = layer(3, a3)
    p1 = _pool(s1) / 8
    a5 = layer(4, p1)
    a6 = layer(5, a5)
    u7 = layer(6, a6)
    t7 = _up(u7) + s1
    a8 = layer(7, t7)
    u9 = layer(8, a8)
    t9 = _up(u9) + s0
    hd = layer(9, t9)
    pred = (noisy + torch.einsum("c,cxyz->xyz", hw, hd) + hb) * mask
    if not train:
        return dict(pred=pred / SCALE)
    norm = 1.0 / (case["nx"] * case["ny"] * case["nz"])
    res = (pred - v["target"].double() * SCALE) * mask
    dy = 2.0 * res * norm
    G = [None] * 10

    def back(i, g, x, masked=None):
        G[i] = torch.cat([_wgrad(g, x, LAYERS[i][0]).reshape(-1), g.sum(dim=(1, 2, 3))])
        if i == 0:
            return None
        d = _conv(g, L[i][0].transpose(1, 2), sign=-1)
        return d if masked is None else d * (masked > 0)

    head = torch.cat([torch.einsum("cxyz,xyz->c", hd, dy), dy.sum().view(1)])
    dt9 = back(9, dy[None] * hw.view(16, 1, 1, 1) * (hd > 0), t9)
    g8 = back(8, _pool(dt9) * (u9 > 0), a8, a8)
    dt7 = back(7, g8, t7)
    g6 = back(6, _pool(dt7) * (u7 > 0), a6, a6)
    g5 = back(5, g6, a5, a5)
    d4 = back(4, g5, p1)
    g3 = back(3, (dt7 + _up(d4) / 8) * (s1 > 0), a3, a3)
    d2 = back(2, g3, p0)
    g1 = back(1, (dt9 + _up(d2) / 8) * (s0 > 0), a1, a1)
    back(0, g1, x16)
    return dict(pred=pred / SCALE, grads=torch.cat(G + [head]), params=None)


def exact(case, seed):
    """None for photon transport and the epochs that hold it: a photon's history is a chain of
    comparisons of rounded numbers, so the maps of given random streams have no 64-bit value."""
    kind = case["kind"]
    if kind == "thermal":
        gen = _gen(seed)
        f = _thermal_fields(case, gen, _body(case["nx"], case["ny"], case["nz"], gen))
        h = float(np.float32(case["voxel_mm"]))
        T, k, rho, q = (f[key].double() for key in ("t0", "k", "rho", "q"))
        for _ in range(case["substeps"]):
            T = _bioheat(T, k, rho, q, h, float(np.float32(SUB)), float(np.float32(H_EFF)), T_AMB)
        return dict(T=T)
    if kind == "ablation":
        return _exact_ablation(case, seed)
    if kind in ("denoise", "train"):
        return _exact_network(case, seed, kind == "train")
    return None
