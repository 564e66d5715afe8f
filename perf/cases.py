"""The work that the performance of this package is measured on.

A case is one call of a public entry point (`meraxes_gb300.api.ReionGridStep`,
`meraxes_gb300.autograd`) on seeded inputs made on the GPU, with the physics of
the package's workloads (`params.workload`): their cell sizes, redshifts, filter
radii, reionization efficiency and escape fraction.

listed()  the cases        draw(rng)  one more of the same ranges
prepare() inputs, the state before the call, and the context
run()     one call and everything that it wrote
work()    bytes and operations that the call cannot do without
exact()   the outputs in 64 bits by plain torch, where a formula gives them
"""
import dataclasses
import math

import numpy as np
import torch

from meraxes_gb300.api import ReionGridStep
from meraxes_gb300.autograd import DeltaT21, PSLoss21, log_bins
from meraxes_gb300.params import growth_factor, sfr_timescale_internal_myr, workload

REION_EFF = 1.0 / 0.15714 * 4000.0 / (1.0 - 0.75 * 0.24)
FESC = 0.01
# grids that a call reads and rewrites: a program hands it new ones (or the
# state that it stepped from) with every snapshot
STATE = ("sfr", "x_e_box_prev", "Tk_box", "N_rec", "z_at_ionization", "J_21_at_ionization", "Gamma12", "vel")


def listed():
    return [
        # the benchmark's snapshot: the whole step of a 512^3 box of an evolving
        # run, as one CUDA graph (what a production run spends its time on)
        {"name": "step_512", "kind": "step", "grid": 512, "base": "evolve_512", "snapshot": 12, "graph": True},
        # the whole step of one box of a parameter study (the batch's largest size)
        {"name": "step_192", "kind": "step", "grid": 192, "base": "full_256", "snapshot": 1, "graph": False},
        # the drop-in for the C driver: the whole step on host grids, copies included
        {"name": "step_host_128", "kind": "step_host", "grid": 128, "base": "full_256", "snapshot": 1},
        # the smallest call: the excursion set of a plain 64^3 box (latency and launches)
        {"name": "bubbles_64", "kind": "bubbles", "grid": 64, "base": "plain_64", "snapshot": 1, "filter": 0,
         "recombinations": 0, "spin": 0},
        # a grid that is no multiple of a power of two, with the Gaussian filter
        {"name": "bubbles_100", "kind": "bubbles", "grid": 100, "base": "full_256", "snapshot": 1, "filter": 2,
         "recombinations": 1, "spin": 0},
        # the excursion set with recombinations and the spin temperature's x_e
        {"name": "bubbles_256", "kind": "bubbles", "grid": 256, "base": "full_256", "snapshot": 1, "filter": 0,
         "recombinations": 1, "spin": 1},
        # the spin temperature of a small and of a large box
        {"name": "spin_96", "kind": "spin", "grid": 96, "base": "evolve_512", "snapshot": 6, "filter": 1},
        {"name": "spin_256", "kind": "spin", "grid": 256, "base": "evolve_512", "snapshot": 10, "filter": 1},
        # forward and backward of the power-spectrum loss (an inference step)
        {"name": "gradient_128", "kind": "gradient", "grid": 128, "base": "diff_256", "snapshot": 1},
        # the 21 cm box with the redshift-space remap
        {"name": "brightness_256", "kind": "brightness", "grid": 256, "base": "full_256", "snapshot": 1, "pecvel": 3},
        # the power spectrum of a box
        {"name": "power_200", "kind": "power", "grid": 200, "base": "full_256", "snapshot": 1},
        # the galaxies of a snapshot into the grids
        {"name": "deposit_256", "kind": "deposit", "grid": 256, "base": "evolve_512", "snapshot": 8,
         "galaxies": 400000},
    ]


def _grid(rng, low, high):
    """An even grid size: most programs take one that transforms well."""
    common = [d for d in (24, 32, 48, 64, 96, 128, 192, 256) if low <= d <= high]
    if rng.random() < 0.6:
        return rng.choice(common)
    return 2 * int(round(0.5 * math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step_host", "bubbles", "bubbles", "bubbles", "spin", "spin", "gradient",
                       "brightness", "power", "deposit"])
    evolving = rng.random() < 0.5
    snap = rng.randint(3, 17) if evolving else 1
    base = "evolve_512" if evolving else "full_256"
    if kind == "step":
        return {"kind": kind, "grid": _grid(rng, 24, 256), "base": base, "snapshot": snap,
                "graph": rng.random() < 0.5}
    if kind == "step_host":
        return {"kind": kind, "grid": _grid(rng, 24, 160), "base": base, "snapshot": snap}
    if kind == "bubbles":
        plain = rng.random() < 0.4
        return {"kind": kind, "grid": _grid(rng, 24, 256), "base": "plain_64" if plain else base,
                "snapshot": 1 if plain else snap, "filter": rng.choice([0, 0, 1, 2]),
                "recombinations": 0 if plain else rng.choice([0, 1, 1]), "spin": 0 if plain else rng.choice([0, 1, 1])}
    if kind == "spin":
        return {"kind": kind, "grid": _grid(rng, 24, 256), "base": base, "snapshot": snap,
                "filter": rng.choice([0, 1, 1, 1, 2])}
    if kind == "gradient":
        return {"kind": kind, "grid": _grid(rng, 24, 160), "base": "diff_256", "snapshot": 1}
    if kind == "brightness":
        return {"kind": kind, "grid": _grid(rng, 24, 256), "base": base, "snapshot": snap, "pecvel": rng.randint(0, 3)}
    if kind == "power":
        return {"kind": kind, "grid": _grid(rng, 24, 300), "base": base, "snapshot": snap}
    return {"kind": kind, "grid": _grid(rng, 24, 256), "base": base, "snapshot": snap,
            "galaxies": int(10 ** rng.uniform(3, 6))}


# ------------------------------------------------------------------ inputs
def _workload(case):
    w = workload(case["base"], case["grid"])
    p = dataclasses.replace(w.params, clumping_factor=2.0)
    kind = case["kind"]
    if case["base"] == "plain_64":
        p.reion_efficiency = 3000.0
        fesc = 1.0
    else:
        p.reion_efficiency = REION_EFF
        fesc = FESC
    if kind == "bubbles":
        p.filter_type, p.flag_recombinations, p.flag_spin_temp = case["filter"], case["recombinations"], case["spin"]
    elif kind == "spin":
        p.ts_heating_filter_type = case["filter"]
    elif kind == "brightness":
        p.flag_pecvel = case["pecvel"]
    elif kind == "gradient":
        p.reion_efficiency, fesc = 1.0, 1.0  # the differentiation workload as it is
    return w, p, fesc


def _waves(D, L):
    kf = 2 * math.pi / L
    k = torch.fft.fftfreq(D, d=1.0 / D, device="cuda") * kf
    kz = torch.arange(D // 2 + 1, device="cuda") * kf
    return (k[:, None, None] ** 2 + k[None, :, None] ** 2) + kz[None, None, :] ** 2


def _field(D, L, gen, smooth=0.0):
    """A Gaussian field of unit variance, P(k) ~ k^-2 exp(-(k / k_Ny)^2)."""
    f = torch.fft.rfftn(torch.randn((D, D, D), generator=gen, device="cuda"))
    k2 = _waves(D, L)
    k2[0, 0, 0] = 1.0
    f *= torch.exp(-0.5 * k2 * ((L / (math.pi * D)) ** 2 + smooth ** 2)) * torch.rsqrt(k2)
    del k2
    f[0, 0, 0] = 0
    f = torch.fft.irfftn(f, s=(D, D, D))
    return f / f.std()


def _padded(real):
    D = real.shape[0]
    out = torch.zeros((D, D, 2 * (D // 2 + 1)), device="cuda")
    out[:, :, :D] = real
    return out


def _stars(delta):
    return torch.where(delta > 0.5, 1e-3 * torch.exp(2.0 * delta), torch.zeros_like(delta))


def _inputs(case, w, p, fesc, n_hist, gen):
    """Grids of one snapshot: density, stars and SFR grown linearly, and the
    state that earlier snapshots of a run leave (the densest cells ionised)."""
    D, snap, kind = p.grid_dim, case["snapshot"], case["kind"]
    z = w.redshifts[snap]
    z_prev = w.redshifts[snap - 1]
    g_norm = growth_factor(w.redshifts[w.snapshots[-1]], p)
    t20 = sfr_timescale_internal_myr(20.0, p)
    base = 0.6 * _field(D, p.box_size, gen)
    delta = torch.clamp(base * (growth_factor(z, p) / g_norm), min=-0.99)
    stars = _stars(delta)
    early = delta > 1.1
    zero, real = torch.zeros_like(delta), {}
    pad = {"deltax": delta, "stars": fesc * stars, "weighted_sfr": fesc * stars / t20, "sfr": stars / t20,
           "N_rec": torch.where(early, 0.05 * delta, zero)}
    if p.flag_spin_temp:
        x_e = torch.clamp(2.5e-4 * (1.0 + 0.5 * delta), min=1e-5)
        pad["x_e_box_prev"] = x_e
        pad["x_e_box"] = x_e
        real["Tk_box"] = 12.0 * torch.pow(1.0 + delta, 2.0 / 3.0)
        real["TS_box"] = torch.clamp(real["Tk_box"] + 5.0, min=2.0)
    real["xH"] = torch.where(early, zero, torch.clamp(1.1 - 0.5 * torch.clamp(delta, min=0), 0.0, 1.0))
    real["z_at_ionization"] = torch.where(early, zero + z_prev, zero - 1.0)
    real["J_21_at_ionization"] = torch.where(early, 0.1 * delta, zero)
    real["Gamma12"] = torch.where(early, 0.05 * delta, zero)
    for name in ("r_bubble", "J_21", "delta_T"):
        real[name] = torch.zeros_like(delta)
    if kind == "brightness":
        v = 50.0 * _field(D, p.box_size, gen, smooth=3.0 * p.box_size / D) * (growth_factor(z, p) / g_norm)
        pad["vel"] = v / (1.0 + z)
    out = {k: _padded(v) for k, v in pad.items()}
    out.update({k: v.contiguous() for k, v in real.items()})
    if p.flag_spin_temp and n_hist > 0 and kind != "brightness":
        hist = torch.zeros((n_hist, out["sfr"].numel()), device="cuda")
        for j in range(min(n_hist, snap + 1)):
            d = torch.clamp(base * (growth_factor(w.redshifts[snap - j], p) / g_norm), min=-0.99)
            hist[j] = _padded(_stars(d) / t20).reshape(-1)
        out["sfr_histories"] = hist
    return out


def _galaxies(case, p, gen):
    """A galaxy list as the deposit reads it: clustered positions, some dead
    galaxies, lognormal masses."""
    n, L = case["galaxies"], p.box_size
    groups = max(1, n // 20)
    centres = L * torch.rand((groups, 3), generator=gen, device="cuda")
    of = torch.randint(0, groups, (n,), generator=gen, device="cuda")
    pos = centres[of] + 0.02 * L * torch.randn((n, 3), generator=gen, device="cuda")
    pos = torch.remainder(pos, L).clamp(0.0, L)
    mass = torch.pow(10.0, torch.randn(n, generator=gen, device="cuda", dtype=torch.float64) - 4.0)
    black = torch.pow(10.0, torch.randn((2, n), generator=gen, device="cuda", dtype=torch.float64) - 5.0)
    kind = torch.multinomial(torch.tensor([0.5, 0.3, 0.1, 0.1], device="cuda"), n, True, generator=gen)
    return {"pos": pos.float().contiguous(), "type": kind.int(), "fesc_weighted_gsm": 0.1 * mass,
            "gross_stellar_mass": mass, "black_hole_mass": black[0].contiguous(),
            "effective_bhm": 0.1 * black[1].contiguous()}


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    w, p, fesc = _workload(case)
    # several boxes share the GPU: room for about sixty filtered spectra each
    D = p.grid_dim
    step = ReionGridStep(p, w.redshifts, max_work_bytes=60 * 8 * D * D * (D // 2 + 16))
    if case.get("graph"):
        step.set_graph()
    s = {"case": case, "step": step, "snapshot": case["snapshot"]}
    if case["kind"] == "deposit":
        n_pad = D * D * 2 * (D // 2 + 1)
        s["galaxies"] = _galaxies(case, p, gen)
        s["grids"] = {k: torch.zeros((D, D, 2 * (D // 2 + 1)), device="cuda") for k in ("stars", "weighted_sfr", "sfr")}
        s["grids"]["sfr_histories"] = torch.rand((step.n_sfr_histories, n_pad), generator=gen, device="cuda")
        s["kept"] = {}  # the call itself shifts the history by a snapshot
        return s
    if case["kind"] == "power":
        x = _field(D, p.box_size, gen)
        s["delta_T"] = (15.0 * torch.exp(0.5 * x) * (x < 1.0)).contiguous()
        return s
    grids = _inputs(case, w, p, fesc, step.n_sfr_histories, gen)
    if case["kind"] == "gradient":
        s["sfr"], s["stars"] = grids.pop("sfr"), grids.pop("stars")
        s["state"], s["edges"], s["params"] = grids, log_bins(step, 20), p
        with torch.no_grad():
            dT = DeltaT21.apply(s["sfr"], s["stars"], torch.tensor(2e40, dtype=torch.float64),
                                torch.tensor(p.nu_xray_gal_threshold, dtype=torch.float64), step, 1, grids)
            _, s["target"], _ = step.ps_loss(dT, s["edges"], [0.0] * 20, grad=False)
        return s
    if case["kind"] == "step_host":
        grids = {k: torch.empty(v.shape, pin_memory=True).copy_(v) for k, v in grids.items()}
        s["arrays"] = {k: v.numpy() for k, v in grids.items()}
    s["grids"] = grids
    changed = {"bubbles": ("N_rec", "z_at_ionization", "J_21_at_ionization", "Gamma12"),
               "spin": ("sfr", "x_e_box_prev", "Tk_box"), "brightness": ("vel",)}.get(case["kind"], STATE)
    s["kept"] = {k: grids[k].clone() for k in changed if k in grids}
    return s


# --------------------------------------------------------------------- run
_WRITTEN = {
    "bubbles": ("xH", "z_at_ionization", "r_bubble", "J_21", "J_21_at_ionization", "Gamma12", "N_rec"),
    "spin": ("x_e_box", "x_e_box_prev", "Tk_box", "TS_box", "sfr"),
    "brightness": ("delta_T", "vel"),
    "deposit": ("stars", "weighted_sfr", "sfr", "sfr_histories"),
}
_WRITTEN["step"] = _WRITTEN["spin"] + _WRITTEN["bubbles"] + ("delta_T",)
_WRITTEN["step_host"] = _WRITTEN["step"]
# the averages of a call, by what it computes
_MEANS = {
    "bubbles": ("volume_weighted_global_xH", "volume_weighted_global_J_21", "mass_weighted_global_xH", "n_radii"),
    "spin": ("volume_ave_J_alpha", "volume_ave_xalpha", "volume_ave_Xheat", "volume_ave_Xion", "volume_ave_TS",
             "volume_ave_TK", "volume_ave_xe", "x_e_ave", "collapse_fraction"),
    "brightness": ("volume_ave_Tb",),
}
_MEANS["step"] = _MEANS["step_host"] = _MEANS["bubbles"] + _MEANS["spin"] + _MEANS["brightness"]


def run(state):
    case, step, snap = state["case"], state["step"], state["snapshot"]
    kind = case["kind"]
    if kind == "power":
        return dict(zip(("k", "power", "error"), step.Compute_PS(state["delta_T"])))
    if kind == "gradient":
        p = state["params"]
        sfr = state["sfr"].detach().requires_grad_(True)
        fesc = torch.tensor(1.0, device="cuda", requires_grad=True)
        lx = torch.tensor(p.lx_gal, dtype=torch.float64, requires_grad=True)
        e0 = torch.tensor(p.nu_xray_gal_threshold, dtype=torch.float64, requires_grad=True)
        dT = DeltaT21.apply(sfr, state["stars"] * fesc, lx, e0, step, 1, state["state"])
        loss = PSLoss21.apply(dT, step, state["edges"], state["target"])
        loss.backward()
        return {"delta_T": dT, "loss": loss.item(), "sfr": sfr.grad, "fesc": fesc.grad, "lx": lx.grad.item(),
                "e0": e0.grad.item()}
    grids = state["grids"]
    # the snapshot's inputs and the state that it steps from
    for name, kept in state["kept"].items():
        grids[name].copy_(kept)
    if kind == "deposit":
        step.construct_baryon_grids(snap, state["galaxies"], grids, 1, 1e-6, 2.0)
        return {k: grids[k] for k in _WRITTEN[kind]}
    if kind == "step":
        means = step.step(snap, grids)
    elif kind == "step_host":
        means = step.step(snap, state["arrays"])
    elif kind == "bubbles":
        means = step.find_HII_bubbles(snap, grids)
    elif kind == "spin":
        means = step.ComputeTs(snap, grids)
    else:
        means = step.ComputeBrightnessTemperatureBox(snap, grids)
    out = {k: grids[k] for k in _WRITTEN[kind] if k in grids}
    out["means"] = {k: means[k] for k in _MEANS[kind]}
    return out


# -------------------------------------------------------------------- work
def work(case):
    """Each grid read once and written once, and each transform's operations
    (5/2 N log2 N of a real transform) and per-cell work."""
    w, p, _ = _workload(case)
    D, kind = p.grid_dim, case["kind"]
    N = float(D) ** 3
    fft = 2.5 * N * math.log2(N)
    radii = len(p.filter_radii())
    G = 3 + bool(p.flag_recombinations) + bool(p.flag_spin_temp)
    S = p.ts_num_filter_steps
    nbytes = flops = 0.0
    if kind in ("bubbles", "step", "step_host"):
        nbytes += 4 * N * (G + 3 + 4 + 2 * bool(p.flag_recombinations))
        flops += fft * G * radii + 20 * N * radii
    if kind in ("spin", "step", "step_host"):
        nbytes += 4 * N * (5 + 4)
        flops += fft * S + N * (14 * S + 200)
    if kind in ("brightness", "step", "step_host"):
        nbytes += 4 * N * 4
        flops += 6 * N
    if kind == "brightness" and case["pecvel"]:
        nbytes += 8 * N
        flops += 2 * fft + 20 * N
    if kind == "power":
        nbytes += 4 * N
        flops += fft + 10 * N
    if kind == "deposit":
        nbytes += case["galaxies"] * 48.0 + 4 * N * 4
        flops += case["galaxies"] * 20.0 + 4 * N
    if kind == "gradient":
        nbytes += 4 * N * (G + 12 + 14)
        flops += fft * (G * radii + 3 * S + 3) + N * (20 * radii + 60 * S + 600)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------- exact
def _k32(D, L):
    """|k| as the filters and the bins take it: float, k = n * float(2 pi / L)."""
    dk = torch.tensor(2.0 * math.pi / L, dtype=torch.float32, device="cuda")
    n = torch.arange(D, device="cuda")
    k = torch.where(n > D // 2, n - D, n).float() * dk
    kz = torch.arange(D // 2 + 1, device="cuda").float() * dk
    return torch.sqrt((k[:, None, None] ** 2 + k[None, :, None] ** 2) + kz[None, None, :] ** 2)


def _exact_bubbles(case, state):
    """find_HII_bubbles with 64-bit transforms and decisions; N_rec has no
    closed form (its recombination table)."""
    w, p, _ = _workload(case)
    D, L, h = p.grid_dim, p.box_size, p.hubble_h
    z = w.redshifts[case["snapshot"]]
    g = {k: v.double()[:, :, :D] for k, v in state["grids"].items() if torch.is_tensor(v) and v.dim() == 3}
    names = ["deltax", "stars", "weighted_sfr"] + ["x_e_box"] * p.flag_spin_temp + ["N_rec"] * p.flag_recombinations
    spectra = {n: torch.fft.rfftn(g[n]) for n in names}
    kmag = _k32(D, float(np.float32(L))).double()
    unit_t = p.unit_length_cm / p.unit_velocity_cm_s
    grav = 6.672e-8 / p.unit_length_cm ** 3 * p.unit_mass_g * unit_t ** 2
    rho = p.omega_m * 3 * (3.2407789e-18 * unit_t) ** 2 / (8 * math.pi * grav)
    pixel = (L / D) ** 3
    xH = torch.ones_like(g["deltax"])
    r_bubble, J21 = torch.zeros_like(xH), torch.zeros_like(xH)
    z_ion, J_ion, gamma = g["z_at_ionization"], g["J_21_at_ionization"], g["Gamma12"]
    radii = p.filter_radii()
    for R in radii:
        last = R == radii[-1]
        f = {}
        for n in names:
            if last:
                f[n] = g[n]
                continue
            x = kmag * float(np.float32(R))
            if p.filter_type == 0:
                W = torch.where(x > 1e-4, 3 * (torch.sin(x) / x ** 3 - torch.cos(x) / x ** 2), torch.ones_like(x))
            elif p.filter_type == 1:
                W = (x * 0.413566994 <= 1).double()
            else:
                W = torch.exp(-(x * 0.643) ** 2 / 2)
            f[n] = torch.fft.irfftn(spectra[n] * W, s=(D, D, D))
        dx = f["deltax"].clamp(min=-1 + 1e-5)
        cut = {n: torch.where(f[n] < 1e-8, torch.zeros_like(dx), f[n]) for n in names if n != "deltax"}
        neutral = 1 - cut["x_e_box"].clamp(max=0.999) if p.flag_spin_temp else torch.ones_like(dx)
        rec = cut["N_rec"] / (1 + dx) if p.flag_recombinations else torch.zeros_like(dx)
        mass = (2 * math.pi) ** 1.5 if p.rtom_filter_type == 1 else 4 / 3 * math.pi
        coll = cut["stars"] / (mass * R ** 3 * rho * (1 + dx)) * (4 / 3) * math.pi * R ** 3 / pixel * p.reion_efficiency
        ionised = coll > neutral * (1 + rec)
        jk = ((1 + z) ** 2 / (4 * math.pi) * p.alpha_uv * 6.6262e-27 * 1e21 * R * p.unit_length_cm
              * p.nion_phot_per_bary / 1.6726e-24 * p.unit_mass_g / p.unit_length_cm ** 3 / unit_t)
        gk = ((1 + z) ** 2 * R * (p.unit_length_cm / h) * 6.3e-18 * p.alpha_uv / (p.alpha_uv + 2.75) / 1e-12
              * (p.unit_mass_g / unit_t) * (p.unit_length_cm / h) ** -3 * p.nion_phot_per_bary / 1.6726e-24)
        j = cut["weighted_sfr"] * jk / pixel
        first = ionised & (xH > 1e-5)
        J21 = torch.where(first, j, J21)
        if p.flag_recombinations:
            gamma = torch.where(first, cut["weighted_sfr"] * gk / pixel, gamma)
        if last:
            xH = torch.where(~ionised & (xH > 1e-5), (neutral - coll).clamp(0, 1), xH)
        xH = torch.where(ionised, torch.zeros_like(xH), xH)
        r_bubble = torch.where(ionised, torch.full_like(xH, R), r_bubble)
        new = (xH < 1e-5) & (z_ion < 0)
        z_ion = torch.where(new, torch.full_like(xH, z), z_ion)
        J_ion = torch.where(new, j * p.gamma_halo_bias, J_ion)
    return {"xH": xH, "z_at_ionization": z_ion, "r_bubble": r_bubble, "J_21": J21, "J_21_at_ionization": J_ion,
            "Gamma12": gamma, "N_rec": None, "means": None}


def _exact_brightness(case, state):
    w, p, _ = _workload(case)
    D, mode = p.grid_dim, case["pecvel"]
    z = w.redshifts[case["snapshot"]]
    g = {k: v.double()[:, :, :D] for k, v in state["grids"].items() if torch.is_tensor(v) and v.dim() == 3}
    omb = p.omega_m * p.baryon_frac
    h2 = p.hubble_h ** 2
    factor = 27 * (omb * h2 / 0.023) * math.sqrt(0.15 / (p.omega_m * h2) * (1 + z) / 10)
    T_cmb = 2.728 * (1 + z)
    dT = factor * g["xH"] * (1 + g["deltax"])
    dT = dT * ((1 + z) / (1000 * g["TS_box"])) if mode > 1 else dT * (1 - T_cmb / g["TS_box"])
    if not mode:
        return {"delta_T": dT, "vel": None, "means": {"volume_ave_Tb": dT.mean()}}
    H = 3.2407789e-18 * p.hubble_h * math.sqrt(p.omega_m * (1 + z) ** 3 + p.omega_lambda)
    v = (1 + z) * g["vel"] * (1000 * 100 / 3.086e24) * (1 / (1 + z)) ** -1
    kz = torch.arange(D // 2 + 1, device="cuda").double() * (2 * math.pi / p.box_size)
    grad = torch.fft.irfftn(torch.fft.rfftn(v) * p.hubble_h * 1j * kz, s=(D, D, D))
    if mode == 1:
        dT = dT / (grad.clamp(-0.2 * H, 0.2 * H) / H + 1)
    else:
        dT = (1 - torch.exp(-dT / (grad / H + 1).abs())) * 1000 * (g["TS_box"] - T_cmb) / (1 + z)
    if mode == 3:
        # fifty sub-cells of every cell, each moved by the interpolated velocity
        # and shared over the cells that it overlaps
        cw = p.box_size / p.hubble_h / D
        src = torch.where((dT.abs() >= 1e-7) & (g["xH"] >= 1e-7), dT, torch.zeros_like(dT)) / 50
        low, high = (v.roll(1, 2) / H, v / H), (v / H, v.roll(-1, 2) / H)
        col = torch.arange(D, device="cuda").expand(D, D, D)
        dT = torch.zeros_like(dT)
        for i in range(50):
            x = (i + 0.5) / 50
            a, b, t = (*low, x + 0.5) if x <= 0.5 else (*high, x - 0.5)
            left = x - 0.01 + (a + t * (b - a)) / cw
            cell = torch.floor(left)
            share = ((cell + 1 - left) * 50).clamp(0, 1)
            to = (col + cell.long()) % D
            dT.scatter_add_(2, to, src * share)
            dT.scatter_add_(2, (to + 1) % D, src * (1 - share))
    return {"delta_T": dT, "vel": _padded(v.float()).double(), "means": {"volume_ave_Tb": dT.mean()}}


def _exact_power(case, state):
    p = _workload(case)[1]
    D, L = p.grid_dim, p.box_size / p.hubble_h
    dT = state["delta_T"].double()
    power = torch.fft.rfftn((dT - dT.mean()) * (L ** 3 / D ** 3)).abs() ** 2
    kmag = _k32(D, L).reshape(-1)
    dk = np.float32(2 * math.pi / L)
    edges, top = [], dk
    while top < dk * np.float32(D):
        edges.append(top)
        top = np.float32(top * np.float32(1.35))
    edges = torch.tensor(np.array(edges, np.float32), device="cuda")
    b = torch.bucketize(kmag, edges, right=True)
    n = len(edges)
    k = kmag.double()

    def total(x):
        return torch.bincount(b, weights=x, minlength=n + 1)[:n]

    count = total(torch.ones_like(k))
    mean = total(k ** 3 * power.reshape(-1) / (2 * math.pi ** 2 * L ** 3)) / count
    return {"k": total(k) / count, "power": mean, "error": mean / torch.sqrt(count)}


def _exact_deposit(case, state):
    w, p, _ = _workload(case)
    D, g = p.grid_dim, state["galaxies"]
    i = torch.round(g["pos"].double() / p.box_size * D).long()
    i = torch.where(i > D - 1, torch.zeros_like(i), i)
    cell = (i[:, 0] * D + i[:, 1]) * D + i[:, 2]
    live = g["type"] <= 2
    hole = torch.where(g["black_hole_mass"] >= 1e-6, g["effective_bhm"], torch.zeros_like(g["effective_bhm"]))
    z1 = w.redshifts[case["snapshot"]] + 1
    hubble = 3.2407789e-18 * p.unit_length_cm / p.unit_velocity_cm_s
    time = p.reion_sfr_timescale / (hubble * math.sqrt(p.omega_m * z1 ** 3 + p.omega_k * z1 ** 2 + p.omega_lambda))

    def grid(x):
        flat = torch.zeros(D ** 3, dtype=torch.float64, device="cuda")
        flat.index_add_(0, cell[live], x[live])
        out = torch.zeros((D, D, 2 * (D // 2 + 1)), dtype=torch.float64, device="cuda")
        out[:, :, :D] = flat.reshape(D, D, D)
        return out

    return {"stars": grid(g["fesc_weighted_gsm"] + hole),
            "weighted_sfr": grid(g["fesc_weighted_gsm"] + hole * 2.0 / p.alpha_uv) / time,
            "sfr": grid(g["gross_stellar_mass"]) / time, "sfr_histories": None}


def exact(case, seed):
    """None where the outputs come from tables without a formula (the
    frequency integrals of the spin temperature) or from a whole model."""
    how = {"bubbles": _exact_bubbles, "brightness": _exact_brightness, "power": _exact_power,
           "deposit": _exact_deposit}.get(case["kind"])
    return how(case, prepare(case, seed)) if how else None
