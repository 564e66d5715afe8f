"""The line-of-sight remap of Flag_IncludePecVelsFor21cm = 3 (BrightnessTemperature.c:
325-499) on velocities that move sub-cells within a cell, over several cells,
past each other and around the box.  Mode 3 is mode 2 followed by the remap, so
the remap of mode 2's box by the reference's fifty sub-cells, in numpy FP64, has
to give mode 3's box.

Tolerance, of the largest |delta_T| of the box: H(z) here and in the library may
differ by one float ulp, which moves a sub-cell by 6e-8 of its displacement (8
cells at most: 5e-7 cells, each cell receiving from a few cells); the float
positions of the reference's sub-cells, the FP32 counts and the float result
are below 1e-6.  4e-6 in all; with displacements of thousands of cells in one
column (6e-8 x 5000 cells) 2e-3 in that column.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEPS = 50


def _remap(dT, xH, disp):
    """Sub-cell i of cell k, centred at k + (i + 1/2) / 50, moves by the velocity
    interpolated between cell centres; its value goes to the cells it overlaps."""
    D = dT.shape[-1]
    src = np.where((np.abs(dT) >= 1e-7) & (xH >= 1e-7), dT, 0.0).reshape(-1, D).astype(np.float64) / STEPS
    d = disp.reshape(-1, D).astype(np.float64)
    out = np.zeros_like(src)
    rows = np.arange(src.shape[0])[:, None]
    for i in range(STEPS):
        x = (i + 0.5) / STEPS
        if x <= 0.5:
            low = np.roll(d, 1, 1)
            move = low + (x + 0.5) * (d - low)
        else:
            move = d + (x - 0.5) * (np.roll(d, -1, 1) - d)
        lo = x + move - 0.5 / STEPS
        cell = np.floor(lo)
        share = np.clip((cell + 1 - lo) * STEPS, 0.0, 1.0)
        to = (np.arange(D)[None, :] + cell.astype(np.int64)) % D
        np.add.at(out, (rows, to), src * share)
        np.add.at(out, (rows, (to + 1) % D), src * (1 - share))
    return out.reshape(dT.shape)


# columns per block: 1024 / D (30 at 34: the last block of 1156 columns is not
# full; 1 at 1026 would not fit a test)
@pytest.mark.parametrize("D,cells,far", [(2, 0.3, False), (6, 0.05, False), (24, 0.6, False), (34, 3.0, False),
                                         (50, 8.0, False), (34, 0.5, True)])
def test_remap_matches_subcells(D, cells, far):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import dataclasses

    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    w = workload("full_256", D)
    z = np.float32(w.redshifts[1])
    p = w.params
    H = np.float32(3.2407789e-18 * p.hubble_h * np.sqrt(p.omega_m * (1.0 + float(z)) ** 3 + p.omega_lambda))
    cell = p.box_size / p.hubble_h / np.float32(D)
    rng = np.random.default_rng(D)
    disp = rng.uniform(-cells, cells, (D, D, D))
    if far:
        disp[1, 2, :] *= 1e4
    raw = disp * cell * float(H) / ((1.0 + float(z)) ** 2 * (1e5 / 3.086e24))
    shape = (D, D, 2 * (D // 2 + 1))
    vel, deltax = np.zeros(shape, np.float32), np.zeros(shape, np.float32)
    vel[:, :, :D] = raw
    deltax[:, :, :D] = rng.uniform(-0.5, 2.0, (D, D, D))
    xH = np.where(rng.random((D, D, D)) < 0.2, 0.0, rng.random((D, D, D))).astype(np.float32)
    TS = rng.uniform(5.0, 60.0, (D, D, D)).astype(np.float32)

    def run(mode):
        step = ReionGridStep(dataclasses.replace(p, flag_pecvel=mode), w.redshifts)
        g = {"deltax": deltax, "xH": xH, "TS_box": TS, "vel": vel.copy(), "delta_T": np.zeros((D, D, D), np.float32)}
        g = {k: torch.from_numpy(v).cuda() for k, v in g.items()}
        out = step.ComputeBrightnessTemperatureBox(1, g)
        return g["delta_T"].cpu().numpy(), g["vel"].cpu().numpy(), out["volume_ave_Tb"]

    dT2, _, _ = run(2)
    dT3, v, mean = run(3)
    moved = (v[:, :, :D] / H).astype(np.float64) / cell
    want = _remap(dT2, xH, moved)
    top = np.abs(want).max()
    err = np.abs(dT3 - want) / top
    if far:
        assert err[1, 2].max() < 2e-3
        err[1, 2] = 0.0
    assert err.max() < 4e-6
    assert abs(mean - dT3.astype(np.float64).mean()) <= 1e-9 * np.abs(dT3).mean()


# Modes 1 and 2 per cell against FP64 on one velocity mode (whose derivative is
# known), from below to above the cap of 0.2 H and for optical depths from 1e-6
# to 5 (the pairs of floats up to 1/8, FP64 beyond).  The FP32 transform gives
# dv/dx to a few 1e-7 of its largest value; divided by 1 + dv/dx / H >= 1/2:
# 3e-6 relative.  Cells within 1e-5 of the cap may take either side: 1e-5.
@pytest.mark.parametrize("mode,slope", [(1, 0.1), (1, 0.5), (2, 0.0), (2, 0.5)])
def test_cells_match_fp64(mode, slope):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import dataclasses

    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    D = 32
    w = workload("full_256", D)
    p = dataclasses.replace(w.params, flag_pecvel=mode)
    z = float(np.float32(w.redshifts[1]))
    H = 3.2407789e-18 * p.hubble_h * np.sqrt(p.omega_m * (1.0 + z) ** 3 + p.omega_lambda)
    k = 2.0 * np.pi / p.box_size  # velocity_gradient's k, times h
    phase = 2.0 * np.pi * np.arange(D) / D
    rng = np.random.default_rng(5)
    conv = (1.0 + z) ** 2 * (1e5 / 3.086e24)
    shape = (D, D, 2 * (D // 2 + 1))
    vel, deltax = np.zeros(shape, np.float32), np.zeros(shape, np.float32)
    vel[:, :, :D] = slope * H / (k * p.hubble_h) * np.sin(phase) / conv
    deltax[:, :, :D] = rng.uniform(-0.9, 3.0, (D, D, D))
    xH = rng.choice([0.0, 1e-4, 0.3, 1.0], (D, D, D)).astype(np.float32)
    TS = (10.0 ** rng.uniform(-0.7, 3.0, (D, D, D))).astype(np.float32)
    g = {"deltax": deltax, "xH": xH, "TS_box": TS, "vel": vel, "delta_T": np.zeros((D, D, D), np.float32)}
    g = {n: torch.from_numpy(v).cuda() for n, v in g.items()}
    ReionGridStep(p, w.redshifts).ComputeBrightnessTemperatureBox(1, g)
    got = g["delta_T"].cpu().numpy().astype(np.float64)
    h2 = p.hubble_h ** 2
    factor = 27 * (p.omega_m * p.baryon_frac * h2 / 0.023) * np.sqrt(0.15 / (p.omega_m * h2) * (1 + z) / 10)
    T_cmb, ts = 2.728 * (1 + z), TS.astype(np.float64)
    dT = factor * xH.astype(np.float64) * (1 + deltax[:, :, :D].astype(np.float64))
    grad = slope * np.cos(phase)
    if mode == 1:
        want = dT * (1 - T_cmb / ts) / (np.clip(grad, -0.2, 0.2) + 1)
    else:
        tau = dT * (1 + z) / (1000 * ts) / np.abs(grad + 1)
        assert tau.max() > 0.5 and tau[tau > 0].min() < 1e-5
        want = -np.expm1(-tau) * 1000 * (ts - T_cmb) / (1 + z)
    # T_S - T_CMB cancels near equality: its float rounding is on T_S
    scale = np.abs(want) + 1e-7 * np.abs(dT) * T_cmb / np.abs(ts)
    live = scale > 0
    assert np.all(got[~live] == 0)
    err = np.abs(got - want)[live] / scale[live]
    near = np.abs(ts - T_cmb) < 0.05 * T_cmb
    assert err[~near[live]].max() < (1e-5 if mode == 1 else 3e-6)
