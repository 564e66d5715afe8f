"""The frequency-integral tables of ComputeTs built on the device (freq_tables.cu)
against the oracle's (QUADPACK QAG and Brent in C), through the averages that
they enter linearly: X-ray heating, ionisation and J_alpha.

Cases: the X-ray threshold below the helium edge, at its default and above most
shells' unit optical depth (every shell, some, or none shares the lower limit),
a spectral index that is not 1, the first snapshot (no earlier collapse
fraction), a box whose collapse fraction reaches the neutral floor, and a mean
x_e at which the optical depth is not solved for.

Tolerance 1e-5 relative: the tables are FP64 on both sides with the same
quadrature steps; the FP32 coefficients and shell sums contribute about 1e-6.
A quadrature that stopped a bisection earlier or later would differ by up to
its own tolerance of 1e-2.
"""
import dataclasses

import numpy as np
import pytest

from cases import Case, REION_EFF, initial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("snapshot,E0,alpha,stars,x_e", [
    (6, 20.0, 1.0, 1.0, None), (6, 500.0, 1.0, 1.0, None), (6, 2500.0, 1.0, 1.0, None), (12, 500.0, 1.5, 1.0, None),
    (0, 500.0, 1.0, 1.0, None), (19, 300.0, 0.6, 100.0, None), (6, 500.0, 1.0, 1.0, 0.99995)])
def test_tables_match_oracle(snapshot, E0, alpha, stars, x_e, tables_dir):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300 import synthetic as syn
    from meraxes_gb300.api import ReionGridStep
    from oracle import OracleBackend

    w = Case("tables", "evolve_512", 16, {"reion_efficiency": REION_EFF, "clumping_factor": 2.0,
                                          "nu_xray_gal_threshold": E0, "spec_index_xray_gal": alpha},
             fesc=0.01, snapshots=[snapshot]).workload()
    orc = OracleBackend(w.params, w.redshifts, tables_dir)
    gpu = ReionGridStep(w.params, w.redshifts)
    sa = initial(w, orc.n_sfr_histories)
    sa.update(syn.FieldGenerator(w).inputs(snapshot, orc.n_sfr_histories))
    sa["stars"] *= np.float32(stars)
    if x_e is not None:
        sa["x_e_box_prev"][:, :, :16] = np.float32(x_e)
    sb = {k: torch.from_numpy(v.copy()).cuda() for k, v in sa.items()}
    ga = orc.ComputeTs(snapshot, sa)
    gb = gpu.ComputeTs(snapshot, sb)
    assert ga["volume_ave_Xheat"] != 0 and ga["volume_ave_Xion"] != 0
    for name in ("volume_ave_Xheat", "volume_ave_Xion", "volume_ave_J_alpha", "collapse_fraction"):
        assert gb[name] == pytest.approx(ga[name], rel=1e-5), name
