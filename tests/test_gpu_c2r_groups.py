"""Grids without a fused transform: the inverse transforms of several radii (or
shells) go through one cuFFT execution.  Groups of one, of a few with a remainder,
and of the most that fit give the same flags and T_S.

Flags may differ in at most 1e-4 of the cells and T_S by 1e-5 relative: cuFFT may
take another kernel for another batch."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [26, 50, 74, 100])
def test_groups_give_the_same_grids(D, monkeypatch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300 import synthetic as syn
    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    w = workload("full_256", D)
    w.params = dataclasses.replace(w.params, reion_efficiency=31043.3)
    w.fesc = 0.01
    out = []
    for spectra in (5, 15, 35, 400):
        monkeypatch.setenv("MX_MAX_BATCH_SPECTRA", str(spectra))
        step = ReionGridStep(w.params, w.redshifts)
        st = syn.initial_state(w.params, w.redshifts[0])
        st.update(syn.FieldGenerator(w).inputs(1, step.n_sfr_histories))
        g = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in st.items()}
        step.ComputeTs(1, g)
        step.find_HII_bubbles(1, g)
        out.append({k: g[k].cpu().numpy() for k in ("xH", "r_bubble", "TS_box")})
        step.close()
    a = out[0]
    assert 0.0 < (a["xH"] == 0).mean() < 1.0
    for b in out[1:]:
        assert np.abs(a["TS_box"] / b["TS_box"] - 1).max() <= 1e-5
        assert ((a["xH"] == 0) != (b["xH"] == 0)).mean() <= 1e-4
        assert (a["r_bubble"] != b["r_bubble"]).mean() <= 1e-4
