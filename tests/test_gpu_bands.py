"""Band-limited filters (k-space top-hat, Gaussian) on the fused transforms, which
leave out the tiles of modes that the filter zeroes: ComputeTs's shells and
find_HII_bubbles against cuFFT's full transforms, over grids whose widest band
is the whole spectrum, part of it, and one tile (box sizes from small cells to
cells larger than the largest radius).

T_S and T_K within 1e-4 relative (the parity tolerance), flags in at most 1e-4
of the cells."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _grids(w, n_hist):
    from meraxes_gb300 import synthetic as syn

    st = syn.initial_state(w.params, w.redshifts[0])
    st.update(syn.FieldGenerator(w).inputs(w.snapshots[-1], n_hist))
    return st


@pytest.mark.parametrize("filter_type", [1, 2])
@pytest.mark.parametrize("D,cell", [(24, 0.4), (32, 3.0), (48, 10.0), (64, 0.4), (96, 0.4), (128, 1.5), (192, 0.4)])
def test_band_limited_paths_match_cufft(D, cell, filter_type, monkeypatch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    w = workload("evolve_512", D)
    w.params = dataclasses.replace(w.params, box_size=cell * D, reion_efficiency=31043.3, filter_type=filter_type,
                                   ts_heating_filter_type=filter_type, r_bubble_max_recomb=20.0 + 8 * cell)
    w.fesc, w.snapshots = 0.01, [5]
    out = []
    for transform in ("fused", "cufft"):
        monkeypatch.setenv("MX_TRANSFORM", transform)
        step = ReionGridStep(w.params, w.redshifts, max_work_bytes=40 * 8 * D * D * (D // 2 + 16))
        st = _grids(w, step.n_sfr_histories)
        g = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in st.items()}
        step.ComputeTs(5, g)
        ts = {k: g[k].cpu().numpy() for k in ("TS_box", "Tk_box")}
        step.find_HII_bubbles(5, g)
        out.append((ts, {k: g[k].cpu().numpy() for k in ("xH", "r_bubble")}))
    (ta, fa), (tb, fb) = out
    for k in ta:
        assert np.all(np.isfinite(ta[k]))
        assert np.abs(ta[k] / tb[k] - 1).max() <= 1e-4, k
    assert ((fa["xH"] == 0) != (fb["xH"] == 0)).mean() <= 1e-4
    assert (fa["r_bubble"] != fb["r_bubble"]).mean() <= 1e-4
