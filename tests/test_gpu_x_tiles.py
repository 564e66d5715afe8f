"""The x-pass's 128-thread tiles (two to a block of 256, at 64^3 and 128^3), which
the autotuner may pick, against the 256- and 512-thread tiles: the same bits.
Two radii and three fields leave an odd number of tiles at 64^3 (33 x 3 x 1 and
more), so that the last block holds one tile."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,r_max", [(64, 1.2), (64, 20.0), (128, 1.2)])
def test_x_tiles_give_identical_results(D, r_max, monkeypatch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300 import synthetic as syn
    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    w = workload("plain_64", D)
    p = dataclasses.replace(w.params, reion_efficiency=3000.0, r_bubble_max=r_max)
    st = syn.initial_state(p, w.redshifts[0])
    w.params = p
    st.update(syn.FieldGenerator(w).inputs(1))
    out = []
    for threads in (128, 256, 512):
        monkeypatch.setenv("MX_XPASS_THREADS", str(threads))
        step = ReionGridStep(p, w.redshifts)
        assert step.fft_block_sizes()[0] == max(256, threads)
        g = {k: torch.from_numpy(v.copy()).cuda() for k, v in st.items()}
        step.find_HII_bubbles(1, g)
        out.append({k: g[k].cpu().numpy() for k in ("xH", "r_bubble", "J_21", "z_at_ionization")})
    assert 0.0 < out[0]["xH"].mean() < 1.0
    for o in out[1:]:
        for k in o:
            assert np.array_equal(out[0][k], o[k]), k
