"""The x-pass tile sizes that MX_XPASS_THREADS names are the ones that run, as the
context reports them (tiles of 128 threads share a block of 256, so that the block
size does not tell them apart), where the grid has them, and all give the same bits.
At 64^3 with an odd number of radii the last block of 128-thread tiles holds one."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,base", [(32, "plain_64"), (64, "plain_64"), (64, "full_256"), (128, "plain_64"), (48, "plain_64"),
                                    (50, "plain_64")])
def test_named_tile_size_runs(D, base, monkeypatch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300 import synthetic as syn
    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    w = workload(base, D)
    w.params = dataclasses.replace(w.params, reion_efficiency=3000.0)
    n_hist = ReionGridStep(w.params, w.redshifts).n_sfr_histories
    st = syn.initial_state(w.params, w.redshifts[0])
    st.update(syn.FieldGenerator(w).inputs(1, n_hist))
    pow2 = D & (D - 1) == 0
    out = []
    for threads in (128, 256, 512):
        monkeypatch.setenv("MX_XPASS_THREADS", str(threads))
        step = ReionGridStep(w.params, w.redshifts)
        tile = step.fft_x_tile_threads()
        if D == 50:
            assert tile == 0  # cuFFT
        elif not pow2:
            assert tile == 384
        elif threads == 128 and D not in (64, 128):
            assert tile in (256, 512)
        else:
            assert tile == threads
        g = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in st.items()}
        step.find_HII_bubbles(1, g)
        out.append({k: g[k].cpu().numpy() for k in ("xH", "r_bubble", "J_21", "z_at_ionization")})
        step.close()
    for o in out[1:]:
        for k in o:
            assert np.array_equal(out[0][k], o[k]), k
