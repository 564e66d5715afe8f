"""The SFR-history operations of ComputeTs on the padded sfr grid, several in one
pass: the grid that ComputeTs leaves is the oracle's, padding included.  Both add
products of floats in the same order; a C compiler may fuse a product and a sum,
an ulp (1.2e-7) for each of up to four, hence 5e-7 relative."""
import numpy as np
import pytest

from cases import Case, REION_EFF, initial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,snapshot", [(16, 0), (16, 1), (16, 5), (22, 8), (24, 12), (32, 19)])
def test_sfr_grid_is_the_oracles(D, snapshot, tables_dir):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300 import synthetic as syn
    from meraxes_gb300.api import ReionGridStep
    from oracle import OracleBackend

    w = Case("sfr_ops", "evolve_512", D, {"reion_efficiency": REION_EFF}, fesc=0.01, snapshots=[snapshot]).workload()
    orc = OracleBackend(w.params, w.redshifts, tables_dir)
    gpu = ReionGridStep(w.params, w.redshifts)
    sa = initial(w, orc.n_sfr_histories)
    sa.update(syn.FieldGenerator(w).inputs(snapshot, orc.n_sfr_histories))
    sa["sfr"][:, :, D:] = np.float32(3.0)  # padding
    before = sa["sfr"].copy()
    sb = {k: torch.from_numpy(v.copy()).cuda() for k, v in sa.items()}
    orc.ComputeTs(snapshot, sa)
    gpu.ComputeTs(snapshot, sb)
    assert snapshot == 0 or not np.array_equal(before, sa["sfr"])  # no history, no operations
    assert np.all(np.abs(sb["sfr"].cpu().numpy() - sa["sfr"]) <= 5e-7 * np.abs(sa["sfr"]))
