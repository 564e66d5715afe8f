"""The host fallback of ComputeTs's frequency tables, which takes over where an
adaptive integral outgrows the device's interval list (never on ordinary inputs):
with the list cut to a few intervals, in a call of its own, inside a captured step
and in the adjoint's three sets, against the device's tables.

Tolerance 1e-6 relative on averages and parameter gradients: host and device take
the same quadrature steps in FP64, so their tables agree to rounding, which the FP32
coefficients (6e-8) and sums see; E0's gradient is a difference of tables over 2e-3
of E0, 500 times their FP32 roundings at most: 5e-5.  A table of a few intervals
would be off by 1e-2 and more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("intervals", [2, 5, 12])
def test_host_tables_match_device_tables(intervals, monkeypatch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300 import synthetic as syn
    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    D = 16
    w = workload("diff_256", D)
    n_hist = ReionGridStep(w.params, w.redshifts).n_sfr_histories
    st = syn.initial_state(w.params, w.redshifts[0])
    st.update(syn.FieldGenerator(w).inputs(1, n_hist))
    st.setdefault("delta_T", np.zeros((D, D, D), np.float32))
    names = ("volume_ave_Xheat", "volume_ave_Xion", "volume_ave_J_alpha", "volume_ave_TS", "collapse_fraction", "x_e_ave")

    def run(how):
        step = ReionGridStep(w.params, w.redshifts)
        g = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in st.items()}
        if how == "host":
            out = step.ComputeTs(1, {k: v.copy() for k, v in st.items()})
        elif how == "plain":
            out = step.ComputeTs(1, g)
        elif how == "graph":
            step.set_graph()
            out = step.step(1, g)
        else:
            grad = torch.linspace(-1.0, 2.0, D ** 3, device="cuda").reshape(D, D, D)
            saved = {k: v.clone() for k, v in g.items()}
            step.step(1, saved)
            before = step.freq_fallbacks()
            saved.update({k: g[k] for k in ("sfr", "x_e_box_prev", "Tk_box")})
            gs, _, lx, e0 = step.adjoint(1, saved, grad)
            return [lx, gs.double().abs().sum().item()], e0, step.freq_fallbacks() - before
        return [out[n] for n in names], 0.0, step.freq_fallbacks()

    for how, sets in (("plain", 1), ("host", 1), ("graph", 1), ("adjoint", 3)):
        monkeypatch.delenv("MX_FREQ_INTERVALS", raising=False)
        want, want_e0, none = run(how)
        monkeypatch.setenv("MX_FREQ_INTERVALS", str(intervals))
        got, got_e0, taken = run(how)
        assert (none, taken) == (0, sets), how
        assert got == pytest.approx(want, rel=1e-6), how
        assert got_e0 == pytest.approx(want_e0, rel=5e-5), how
