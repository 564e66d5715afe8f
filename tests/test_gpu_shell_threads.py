"""ComputeTs and the adjoint of contexts on several host threads, whose kernels take as
much shared memory as the context has shells: with 64 shells on some threads and 3 on
the others every call succeeds and gives what it gives alone."""
import dataclasses
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STATE = ("sfr", "x_e_box_prev", "Tk_box")


@pytest.mark.parametrize("adjoint", [False, True])
def test_shell_counts_of_concurrent_calls(adjoint):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300 import synthetic as syn
    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    D, calls = 8, []
    for i in range(8):
        w = workload("diff_256", D)
        w.params = dataclasses.replace(w.params, ts_num_filter_steps=3 if i % 2 else 64)
        step = ReionGridStep(w.params, w.redshifts)
        st = syn.initial_state(w.params, w.redshifts[0])
        st.update(syn.FieldGenerator(w).inputs(1, step.n_sfr_histories))
        g = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in st.items()}
        if adjoint:  # of a step that has run
            step.step(1, g)
        grad = torch.ones((D, D, D), device="cuda")
        calls.append((step, g, {k: g[k].clone() for k in STATE}, grad, torch.cuda.Stream()))
    torch.cuda.synchronize()

    def once(i):
        step, g, kept, grad, stream = calls[i]
        with torch.cuda.stream(stream):
            for k in STATE:
                g[k].copy_(kept[k])
            if adjoint:
                out = step.adjoint(1, g, grad)
                return out[2], out[3]
            out = step.ComputeTs(1, g)
            return out["volume_ave_TS"], out["volume_ave_J_alpha"]

    alone = [once(i) for i in range(8)]
    assert alone[0] == once(0)
    errors = []

    def work(i):
        try:
            for _ in range(400):
                assert once(i) == alone[i]
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
