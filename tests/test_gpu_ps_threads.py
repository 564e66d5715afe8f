"""Power spectra of contexts on several host threads, whose kernel takes as much
shared memory as the call has bins: with many bins on some threads and few on the
others every call succeeds and gives what it gives alone.  Plain library calls, so
that the threads spend their time in them and not in Python."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_bin_counts_of_concurrent_calls():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    D, w, calls = 8, workload("plain_64", 8), []
    for i in range(8):
        bins = 2 if i % 2 else 47
        step = ReionGridStep(w.params, w.redshifts)
        box = torch.rand((D, D, D), device="cuda")
        edges = (ctypes.c_float * (bins + 1))(*np.geomspace(0.05, 5.0, bins + 1).tolist())
        loss, power, stream = ctypes.c_double(), (ctypes.c_float * bins)(), torch.cuda.Stream()
        args = (step.ctx, box.data_ptr(), bins, edges, (ctypes.c_float * bins)(), ctypes.byref(loss), power, None,
                ctypes.c_void_p(stream.cuda_stream))
        calls.append((step, box, stream, args, loss, power))
    torch.cuda.synchronize()
    alone = []
    for step, _, _, args, loss, power in calls:
        assert step.lib.mx_ps_loss_device(*args) == 0
        alone.append((loss.value, list(power)))
    failed, changed = [0] * 8, [0] * 8

    def work(i):
        step, _, _, args, loss, power = calls[i]
        for _ in range(4000):
            if step.lib.mx_ps_loss_device(*args) != 0:
                failed[i] += 1
            elif (loss.value, list(power)) != alone[i]:
                changed[i] += 1

    threads = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert failed == [0] * 8 and changed == [0] * 8
