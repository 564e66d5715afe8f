"""Grids without a fused transform, whose cuFFT executions hold as many radii (or
shells) as the context's memory and 64 MB allow.

Same bits in contexts of different memory: a spectrum's transform does not depend on
the batch that it is executed in, so nor do grids and averages.  And the batch
runner's estimate of a context's memory holds the plans' work areas, which are made
by the first calls: at 74 = 2 x 37 cuFFT transforms out of place, with work areas as
large as the spectra."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("D", [2, 18, 26, 46, 62, 98, 106, 122])
def test_same_bits_in_contexts_of_any_memory(D):
    import torch

    from meraxes_gb300 import synthetic as syn
    from meraxes_gb300.api import ReionGridStep
    from meraxes_gb300.params import workload

    w = workload("full_256", D)
    w.params = dataclasses.replace(w.params, reion_efficiency=31043.3)
    w.fesc = 0.01
    out = []
    for spectra in (0, 25, 12, 1):
        step = ReionGridStep(w.params, w.redshifts, max_work_bytes=spectra * 8 * D * D * (D // 2 + 1))
        st = syn.initial_state(w.params, w.redshifts[0])
        st.update(syn.FieldGenerator(w).inputs(1, step.n_sfr_histories))
        g = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in st.items()}
        means = step.step(1, g)
        means.pop("gpu_launches", None)
        out.append(({k: v.cpu().numpy() for k, v in g.items()}, means))
        step.close()
    for grids, means in out[1:]:
        assert means == out[0][1]
        for k, v in grids.items():
            assert np.array_equal(v, out[0][0][k], equal_nan=True), k


def test_memory_plan_covers_the_plans():
    import torch

    from meraxes_gb300.batch import BatchRunner, Instance

    # kernels and cuFFT's modules are loaded by a first box
    BatchRunner([Instance(74, 3, 2e40, 0.1)], max_workers_per_size=1).run()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    free0, reserved0, held0 = torch.cuda.mem_get_info()[0], torch.cuda.memory_reserved(), torch.cuda.memory_allocated()
    runner = BatchRunner([Instance(74, 4, 2e40, 0.1)], max_workers_per_size=1)
    new_step, steps = runner._new_step, []
    runner._new_step = lambda D: steps.append(new_step(D)) or steps[-1]  # kept: its memory is what is measured
    runner.run()
    torch.cuda.synchronize()
    library = free0 - torch.cuda.mem_get_info()[0] - (torch.cuda.memory_reserved() - reserved0)
    tensors = torch.cuda.max_memory_allocated() - held0
    assert len(steps) == 1
    assert 0 < library + tensors <= runner.ctx_bytes[74]
