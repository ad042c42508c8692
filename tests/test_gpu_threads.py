"""Contexts of several host threads launch side by side (GPU tests): some with launches of a single warp,
one with blocks of ten warps, which need more shared memory than a kernel has without asking. Every call succeeds, and the records equal
those of the same calls one at a time."""
import threading

import numpy as np
import pytest

from ragdoll_b200.synth import grating_clip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
def test_launches_of_several_sizes_from_several_threads(form):
    import torch

    from ragdoll_b200.engine import RG_FORM_FULLSEARCH, RG_FRAME_IDR, Engine

    def job(S, F, grid):
        w, h = 16, 16
        clip = grating_clip(w, h, F * S, seed=S, motion=2.0, rects=1)
        planes = [torch.from_numpy(np.ascontiguousarray(p)).cuda() for f in clip for p in f]
        eng = Engine(w, h, 30, profile=2, num_streams=S, max_frames=F)
        if form:
            eng.set_analysis_form(RG_FORM_FULLSEARCH, 8)
        eng.set_pipeline_tuning(grid=grid)
        torch.cuda.synchronize()
        args = ([p.data_ptr() for p in planes], w, (w + 1) // 2, [RG_FRAME_IDR] * (F * S), F)
        eng.analyse_gops_device(*args)
        return eng, args, eng.records_gops(F).tobytes(), planes
    small, large = [job(1, 1, 1) for _ in range(4)], job(64, 12, 0)
    errors, stop = [], threading.Event()

    def work(j, calls):
        eng, args, want, _ = j
        try:
            while calls and not stop.is_set():
                eng.analyse_gops_device(*args)
                eng.sync()
                calls -= 1
            if eng.records_gops(args[-1]).tobytes() != want:
                errors.append("records differ")
        except Exception as e:  # a refused launch
            errors.append(repr(e))
            stop.set()
    threads = [threading.Thread(target=work, args=(j, -1)) for j in small]
    for t in threads:
        t.start()
    work(large, 3000)
    stop.set()
    for t in threads:
        t.join()
    assert not errors, errors
