"""rg_analyse_batch of many streams by one launch whose warps meet, and of more segments than a tuned context's
warps by the per-diagonal launches, against the per-diagonal launches (taken where the reconstruction before
deblocking is kept): records and final reconstructions are integers, equal (GPU tests)."""
import numpy as np
import pytest

from ragdoll_b200.synth import grating_clip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [0, 1700, 64])  # 0.17 segments ready a warp (IDR pictures apart, others meet), 0.23 (all meet), 6.2 (per-diagonal)
@pytest.mark.parametrize("kinds", ["idr", "p", "mixed"])
def test_many_streams(kinds, grid):
    from ragdoll_b200.engine import RG_FRAME_IDR, RG_FRAME_P, Engine
    w, h, S, N = 173, 109, 128, 3
    clips = [grating_clip(w, h, N, seed=40 + s % 7, motion=3.0 + s % 5, rects=1) for s in range(S)]
    a, b = (Engine(w, h, 27, profile=2, num_streams=S) for _ in range(2))
    a.set_pipeline_tuning(grid=grid)
    b.keep_unfiltered(True)
    for f in range(N):
        ks = [RG_FRAME_IDR if f == 0 or kinds == "idr" or (kinds == "mixed" and (s + f) % 3 == 0) else RG_FRAME_P for s in range(S)]
        frames = [clips[s][f] for s in range(S)]
        assert a.analyse(frames, ks).tobytes() == b.analyse(frames, ks).tobytes(), f"picture {f}"
        for s in range(S):
            for p, q in zip(a.recon_coded(s), b.recon_coded(s)):
                assert np.array_equal(p, q), f"picture {f} stream {s}"
