"""rg_analyse_batch by one persistent launch equals the per-diagonal launches (taken where the
reconstruction before deblocking is kept): records and final reconstruction, integers, for sizes of one
macroblock, one row, one column and ragged edges, mixed picture kinds, all profiles, and through
alternating calls of one and of several pictures (GPU tests)."""
import numpy as np
import pytest

from ragdoll_b200.synth import grating_clip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,S", [(16, 16, 1), (200, 16, 1), (16, 120, 2), (61, 45, 3), (320, 180, 1), (320, 180, 5)])
@pytest.mark.parametrize("profile", [0, 1, 2])
def test_one_launch_equals_per_diagonal(w, h, S, profile):
    from ragdoll_b200.engine import RG_FRAME_IDR, RG_FRAME_P, Engine
    N = 5
    clips = [grating_clip(w, h, N + 2, seed=90 + s, motion=6.0, rects=2) for s in range(S)]
    a, b = (Engine(w, h, 24 + 4 * profile, profile=profile, num_streams=S, max_frames=2) for _ in range(2))
    b.keep_unfiltered(True)
    for f in range(N):
        kinds = [RG_FRAME_IDR if f == 0 or (f == 3 and s == 1) else RG_FRAME_P for s in range(S)]
        frames = [clips[s][f] for s in range(S)]
        assert a.analyse(frames, kinds).tobytes() == b.analyse(frames, kinds).tobytes(), f"picture {f}"
        for s in range(S):
            for p, q in zip(a.recon_coded(s), b.recon_coded(s)):
                assert np.array_equal(p, q), f"picture {f} stream {s}"
        if f == 2:  # a call of two pictures between the single ones
            two = [[clips[s][N + k] for s in range(S)] for k in range(2)]
            ks = [[RG_FRAME_P] * S] * 2
            assert a.analyse_gops(two, ks).tobytes() == b.analyse_gops(two, ks).tobytes()
