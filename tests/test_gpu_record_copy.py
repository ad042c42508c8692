"""Records copied while the launch that writes them still runs (rg_copy_records_gops right after a
device-source call) equal the copy of a finished launch: whole calls, leading pictures only, more
pictures than the last call had, contexts of one group launch, and a launch whose wait gave up
(one warp, a lag of one macroblock-time) and is re-run. Records are integers: equal (GPU tests)."""
import numpy as np
import pytest

from ragdoll_b200.synth import grating_clip

pytestmark = pytest.mark.gpu
S, F = 3, 4


def _device_call(w, h, seed):
    import torch
    clips = [grating_clip(w, h, F, seed=seed + s, motion=5.0, rects=2) for s in range(S)]
    planes = [[torch.from_numpy(np.ascontiguousarray(p)).cuda() for p in clips[s][f]] for f in range(F) for s in range(S)]
    torch.cuda.synchronize()
    return planes, [t.data_ptr() for pic in planes for t in pic]


def _kinds(first):
    from ragdoll_b200.engine import RG_FRAME_IDR, RG_FRAME_P
    return [RG_FRAME_IDR if f == 0 and first else RG_FRAME_P for f in range(F) for _ in range(S)]


@pytest.mark.parametrize("w,h", [(16, 16), (176, 144), (640, 352)])
@pytest.mark.parametrize("give_up", [False, True])
def test_copy_while_running(w, h, give_up):
    from ragdoll_b200.engine import Engine
    keep, ptrs = _device_call(w, h, 40)
    if give_up and w > 176:
        pytest.skip("one warp takes the whole clip")
    a, b = (Engine(w, h, 27, profile=2, num_streams=S, max_frames=F) for _ in range(2))
    for call in range(2):
        n = F if call == 0 else 2
        if give_up:
            a.set_pipeline_tuning(lag=1, grid=1, timeout_ms=300)
        for e in (a, b):
            e.analyse_gops_device(ptrs[:n * S * 3], w, (w + 1) // 2, _kinds(call == 0)[:n * S], n)
        b.sync()
        want = b.records_gops(F)  # the second call leaves the first one's later pictures
        assert a.records_gops(1).tobytes() == want[:1].tobytes()
        assert a.records_gops(F).tobytes() == want.tobytes()
        for e in (a, b):
            e.analyse_gops_device(ptrs[:n * S * 3], w, (w + 1) // 2, _kinds(True)[:n * S], n)
        b.sync()
        assert a.records_gops(F).tobytes() == b.records_gops(F).tobytes()


def test_copy_of_a_group_while_running():
    from ragdoll_b200.engine import Engine
    sizes = [(640, 352), (176, 144), (96, 80)]
    calls = [_device_call(w, h, 60 + w) for w, h in sizes]
    sets = [[Engine(w, h, 30, profile=2, num_streams=S, max_frames=F) for w, h in sizes] for _ in range(2)]
    for call in range(2):
        for engs in sets:
            Engine.analyse_gops_group(engs, [c[1] for c in calls], [w for w, _ in sizes], [(w + 1) // 2 for w, _ in sizes],
                                      [_kinds(call == 0)] * len(sizes), F)
        for e in sets[1]:
            e.sync()
        for a, b in zip(*sets):
            assert a.records_gops(F).tobytes() == b.records_gops(F).tobytes()


@pytest.mark.parametrize("order", [(0, 1, 2), (2, 1, 0)])
def test_group_contexts_fetched_before_the_launch_ends_go_on(order):
    """A context's records fetched while other contexts of the launch still run: its reconstruction, its
    next group call and one of its own equal those of contexts synchronised after each launch."""
    from ragdoll_b200.engine import Engine
    sizes = [(96, 80), (176, 144), (1280, 720)]
    calls = [_device_call(w, h, 70 + w) for w, h in sizes]
    sets = [[Engine(w, h, 30, profile=2, num_streams=S, max_frames=F) for w, h in sizes] for _ in range(2)]
    args = ([c[1] for c in calls], [w for w, _ in sizes], [(w + 1) // 2 for w, _ in sizes])
    for call in range(2):
        got = {}
        Engine.analyse_gops_group(sets[0], *args, [_kinds(call == 0)] * 3, F)
        for i in order:
            got[i] = sets[0][i].records_gops(F)
        Engine.analyse_gops_group(sets[1], *args, [_kinds(call == 0)] * 3, F)
        for e in sets[1]:
            e.sync()
        for i in order:
            assert got[i].tobytes() == sets[1][i].records_gops(F).tobytes()
    w, h = sizes[0]
    for s in sets:
        s[0].analyse_gops_device(calls[0][1], w, (w + 1) // 2, _kinds(False), F)
    assert sets[0][0].records_gops(F).tobytes() == sets[1][0].records_gops(F).tobytes()
    for a, b in zip(*sets):
        for k in range(S):
            for p, q in zip(a.recon_coded(k), b.recon_coded(k)):
                assert np.array_equal(p, q)
