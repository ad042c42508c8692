"""Search forms whose waits run out in a launch of several warps a block (GPU tests): warps that wait take
part in their neighbours' integer searches, and every wait -- for a segment, for the reference picture, for
search units that others took -- may give up. Nothing of such a macroblock may be published: the call is
re-run, and its records and reconstructions equal the oracle's (integers). Ranges 8 and 24 have no columns
past whole groups of 32 or a group of their own, 16 has one; two-macroblock segments keep a warp at the same
row after the macroblock whose wait gave up."""
import ctypes

import numpy as np
import pytest

from gpu_parity_util import SEARCH_FIELDS, first_pixel_mismatch, first_record_mismatch
from oracle_lib import OracleEncoder
from ragdoll_b200.synth import grating_clip

pytestmark = pytest.mark.gpu
QP = 26
SHORT = dict(lag=1, seg=2, timeout_ms=1)   # the next picture's segments before their reference: waits run out


def _expected(clip, w, h, rng_):
    orc = OracleEncoder(w, h, QP, profile=2, keyint=len(clip) + 1)
    orc.set_form(1, rng_)
    return orc, [orc.encode(fr)[1] for fr in clip]


def _check(clip, w, h, rng_, records, recon):
    orc, want = _expected(clip, w, h, rng_)
    for f, r in enumerate(want):
        m = first_record_mismatch(r, records[f], orc.mb_w, SEARCH_FIELDS)
        assert m is None, f"picture {f}: {m}"
    for p, (a, b) in enumerate(zip(orc.recon(filtered=True), recon)):
        assert first_pixel_mismatch(a, b) is None, f"plane {p}"


@pytest.mark.parametrize("rng_", [8, 16, 24])
def test_streamed_search_gives_up_and_is_run_again(rng_):
    """Pictures fetched while the launch runs are exact too: one that did not finish is reported so."""
    from ragdoll_b200.engine import RECORD_DTYPE, RG_FORM_FULLSEARCH, RG_FRAME_IDR, RG_FRAME_P, Engine, lib
    w, h, S, F = 176, 112, 8, 6
    clips = [grating_clip(w, h, F, seed=1300 + s, motion=8.0, rects=2) for s in range(S)]
    eng = Engine(w, h, QP, profile=2, num_streams=S, max_frames=F)
    eng.set_analysis_form(RG_FORM_FULLSEARCH, rng_)
    eng.set_pipeline_tuning(**SHORT)
    out = np.zeros((F, S, eng.n_mb), RECORD_DTYPE)
    planes = [np.ascontiguousarray(p) for f in range(F) for s in range(S) for p in clips[s][f]]
    ptrs = (ctypes.c_void_p * len(planes))(*[p.ctypes.data for p in planes])
    kinds = (ctypes.c_int32 * (F * S))(*[RG_FRAME_IDR if f == 0 else RG_FRAME_P for f in range(F) for _ in range(S)])
    L = lib()
    assert L.rg_analyse_gops_stream(eng.h, ptrs, w, (w + 1) // 2, kinds, F, out.ctypes.data) == 0
    early, unfinished = {}, set()
    while len(early) + len(unfinished) < F * S:
        for i in range(F * S):
            if i in early or i in unfinished:
                continue
            st = L.rg_analyse_gops_fetch(eng.h, out.ctypes.data, i)
            assert st in (0, 1, 2), st
            if st == 1:
                early[i] = out[i // S, i % S].tobytes()
            elif st == 2:
                unfinished.add(i)
    assert unfinished, "no wait ran out"
    assert L.rg_analyse_gops_wait(eng.h, out.ctypes.data) == 0
    for i, r in early.items():
        assert out[i // S, i % S].tobytes() == r, f"picture {i} was handed out before it was final"
    for s in range(S):
        _check(clips[s], w, h, rng_, out[:, s], eng.recon_coded(s))


@pytest.mark.parametrize("rng_", [8, 24])
def test_group_search_gives_up_and_is_run_again(rng_):
    import torch

    from ragdoll_b200.engine import RG_FORM_FULLSEARCH, RG_FRAME_IDR, RG_FRAME_P, Engine
    sizes, F = [(96, 64, 4), (176, 112, 6)], 5
    engs, clips, keep, planes, kinds = [], [], [], [], []
    for i, (w, h, S) in enumerate(sizes):
        e = Engine(w, h, QP, profile=2, num_streams=S, max_frames=F)
        e.set_analysis_form(RG_FORM_FULLSEARCH, rng_)
        e.set_pipeline_tuning(**SHORT)
        c = [grating_clip(w, h, F, seed=1400 + 10 * i + s, motion=8.0, rects=2) for s in range(S)]
        t = [torch.from_numpy(np.ascontiguousarray(p)).cuda() for f in range(F) for s in range(S) for p in c[s][f]]
        engs.append(e)
        clips.append(c)
        keep.append(t)
        planes.append([x.data_ptr() for x in t])
        kinds.append([RG_FRAME_IDR if f == 0 else RG_FRAME_P for f in range(F) for _ in range(S)])
    torch.cuda.synchronize()
    Engine.analyse_gops_group(engs, planes, [w for w, _, _ in sizes], [(w + 1) // 2 for w, _, _ in sizes], kinds, F)
    for (w, h, S), e, c in zip(sizes, engs, clips):
        got = e.records_gops(F)
        for s in range(S):
            _check(c[s], w, h, rng_, got[:, s], e.recon_coded(s))
