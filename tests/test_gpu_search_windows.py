"""The integer search's window shapes against the oracle (GPU tests): ranges whose windows are a vector a
lane (2 R + 1 squared up to 32 vectors), a few columns past whole groups of 32, a group of their own,
and the largest range, on pictures small enough that the vector bounds clip them to any width. Records
and reconstruction are integers: equal."""
import numpy as np
import pytest

from gpu_parity_util import SEARCH_FIELDS, first_pixel_mismatch, first_record_mismatch
from oracle_lib import OracleEncoder

pytestmark = pytest.mark.gpu


def _clip(w, h, n, seed):
    """A wrapped random field seen at large random displacements."""
    rng = np.random.default_rng(seed)
    planes = [rng.integers(0, 256, (h, w) if p == 0 else ((h + 1) // 2, (w + 1) // 2)).astype(np.float64) for p in range(3)]
    for _ in range(2):
        planes = [(p + np.roll(p, 1, 0) + np.roll(p, 1, 1) + np.roll(p, (1, 1), (0, 1))) / 4 for p in planes]
    out = []
    for _ in range(n):
        dy, dx = 2 * rng.integers(-20, 21, 2)
        out.append(tuple(np.ascontiguousarray(np.clip(np.roll(p, (dy >> (i > 0), dx >> (i > 0)), (0, 1)) + rng.integers(-2, 3, p.shape), 0, 255)
                                              .astype(np.uint8)) for i, p in enumerate(planes)))
    return out


@pytest.mark.parametrize("rng_", [1, 2, 3, 4, 15, 17, 18, 33, 64])
@pytest.mark.parametrize("w,h", [(16, 16), (70, 50), (160, 96)])
def test_fullsearch_windows(w, h, rng_):
    from ragdoll_b200.engine import RG_FORM_FULLSEARCH, RG_FRAME_IDR, RG_FRAME_P, Engine
    N, qp = 3, 28
    clip = _clip(w, h, N, 7 * rng_ + w)
    eng = Engine(w, h, qp, profile=2, num_streams=1, max_frames=N)
    eng.set_analysis_form(RG_FORM_FULLSEARCH, rng_)
    got = eng.analyse_gops([[f] for f in clip], [[RG_FRAME_IDR]] + [[RG_FRAME_P]] * (N - 1))
    orc = OracleEncoder(w, h, qp, profile=2, keyint=30)
    orc.set_form(1, rng_)
    for f, fr in enumerate(clip):
        _, want = orc.encode(fr)
        m = first_record_mismatch(want, got[f, 0], orc.mb_w, SEARCH_FIELDS)
        assert m is None, f"picture {f}: {m}"
    for p, (a, b) in enumerate(zip(orc.recon(filtered=True), eng.recon_coded(0))):
        assert first_pixel_mismatch(a, b) is None, f"plane {p}"
