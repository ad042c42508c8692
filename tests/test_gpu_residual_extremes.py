"""Records and reconstructions equal the oracle's where the residual is at its limits: full-range
noise, checkerboards and flat pictures at the lowest and highest QPs (the largest coefficients and
levels, every 4x4 and 8x8 block coded, none coded), on sizes that are no macroblock multiple."""
import numpy as np
import pytest

from gpu_parity_util import run_parity

pytestmark = pytest.mark.gpu


def _frames(kind, w, h, n, seed):
    rng = np.random.default_rng(seed)
    out = []
    for f in range(n):
        planes = []
        for pw, ph in ((w, h), ((w + 1) // 2, (h + 1) // 2), ((w + 1) // 2, (h + 1) // 2)):
            if kind == "noise":      # two values only: the largest differences there are
                p = rng.integers(0, 2, (ph, pw)) * 255
            elif kind == "checker":  # the prediction of the last picture inverted
                p = ((np.add.outer(np.arange(ph), np.arange(pw)) + f) & 1) * 255
            elif kind == "steps":    # 4x4 tiles of random levels, moving by one sample
                t = rng.integers(0, 256, (ph // 4 + 3, pw // 4 + 3)) if f == 0 else tiles[len(planes)]
                if f == 0:
                    tiles = [] if not planes else tiles
                    tiles.append(t)
                p = np.kron(t, np.ones((4, 4), int))[f:f + ph, f:f + pw]
            else:                    # nearly flat: P_Skip and empty blocks
                p = np.full((ph, pw), 128) + (rng.random((ph, pw)) < 0.01)
            planes.append(np.ascontiguousarray(p.astype(np.uint8)))
        out.append(tuple(planes))
    return out


@pytest.mark.parametrize("qp", [1, 6, 11, 51])
@pytest.mark.parametrize("kind", ["noise", "checker", "steps", "flat"])
@pytest.mark.parametrize("w,h,profile", [(50, 38, 2), (33, 47, 0)])
def test_residual_extremes_match_the_oracle(kind, qp, w, h, profile):
    from ragdoll_b200.engine import Engine

    eng = Engine(w, h, qp, profile=profile)
    eng.keep_unfiltered(True)
    fails = run_parity(_frames(kind, w, h, 3, seed=qp * 7 + w), w, h, qp, profile, keyint=8, engine=eng)
    assert not fails, "\n".join(fails)
