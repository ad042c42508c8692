"""The network's kernels at the edges of their work (GPU tests).

Training: batches of one sample, around the samples a block takes and a whole grid of blocks, a smaller
batch after a larger one, against the float64 oracle. Tolerance: a gradient element is a sum of at most
n * 324 products of f32 values of one magnitude, each rounded to 2^-24: below 1e-4 of the largest
gradient for these batches with random signs; 1e-3 is what the repository's other gradient test takes.
The sums are in a fixed order: a second pass gives the same bits.

Coarse motion: ranges whose columns are whole groups of 32, a few more, or a partial group, odd widths
(unaligned rows), pictures of fewer and of more than eight macroblocks a row: equal to the host's."""
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))
import candidate_net_oracle as cno  # noqa: E402
from ragdoll_b200.synth import grating_clip  # noqa: E402
from test_gpu_net import _coarse_motion, _params  # noqa: E402

pytestmark = pytest.mark.gpu


def test_training_batches():
    import torch

    from ragdoll_b200.learned import CandidateNet
    rng = np.random.default_rng(11)
    p = _params(12)
    net = CandidateNet(0, params=p)
    for n in (1, 2, 9, 150, 33, 1):
        crops = rng.integers(0, 256, (n, 2, 24, 24)).astype(np.uint8)
        part = rng.integers(-1, 4, n).astype(np.int32)
        i4 = rng.integers(-1, 9, (n, 16)).astype(np.int32)
        mv = rng.normal(0, 1.5, (n, 2)).astype(np.float32)
        mvv = rng.integers(0, 2, n).astype(np.int32)
        part[0], i4[0, 0], mvv[0] = 1, 3, 1
        d = {k: torch.from_numpy(v).cuda() for k, v in dict(c=crops, p=part, i=i4, m=mv, v=mvv).items()}
        args = (d["c"].data_ptr(), n, d["p"].data_ptr(), d["i"].data_ptr(), d["m"].data_ptr(), d["v"].data_ptr(), 0.5)
        loss, grads = net.forward_backward(*args, want_grads=True)
        grads = np.array(grads)
        want_loss, want, _ = cno.forward_backward(p.astype(np.float64), crops, part, i4, mv, mvv, 0.5)
        assert abs(loss - want_loss) <= 1e-4 * max(1.0, abs(want_loss)), n
        assert np.abs(grads - want).max() <= 1e-3 * np.abs(want).max(), n
        again = net.forward_backward(*args, want_grads=True)
        assert again[0] == loss and np.array_equal(np.array(again[1]), grads), n


@pytest.mark.parametrize("w,h", [(16, 16), (33, 50), (150, 84), (289, 33)])
@pytest.mark.parametrize("search_range", [2, 6, 30, 32, 36, 62, 64])
def test_coarse_ranges(w, h, search_range):
    import torch

    from ragdoll_b200.engine import HINT_DTYPE
    from ragdoll_b200.learned import CandidateNet, hints_for
    frames = grating_clip(w, h, 2, seed=w + search_range, motion=9.0, rects=2)
    cur, prev = (np.ascontiguousarray(f[0]) for f in (frames[1], frames[0]))
    net = CandidateNet(0, params=_params(8))
    net.set_coarse_range(search_range)
    tc, tp = torch.from_numpy(cur).cuda(), torch.from_numpy(prev).cuda()
    hints, _ = hints_for(net, [tc.data_ptr()], [tp.data_ptr()], w, h, w)
    net.check()
    torch.cuda.synchronize()
    got = hints[0].cpu().numpy().view(HINT_DTYPE)
    assert (got["flags"] == 1).all()
    assert np.array_equal(got["mv_coarse"].astype(np.int32), _coarse_motion(cur, prev, search_range // 2))
