"""The SSIM passes at the edges of their strips and chunks, against the oracle (GPU tests).

Both strip shapes (4 rows x 256 windows for few pairs, 16 x 64 for many), planes a window more and
less than a whole chunk or strip, odd sizes at every scale, rows that are not whole words and bases
that are not aligned. Tolerance: a row's f32 sum of n windows in [-1, 1] is within n^2 / 2 units of 2^-24
of the exact one whatever the rounding, and the oracle's order is kept, which leaves the usual 1e-6; one
wrong window of the largest plane here (8,000 windows of values 0.01 .. 1 apart) is further off.
"""
import numpy as np
import pytest

import oracle_lib

pytestmark = pytest.mark.gpu

TOL = 1e-6
SIZES = [(8, 8), (11, 9), (16, 16), (18, 35), (260, 68), (261, 69), (1028, 20), (1032, 67), (1033, 129), (517, 131)]


def _planes(w, h, pad, offset, seed):
    rng = np.random.default_rng(seed)
    a = np.zeros(offset + (h + 1) * (w + pad), np.uint8)
    b = np.zeros_like(a)
    va = a[offset:offset + h * (w + pad)].reshape(h, w + pad)[:, :w]
    vb = b[offset:offset + h * (w + pad)].reshape(h, w + pad)[:, :w]
    va[:] = rng.integers(0, 256, (h, w))
    vb[:] = np.clip(va.astype(int) + rng.integers(-20, 21, (h, w)), 0, 255)
    return a, b, va, vb


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("pad,offset", [(0, 0), (0, 1), (3, 2)])
def test_plane_noalloc(w, h, pad, offset):
    import torch
    from ragdoll_b200.engine import ssim_plane_device_noalloc
    a, b, va, vb = _planes(w, h, pad, offset, w * 7 + h)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    out = torch.zeros(2, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ssim_plane_device_noalloc(da.data_ptr() + offset, w + pad, db.data_ptr() + offset, w + pad, w, h, out.data_ptr())
    torch.cuda.synchronize()
    s, m = out.cpu().tolist()
    assert abs(s - oracle_lib.ssim_plane(va, vb)) <= TOL
    assert abs(m - oracle_lib.ms_ssim_plane(va, vb)) <= TOL


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("copies", [1, 300])
def test_batch(w, h, copies):
    """One pair (flat strips) and 300 (tall strips) of the same planes."""
    import torch
    from ragdoll_b200.engine import ssim_batch_device
    a, b, va, vb = _planes(w, h, 1, 1, w * 5 + h)
    da, db = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    torch.cuda.synchronize()
    s, m = ssim_batch_device([da.data_ptr() + 1] * copies, [db.data_ptr() + 1] * copies, w, h, w + 1, w + 1)
    assert np.abs(s - oracle_lib.ssim_plane(va, vb)).max() <= TOL and len(set(s.tolist())) == 1
    assert np.abs(m - oracle_lib.ms_ssim_plane(va, vb)).max() <= TOL and len(set(m.tolist())) == 1
