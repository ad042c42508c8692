"""The device memory that the SSIM calls keep between calls: bounded, given back on request, and calls from
several threads and streams meanwhile give the same values (GPU test)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_kept_memory_is_bounded_and_given_back():
    import torch

    from ragdoll_b200.engine import ssim_batch_device, trim_metrics_memory
    w, h, n = 1920, 1080, 150   # 207 MB of pyramids
    planes = torch.randint(0, 256, (4, h, w), dtype=torch.uint8, device="cuda")
    args = ([planes[i % 3].data_ptr() for i in range(n)], [planes[3].data_ptr()] * n, w, h, w, w)
    small = (args[0][:3], args[1][:3], w, h, w, w)
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    want = ssim_batch_device(*small)
    torch.cuda.synchronize()
    trim_metrics_memory()
    start = free()
    got = ssim_batch_device(*args)
    for k in range(2):
        assert np.array_equal(got[k], np.tile(want[k], n // 3))
    torch.cuda.synchronize()
    assert start - free() <= (128 << 20) + (32 << 20)   # the threshold and a granule of the pool
    ssim_batch_device(*small)
    trim_metrics_memory()
    assert start - free() <= 2 << 20
    bad = []

    def work():
        st = torch.cuda.Stream()
        for _ in range(30):
            r = ssim_batch_device(*small, stream=st.cuda_stream)
            if not all(np.array_equal(r[k], want[k]) for k in range(2)):
                bad.append(r)
            trim_metrics_memory()
    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
