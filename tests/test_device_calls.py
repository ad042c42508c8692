"""What the library's host code allocates, and on which of two devices where the current one is not the
context's, against a stand-in for the CUDA runtime (fake_cudart.c; no GPU)."""
import os
import shutil
import subprocess
import sys
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
CUDA_INCLUDE = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"
PRELUDE = """
import ctypes, sys
sys.path.insert(0, sys.argv[2])
import numpy as np
fake = ctypes.CDLL(sys.argv[1])
fake.fake_log.restype = fake.fake_launches.restype = ctypes.c_char_p
from ragdoll_b200.engine import RG_FRAME_IDR, RG_FRAME_P, Engine, RgError, lib
log = lambda: [l.split() for l in fake.fake_log().decode().split("\\n")[:-1]]
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    cc = shutil.which("gcc")
    if not cc or not CUDA_INCLUDE.exists():
        pytest.skip("needs gcc and the CUDA headers")
    so = tmp_path_factory.mktemp("fake") / "libfake_cudart.so"
    subprocess.run([cc, "-shared", "-fPIC", "-O1", f"-I{CUDA_INCLUDE}", "-o", str(so), str(HERE / "fake_cudart.c")], check=True)
    return so


def _run(fake, body):
    r = subprocess.run([sys.executable, "-c", PRELUDE + body, str(fake), str(HERE.parent)], env={**os.environ, "LD_PRELOAD": str(fake)},
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_buffers_of_a_first_call_are_on_the_contexts_device(fake):
    """A call while another device is current is refused by its launch, as ever; what it allocated on the way
    is the context's for the calls to come, and therefore on the context's device."""
    _run(fake, """
w = h = 32
eng = Engine(w, h, 30, profile=2, device=0, max_frames=2)
planes = [np.zeros(w * h, np.uint8) for _ in range(3)] * 2
args = ([p.ctypes.data for p in planes], w, w // 2, [RG_FRAME_IDR, RG_FRAME_P], 2)
fake.cudaSetDevice(1)
fake.fake_clear()
try:
    eng.analyse_gops_device(*args)
    raise SystemExit("accepted")
except RgError:
    pass
fake.cudaSetDevice(0)
eng.analyse_gops_device(*args)
eng.records_gops(2)
made = log()
assert {"malloc", "stream"} <= {l[0] for l in made}, made
assert all(l[1] == "0" for l in made), made
""")


def test_destroying_a_context_trims_its_devices_metrics_pool(fake):
    _run(fake, """
from ragdoll_b200.engine import ssim_batch_device
eng = Engine(32, 32, 30, profile=2, device=0)
plane = np.zeros(1024, np.uint8).ctypes.data
for device in (0, 1):
    ssim_batch_device([plane], [plane], 32, 32, 32, 32, device=device)
fake.cudaSetDevice(1)
fake.fake_clear()
eng.close()
assert [l for l in log() if l[0] == "trim"] == [["trim", "0", "to", "0"]], log()
""")


def test_metrics_memory_is_given_back_on_request(fake):
    _run(fake, """
from ragdoll_b200.engine import ssim_batch_device, trim_metrics_memory
plane = np.zeros(1024, np.uint8).ctypes.data
trim_metrics_memory(1)                      # nothing kept yet
ssim_batch_device([plane], [plane], 32, 32, 32, 32, device=1)
fake.fake_clear()
trim_metrics_memory(0)
trim_metrics_memory(1)
assert log() == [["trim", "1", "to", "0"]], log()
for device in (-1, 64):
    try:
        trim_metrics_memory(device)
        raise SystemExit("accepted")
    except RgError:
        pass
""")


def test_ssim_strips_follow_the_devices_sms(fake):
    """Tall strips (16 window rows) once there are two blocks an SM of them, flat ones (4) before: four planes
    of 1080 rows are 68 tall strips."""
    _run(fake, """
from ragdoll_b200.engine import ssim_batch_device
plane = np.zeros(64 * 1080, np.uint8).ctypes.data
for sms, strips in ((34, 17), (35, 68), (148, 68)):
    ctypes.c_int.in_dll(fake, "fake_sms").value = sms
    fake.fake_clear()
    ssim_batch_device([plane] * 4, [plane] * 4, 64, 1080, 64, 64)
    grids = [tuple(map(int, l.split())) for l in fake.fake_launches().decode().split("\\n")[:-1]]
    assert grids[0] == (strips, 4), (sms, grids)
""")


def test_training_scratch_grows_with_the_activations(fake):
    """The six maps of a sample are 309,248 bytes; the partial sums are a few rows a sample and a row a block
    of the weight gradients, of which there are no more than SMs. A smaller batch allocates nothing."""
    _run(fake, """
from ragdoll_b200.learned import CandidateNet
n = 4096
net = CandidateNet(0)
buf = np.zeros(n * 1152, np.uint8)
fake.fake_clear()
for batch in (n, n, 150, 1):
    net.forward_backward(buf.ctypes.data, batch, buf.ctypes.data, buf.ctypes.data, buf.ctypes.data, buf.ctypes.data)
    if batch == n:
        size = sum(int(l[2]) for l in log())
    assert size <= 1.05 * n * 309248, size / n
    assert size == sum(int(l[2]) for l in log())
""")
