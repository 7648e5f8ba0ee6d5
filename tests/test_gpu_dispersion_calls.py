"""mfdm_dispersion_image on a B200 from several threads, after the device's context
was reset, and what it leaves of the device's memory."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def image(mfdm, nt, ntr, seed=1):
    rng = np.random.default_rng([nt, ntr, seed])
    g = rng.standard_normal((nt, ntr)).astype(np.float32)
    return mfdm.dispersion_image(g, np.arange(float(ntr)), 500.0, 1500.0, 1500.0, 1.0)[2]


def test_calls_of_two_threads_do_not_disturb_each_other(mfdm):
    """A long gather needs 96 KB of shared memory a block, a short one 33 KB: a
    kernel's limit is common to all threads, so calls of one must not lower the
    other's."""
    want = {nt: image(mfdm, nt, 3) for nt in (4096, 64)}
    bad = []

    def work(nt):
        for _ in range(1000):
            try:
                if not np.array_equal(image(mfdm, nt, 3), want[nt]):
                    bad.append((nt, "another image"))
            except mfdm.MfdmError as e:
                bad.append((nt, str(e)))

    threads = [threading.Thread(target=work, args=(nt,)) for nt in want]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, (len(bad), bad[:3])


AFTER_RESET = """
import ctypes, importlib, os, sys
import numpy as np
sys.path.insert(0, os.getcwd())
mfdm = importlib.import_module("marineseis-fdm-2d_b200")
g = np.random.default_rng(1).standard_normal((96, 8)).astype(np.float32)
image = lambda: mfdm.dispersion_image(g, np.arange(8.0), 500.0, 1500.0, 1510.0, 5.0)[2]
first = image()
for _ in range(2):
    assert ctypes.CDLL("libcuda.so.1").cuDevicePrimaryCtxReset_v2(0) == 0  # what cudaDeviceReset does
    for _ in range(2):
        assert np.array_equal(image(), first)
"""


def child(code):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True,
                       timeout=120)
    assert p.returncode == 0, p.stderr[-2000:]


def test_a_call_after_a_device_reset(mfdm):
    """Nothing that a call keeps outlives the context it was made in (in a process
    of its own: a reset ends the context of the whole process)."""
    child(AFTER_RESET)


def test_a_large_call_gives_its_memory_back(mfdm):
    """8000 x 2000 samples take 190 MB; 64 MiB may stay (and 4 MiB for what else
    the process allocates meanwhile)."""
    import torch
    image(mfdm, 8000, 8)  # the kernels are loaded
    free = torch.cuda.mem_get_info()[0]
    image(mfdm, 8000, 2000)
    assert free - torch.cuda.mem_get_info()[0] <= 68 << 20


FULL_DEVICE = """
import importlib, os, sys
import numpy as np, torch
sys.path.insert(0, os.getcwd())
mfdm = importlib.import_module("marineseis-fdm-2d_b200")
modelgen = importlib.import_module("marineseis-fdm-2d_b200.modelgen")
m = modelgen.make_model(640, 200, 200, npd=20, fpeak=20.0, nt=10, src_x=[200], src_z=[100])
with mfdm.Solver.from_model(m) as s:  # the kernels are loaded
    need = s.info()["device_bytes"]
    s.step(2)
g = np.ones((2000, 1200), np.float32)
mfdm.dispersion_image(g, np.arange(1200.0), 500.0, 1500.0, 1500.0, 1.0)  # 48 MB
free = torch.cuda.mem_get_info()[0]
assert (24 << 20) < need < (50 << 20), need
hold = torch.empty(free - (20 << 20), dtype=torch.uint8, device="cuda")
with mfdm.Solver.from_model(m) as s:
    s.step(2)
"""


def test_the_memory_kept_does_not_keep_a_model_out(mfdm):
    """A model that fits the device beside what others hold opens also after an image."""
    child(FULL_DEVICE)
