"""mfdm_dispersion_image on a B200 from several threads, and after the device's
context was reset."""
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


def test_a_call_after_a_device_reset(mfdm):
    """Nothing that a call keeps outlives the context it was made in (in a process
    of its own: a reset ends the context of the whole process)."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    p = subprocess.run([sys.executable, "-c", AFTER_RESET], cwd=root, capture_output=True, text=True,
                       timeout=120)
    assert p.returncode == 0, p.stderr[-2000:]
