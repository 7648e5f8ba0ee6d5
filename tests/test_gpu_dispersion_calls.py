"""mfdm_dispersion_image called from several threads on a B200."""
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
