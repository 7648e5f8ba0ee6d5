"""A batched shot equals the same shot run alone, bit for bit, at sizes where the
batch's cells and one shot's lie on different sides of the lines at which the
library changes its stage build (0.5 M cells), its form of accumulation (2.5 M)
and its tile height."""
import copy
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

modelgen = importlib.import_module("marineseis-fdm-2d_b200.modelgen")

NT = 96  # the wave reaches the strips, whose arithmetic the builds contract differently


# nx, nz, boundary type, shots
@pytest.mark.parametrize("nx,nz,bdy,n", [(160, 121, 2, 64), (160, 121, 2, 140), (403, 301, 1, 24),
                                         (1201, 803, 2, 3)])
def test_batch_equals_its_shots_at_every_size(mfdm, nx, nz, bdy, n):
    m = modelgen.make_model(nx, nz // 2, nz - nz // 2, npd=20, fpeak=20.0, nt=NT, src_x=[nx // 2],
                            src_z=[nz // 4], boundary_type=bdy, amp=10.0, wavelength=1.5 * nx,
                            perturb=0.03, corr_len=30.0, seed=3)
    shots = [(nx // 3 + k % 40, nz // 4, 20.0 + k % 7, m.beta0) for k in range(n)]
    with mfdm.Batch.from_model(m, shots) as b:
        b.step(NT)
        got = [(b.records(shot=k), [b.field(f, shot=k) for f in mfdm.FIELDS]) for k in (0, n - 1)]
    for (rec, fields), (x, z, f, beta0) in zip(got, (shots[0], shots[-1])):
        one = copy.deepcopy(m)
        one.src_x, one.src_z, one.fpeak, one.beta0 = [x], [z], f, beta0
        with mfdm.Solver.from_model(one) as s:
            s.step(NT)
            alone = s.records()
            for q in rec:
                assert np.array_equal(rec[q], alone[q]), q
            for a, name in zip(fields, mfdm.FIELDS):
                assert np.array_equal(a, s.field(name)), name
