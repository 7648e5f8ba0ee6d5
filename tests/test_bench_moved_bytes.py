"""The bytes bench.py holds against the copy rate are those of the form that runs (no
GPU needed): 16 floats a state value where every stage adds to the accumulator, 12
where one stage a step does (from 2.5 M cells with the build for large grids, and
solid only at every size), so that a fraction of the copy rate cannot pass 1."""
import importlib
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
bench = importlib.import_module("bench")


class Grid:
    def __init__(self, nx, nz_f, nz_s, npd=20):
        self.nx, self.nz_f, self.nz_s, self.npd, self.cells = nx, nz_f, nz_s, npd, nx * (nz_f + nz_s)


@pytest.mark.parametrize("nx,nz_f,nz_s,build,once", [(4096, 1024, 1025, 4, True), (4096, 1024, 1025, 3, False),
                                                     (1200, 304, 497, 4, False), (2500, 500, 500, 4, True),
                                                     (2499, 500, 500, 4, False), (160, 61, 60, 3, False)])
@pytest.mark.parametrize("shots", [1, 64])
def test_bytes_follow_the_form_that_runs(nx, nz_f, nz_s, build, once, shots):
    m = Grid(nx, nz_f, nz_s)
    strips = 2 * m.npd * (nz_f - 3) + 2 * m.npd * (nz_s - 3) + m.npd * (nx - 6)
    n = 12 if once else 16
    state = (nx * (3 * nz_f + 5 * nz_s) + 4 * strips) * n
    coefs = nx * (6 * nz_f + 9 * nz_s) * 4
    assert bench.step_bytes(m, shots, build) == (shots * state + coefs) * 4


def test_solid_only_bytes():
    m = Grid(2048, 0, 2048)
    assert bench.solid_step_bytes(m) == m.cells * 384
