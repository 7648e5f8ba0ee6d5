"""The tuner times and reports tile heights that the launches run: the kernels round a
height up to a multiple of 8 and cap it at 48, so another one would be a launch timed
twice and a height that no launch has."""
import importlib

import pytest

pytestmark = pytest.mark.gpu

modelgen = importlib.import_module("marineseis-fdm-2d_b200.modelgen")


@pytest.mark.parametrize("nx,nz", [(640, 400), (800, 400), (720, 448), (560, 496), (680, 520), (760, 440)])
def test_reported_heights_run(mfdm, nx, nz):
    m = modelgen.make_model(nx, nz // 2, nz - nz // 2, npd=20, fpeak=20.0, nt=10, src_x=[nx // 2],
                            src_z=[nz // 4])
    with mfdm.Solver.from_model(m) as s:
        assert s.autotune() in (8, 16, 24, 32, 40, 48)
