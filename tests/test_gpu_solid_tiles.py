"""The solid-only stage kernel's tiling at the sizes where it can go wrong, on a
B200: the smallest grids, strips that meet, bands that reach the surface rows, no
strip at all, tiles of one column or row, and both builds (the line is at 600,000
cells), each held to the FP32 oracle.
"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

modelgen = importlib.import_module("marineseis-fdm-2d_b200.modelgen")

NT = 70  # two captured runs of 32 steps and single steps
# Both run the same FP32 operator; a step's relative rounding is below 2^-22 (four
# stage roundings), 70 steps in one direction 1.7e-5, as a random walk 2e-6.
TOL = 1e-5

# nx, nz, npd, boundary type
CASES = [
    (8, 9, 1, 2),       # the smallest grid: surface rows and bottom band only
    (11, 34, 2, 1),     # the smallest four-side grid
    (46, 30, 20, 2),    # the side strips meet: no interior column
    (99, 28, 20, 2),    # the bottom band reaches the surface rows
    (70, 41, 0, 2),     # no absorbing strip
    (161, 60, 40, 2),   # strips wider than a tile
    (129, 60, 13, 2),   # interior of whole tiles and one column more
    (103, 48, 20, 1),   # four-side CPML: two rows between the bands
    (801, 803, 20, 2),  # the build for large grids, remainders both ways
    (801, 803, 20, 1),
]


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


def make(nx, nz, npd, bdy):
    flat = nx < 60 or nz < 30
    m = modelgen.make_solid_model(nx, nz, npd=npd, fpeak=40.0, nt=NT, src_x=[nx // 2, nx // 3],
                                  src_z=[min(nz - 4, 6 if bdy == 2 else 30)] * 2,
                                  amp=0.0 if flat else 4.0, boundary_type=bdy)
    m.thickness = max(m.thickness, m.h)
    return m


@pytest.mark.parametrize("nx,nz,npd,bdy", CASES)
def test_solid_tiles_match_the_oracle(mfdm, oracle, nx, nz, npd, bdy):
    m = make(nx, nz, npd, bdy)
    ref = oracle.forward_solid(m, NT, oracle.record_gap(m.dt), 32, final_fields=True)
    # vz on the row of the source is what symmetry leaves over: where the FP32
    # oracle's own error there is above TOL, two FP32 runs differ by up to twice that
    svz64 = oracle.forward_solid(m, NT, oracle.record_gap(m.dt), 64)["svz"]
    rec_tol = max(TOL, 2 * rel_l2(ref["svz"], svz64))
    with mfdm.SolidSolver.from_model(m) as s:
        s.set_shot(0)
        s.step(NT)
        assert rel_l2(s.records()["svz"], ref["svz"]) <= rec_tol
        for q, n in enumerate(("solid_vx", "solid_vz", "solid_sx", "solid_sz", "solid_sxz")):
            assert rel_l2(s.field(n), ref["solid"][q]) <= TOL, n


def test_a_new_shot_keeps_nothing_of_the_last(mfdm):
    """The captured steps outlive a change of shot: the source cell is read on the
    device, so each shot equals the same shot on a fresh handle bit for bit."""
    def shots(make_solver, names):
        def run(s, k):
            s.set_shot(k)
            s.step(NT)
            return [s.records()["svz"]] + [s.field(n) for n in names]
        with make_solver() as s:
            reused = [run(s, k) for k in (0, 1, 0)]
        for k, got in zip((0, 1, 0), reused):
            with make_solver() as s:
                for a, b in zip(got, run(s, k)):
                    assert np.array_equal(a, b)
        assert not np.array_equal(reused[0][1], reused[1][1])

    solid = make(129, 60, 13, 2)
    shots(lambda: mfdm.SolidSolver.from_model(solid), ["solid_vx", "solid_sz"])
    both = modelgen.curvilinear(160, 121, nt=NT)
    both.src_x, both.src_z = [60, 100], [both.src_z[0]] * 2
    shots(lambda: mfdm.Solver.from_model(both), ["solid_vx", "fluid_p"])
