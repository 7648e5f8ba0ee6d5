"""The stage kernels' tiling at the sizes where it can go wrong, on a B200.

A stage launch cuts the grid into interface columns, conservative rows, PML
tiles (32 x 8) and interior tiles (32 columns, a multiple of 8 rows). Each case
below has an edge of that cut: the smallest grid, no interior columns or rows,
no PML at all, a strip wider than a tile, tiles of one column or one row. Every
build and a short and a tall tile are held to the FP32 oracle.
"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

modelgen = importlib.import_module("marineseis-fdm-2d_b200.modelgen")

NT = 60
# Both run the same FP32 operator; a step's relative rounding is below 2^-22 (four
# stage roundings), 60 steps in one direction 1.5e-5, as a random walk 2e-6.
TOL = 1e-5

# nx, nz_f, nz_s, npd, boundary type
CASES = [
    (8, 8, 8, 1, 2),        # the smallest grid: no interior at all
    (46, 24, 24, 20, 2),    # the side strips meet: no interior column
    (97, 9, 31, 20, 2),     # fluid without interior rows
    (99, 30, 23, 20, 2),    # the bottom band reaches the first solid rows
    (70, 40, 41, 0, 2),     # no absorbing strip
    (161, 50, 60, 40, 2),   # strips wider than a tile
    (129, 41, 52, 13, 2),   # interior of whole tiles and one column more
    (103, 42, 47, 20, 1),   # four-side CPML
    (75, 23, 40, 20, 1),    # the top band reaches the conservative rows
]


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("nx,nz_f,nz_s,npd,bdy", CASES)
def test_tiles_match_the_oracle(mfdm, oracle, nx, nz_f, nz_s, npd, bdy):
    flat = nx < 60 or nz_f < 20
    m = modelgen.make_model(nx, nz_f, nz_s, npd=npd, fpeak=40.0, nt=NT, src_x=[nx // 2],
                            src_z=[max(3, nz_f - 6)], amp=0.0 if flat else 6.0, wavelength=150.0,
                            perturb=0.0 if flat else 0.05, corr_len=20.0, seed=3,
                            boundary_type=bdy, flat_sides=2 * npd + 20 < nx)
    m.thickness = max(m.thickness, m.h)
    ref = oracle.forward(m, NT, oracle.record_gap(m.dt), precision=32, final_fields=True)
    names = list(mfdm.FIELDS)
    want = dict(zip(names, list(ref["fluid"]) + list(ref["solid"])))
    for blocks in (2, 3, 4):
        for seg in (8, 48):
            with mfdm.Solver.from_model(m) as s:
                s.set_blocks_per_sm(blocks)
                s.set_tile(seg)
                s.set_shot(0)
                s.step(NT)
                rec = s.records()
                for q in ("svx", "svz", "fp"):
                    assert rel_l2(rec[q], ref[q]) <= TOL, (blocks, seg, q)
                for n in names:
                    assert rel_l2(s.field(n), want[n]) <= TOL, (blocks, seg, n)


def test_batch_of_many_cells_matches_one_shot(mfdm):
    """A batch above 2.5 M cells accumulates once a step, one of its shots alone
    in every stage: the same scheme, so they agree to FP32 rounding (2^-24 a
    rounding, at most four a step, the cancellation of the once-a-step weights
    included: 1e-5 over 60 steps)."""
    m = modelgen.curvilinear(320, 200, nt=NT)
    shots = [(40 + 6 * k, m.src_z[0], 25.0, m.beta0) for k in range(40)]  # 2.57 M cells
    with mfdm.Batch.from_model(m, shots) as b:
        b.step(NT)
        got = [(b.records(shot=k), b.field("fluid_p", shot=k)) for k in (0, 39)]
    for (rec, p), (x, z, f, beta0) in zip(got, (shots[0], shots[39])):
        one = modelgen.curvilinear(320, 200, nt=NT)
        one.src_x, one.src_z, one.fpeak, one.beta0 = [x], [z], f, beta0
        with mfdm.Solver.from_model(one) as s:
            s.step(NT)
            assert rel_l2(p, s.field("fluid_p")) <= TOL
            ref = s.records()
            for q in rec:
                assert rel_l2(rec[q], ref[q]) <= TOL, q


@pytest.mark.parametrize("nx,nz_f,nz_s,bdy", [(46, 24, 24, 2), (160, 60, 61, 2), (403, 150, 151, 1),
                                              (1000, 300, 301, 2)])
def test_chained_launches_equal_plain_ones(mfdm, nx, nz_f, nz_s, bdy):
    """Captured steps let a stage launch start as the one before it ends; timing
    each kernel launches them one after the other. The same kernels on the same
    data: equal bit for bit (both builds below 2.5 M cells, 96 steps)."""
    m = modelgen.make_model(nx, nz_f, nz_s, npd=20, fpeak=20.0, nt=96, src_x=[nx // 2],
                            src_z=[nz_f - 8 if nz_f < 40 else nz_f // 2], boundary_type=bdy)
    out = []
    for per_kernel in (False, True):
        with mfdm.Solver.from_model(m) as s:
            s.set_shot(0)
            s.time_steps(96, per_kernel=per_kernel)
            out.append([s.field(n) for n in mfdm.FIELDS] + list(s.records().values()))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
