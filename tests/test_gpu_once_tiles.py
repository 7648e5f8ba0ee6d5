"""The stage kernels that accumulate once a step (grids from 2.5 M cells) on a B200, at
the edges of their tiling and in place in the adjoint's slots.

The other builds accumulate in every stage and are held to the FP32 oracle at these
edges on small grids (tests/test_gpu_stage_tiles.py); here build 4, which accumulates
once a step at these sizes, is held to build 3 on grids of the same edges, long in one
direction, from a state of noise in every cell.
"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

modelgen = importlib.import_module("marineseis-fdm-2d_b200.modelgen")

NT = 20
# Two forms of one FP32 scheme: a step's relative rounding is below 2^-22 (four stage
# roundings), 20 steps in one direction 5e-6, twice that for the two forms.
TOL = 1e-5

# nx, nz_f, nz_s, npd, boundary type
CASES = [
    (46, 27200, 27300, 20, 2),  # the side strips meet: no interior column
    (60001, 9, 35, 20, 2),      # fluid without interior rows, a bottom band near the interface
    (1600, 790, 800, 0, 2),     # no absorbing strip
    (1601, 790, 800, 40, 2),    # strips wider than a tile
    (1633, 779, 780, 13, 2),    # interior of whole tiles and one column more
    (1703, 742, 747, 20, 1),    # four-side CPML
    (40003, 23, 40, 20, 1),     # the top band reaches the conservative rows
]


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


def model(nx, nz_f, nz_s, npd, bdy, nt=NT):
    m = modelgen.make_model(nx, nz_f, nz_s, npd=npd, fpeak=40.0, nt=nt, src_x=[nx // 2],
                            src_z=[max(3, nz_f - 6)], amp=0.0, boundary_type=bdy,
                            flat_sides=2 * npd + 20 < nx)
    m.thickness = max(m.thickness, m.h)
    return m


@pytest.mark.parametrize("nx,nz_f,nz_s,npd,bdy", CASES)
def test_once_a_step_matches_every_stage(mfdm, nx, nz_f, nz_s, npd, bdy):
    assert nx * (nz_f + nz_s) >= 2_500_000
    m = model(nx, nz_f, nz_s, npd, bdy)
    rng = np.random.default_rng([nx, nz_f])
    start = {}
    for name in mfdm.FIELDS:  # velocities of 1 um/s beside stresses of about rho c times that
        rows = nz_f if name.startswith("fluid") else nz_s
        scale = 1e-6 if name.endswith(("vx", "vz")) else 5.0
        start[name] = scale * rng.standard_normal((rows, nx)).astype(np.float32)

    def run(build, seg):
        with mfdm.Solver.from_model(m) as s:
            s.set_blocks_per_sm(build)
            s.set_tile(seg)
            for name, v in start.items():
                s.set_field(name, v)
            s.step(NT)
            return {**{n: s.field(n) for n in mfdm.FIELDS}, **s.records()}

    want = run(3, 8)
    for seg in (0, 8, 48):
        got = run(4, seg)
        assert any(not np.array_equal(got[q], want[q]) for q in want)  # another form indeed
        for q in want:
            assert np.all(np.isfinite(got[q])) and np.any(want[q]), q
            assert rel_l2(got[q], want[q]) <= TOL, (seg, q)


def test_adjoint_in_place_above_the_line(mfdm):
    """Kept, recomputed and twice recomputed steps run in place in slot buffers: the
    same kernels on the same values, so records and gradients are equal bit for bit."""
    nt, every = 12, 4
    m = model(1703, 742, 760, 20, 2, nt=nt)
    rng = np.random.default_rng(5)
    out = []
    with mfdm.Solver.from_model(m) as s:
        s.set_shot(0, reset=True)
        info = s.info()
        assert info["blocks_per_sm"] == 4
        s.step(nt)
        plain = s.records()
        ns = -(-nt // info["gap"])
        res = {k: rng.standard_normal((ns, m.nx)).astype(np.float32) for k in ("svx", "svz", "fp")}
        segment = every * 4 * 4 * 8 * (info["nz_f"] + info["nz_s"]) * info["pitch"]
        for memory, inner in ((0, 0), (2 * segment, 0), (1 << 40, 0), (0, 2)):
            s.adjoint_memory(memory)
            s.adjoint_inner(inner)
            rec = s.adjoint_forward(nt, ckpt_every=every)
            for k in rec:
                assert np.array_equal(rec[k], plain[k]), (memory, inner, k)
            out.append(s.adjoint_backward(res))
    for g in out[1:]:
        for k in g:
            assert np.any(g[k]) and np.array_equal(g[k], out[0][k]), k
