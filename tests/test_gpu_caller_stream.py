"""mfdm_update_rk4 on the caller's own stream on a B200: samples that are still to be
written when the receiver buffer grows are not lost."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

modelgen = importlib.import_module("marineseis-fdm-2d_b200.modelgen")


def test_records_grow_behind_pending_steps(mfdm):
    import torch
    m = modelgen.make_model(97, 40, 44, npd=10, fpeak=40.0, dt=2.5e-4, nt=6, src_x=[48], src_z=[30])
    # a sample every 4 steps; room for 6 steps' source values and 2 samples, doubled as
    # needed: step 24 finds no more room for the first, step 32 for the second alone
    nt = 40
    out = []
    for own in (False, True):
        with mfdm.Solver.from_model(m) as s:
            s.set_shot(0, reset=True)
            stream = torch.cuda.Stream() if own else None
            assert s.info()["gap"] == 4
            for it in range(nt):
                if own and it == 28:
                    with torch.cuda.stream(stream):
                        torch.cuda._sleep(100_000_000)  # the steps from here wait about 50 ms
                s.update_rk4(it, stream.cuda_stream if own else None)
            if own:
                stream.synchronize()
            s.synchronize()
            out.append(s.records())
    assert np.any(out[0]["fp"][:3])
    for q in out[0]:
        assert np.array_equal(out[1][q], out[0][q]), q
