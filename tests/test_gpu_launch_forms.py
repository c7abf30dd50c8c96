"""The plain path's face runs and one-cluster loop, and the bookkeeping of the
mixed general form's driver loop, over parts of their index space that
tests/test_gpu_plain_kernels.py leaves out: runs of two to eight faces with a short
last one along every axis, the loop with PLM and HLLE, steps to an end time."""
import numpy as np
import pytest

import test_gpu_plain_kernels as kernels
from helpers import oracle_config
from mara2_gb300.solver import Solver


# a thread takes (faces of an axis) / 233472 consecutive faces, at least two
# from twice that and at most eight
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(96, 82, 72), (850, 840, 1), (1380, 1370, 1)])
def test_face_runs_with_a_short_last_one_match_oracle(gpu_lib, port, shape):
    s, P = kernels._state("hydro", shape, "plm", "hllc", "outflow", 1, True)
    ref = P.copy()
    status, _, dts = port.run(oracle_config(s), ref, 1, s.cfl, s.t_final)
    assert status == 0
    with Solver(s, "fp64") as g:
        g.upload(P)
        g.advance(dts[0])
        g.synchronize()
        out = g.download()
    assert np.array_equal(out[s.interior()].view(np.uint64), ref[s.interior()].view(np.uint64))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [6, 33, 1000, 4096])
def test_plain_1d_loop_with_plm_and_hlle_matches_single_steps(gpu_lib, n):
    kernels.test_plain_1d_loop_matches_single_steps(gpu_lib, n, "outflow", "plm", "hlle", 2)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "mixed_fp64"])
@pytest.mark.parametrize("law,shape,recon,rk", [("hydro", (33, 6, 7), "plm", 2), ("hydro", (40, 21, 1), "weno5", 3),
                                                ("mhd", (20, 9, 7), "plm", 3), ("rmhd", (35, 9, 1), "plm", 1)])
def test_mixed_general_loop_matches_single_steps(gpu_lib, law, shape, recon, rk, precision):
    """Clock, step count and bits of the driver loop against the same steps
    taken one call at a time, in two runs and to an end time."""
    s, P = kernels._state(law, shape, recon, "hlle", "periodic", rk, False)

    def steps(count, t_final=np.inf):
        with Solver(s, precision) as g:
            g.upload(P)
            t, taken = 0.0, 0
            while taken < count and t < t_final:
                dt = min(s.cfl * g.courant(), t_final - t)
                g.advance(dt)
                t, taken = t + dt, taken + 1
            return g.download(), t, taken

    with Solver(s, precision) as g:
        g.upload(P)
        taken = g.run(4) + g.run(3)
        a, t = g.download(), g.t
    b, tb, nb = steps(7)
    assert (t, taken) == (tb, nb)
    assert np.array_equal(a.view(np.uint64), b.view(np.uint64))
    end = 0.6 * t
    with Solver(s, precision) as g:
        g.upload(P)
        taken = g.run(50, t_final=end)
        a, t = g.download(), g.t
    b, tb, nb = steps(50, end)
    assert (t, taken) == (tb, nb)
    assert np.array_equal(a.view(np.uint64), b.view(np.uint64))
