"""The plain FP64 path's flux tiles, flux runs and one-cluster driver loop, and
the mixed general update's slice-wide launch, at the sizes where their index
arithmetic can go wrong: a tile holds 32 faces along x, or 8 along y and z in
four columns; runs of faces begin at 2^17 zones; a cluster shares up to 4096
zones of a 1-D grid among up to 16 blocks.

Hydro and MHD match the oracle bit for bit; RMHD to 1e-12 (the oracle calls
the host's acos, cos and sin, which are not correctly rounded everywhere)."""
import numpy as np
import pytest

from helpers import oracle_config, parity_error, rel_l1_max
from mara2_gb300 import workloads as W
from mara2_gb300.scheme import Scheme
from mara2_gb300.solver import Solver


def _state(law, shape, recon, riemann, bc, rk, odd):
    """A rough state (a jump in every zone).  ``odd``: some zones hold values
    that the lean forms hand to the general ones (subnormal velocities and
    fields, zeros of both signs)."""
    s = Scheme(law=law, recon=recon, riemann=riemann, bc=bc, rk_order=rk, shape=shape, plm_theta=1.5,
               gamma=4.0 / 3 if law == "rmhd" else 5.0 / 3, cfl=0.3, t_final=None, steps=2)
    rng = np.random.default_rng(sum(shape) + rk)
    P = W.empty_state(s)
    n = P[s.interior()].shape[:-1]
    Q = np.zeros(n + (P.shape[-1],))
    Q[..., 0] = rng.uniform(0.5, 2.0, n)
    Q[..., 1:4] = rng.uniform(-0.3, 0.3, n + (3,))
    Q[..., 4] = rng.uniform(0.5, 2.0, n)
    if law != "hydro":
        Q[..., 5:8] = rng.uniform(-0.5, 0.5, n + (3,))
    if odd:
        pick = rng.random(n) < 0.03
        for q in range(1, Q.shape[-1]):
            if q != 4:
                Q[..., q] = np.where(pick, rng.choice([0.0, -0.0, 3e-310, -7e-312, 1e-170]), Q[..., q])
    P[s.interior()] = Q
    return s, W.apply_bc_numpy(s, P)


TILES = [
    # law, shape, recon, riemann, bc, rk, odd
    ("hydro", (31, 1, 1), "plm", "hlle", "outflow", 1, False),
    ("hydro", (32, 7, 1), "plm", "hllc", "periodic", 2, True),
    ("hydro", (33, 9, 1), "weno5", "hllc", "reflecting", 1, True),
    ("hydro", (6, 65, 1), "weno5", "hlle", "outflow", 2, False),
    ("hydro", (63, 6, 17), "pcm", "hlle", "periodic", 2, True),
    ("hydro", (8, 33, 8), "plm", "hlle", "reflecting", 3, False),
    ("mhd", (31, 33, 1), "plm", "hlle", "periodic", 2, True),
    ("mhd", (6, 7, 33), "weno5", "hlle", "periodic", 1, False),
    ("mhd", (33, 6, 8), "pcm", "hlle", "outflow", 3, True),
    ("mhd", (34, 9, 1), "plm", "hllc", "periodic", 1, False),
    ("rmhd", (33, 8, 1), "weno5", "hlle", "outflow", 2, False),
    ("rmhd", (35, 9, 1), "weno5", "hlle", "periodic", 2, True),
    ("rmhd", (7, 6, 10), "plm", "hlle", "periodic", 1, True),
    # one below and above the size from which PLM HLLC goes in runs, on each axis
    ("hydro", (363, 361, 1), "plm", "hllc", "outflow", 1, False),
    ("hydro", (362, 363, 1), "plm", "hllc", "outflow", 1, True),
    ("hydro", (131072, 1, 1), "plm", "hllc", "reflecting", 1, False),
    ("hydro", (51, 37, 71), "plm", "hllc", "periodic", 1, True),
    # runs of more than one face, the last one short
    ("hydro", (787, 797, 1), "plm", "hllc", "outflow", 1, False),
]


@pytest.mark.gpu
@pytest.mark.parametrize("law,shape,recon,riemann,bc,rk,odd", TILES)
def test_plain_flux_launches_match_oracle(gpu_lib, port, law, shape, recon, riemann, bc, rk, odd):
    s, P = _state(law, shape, recon, riemann, bc, rk, odd)
    c = oracle_config(s)
    ref = P.copy()
    status, _, dts = port.run(c, ref, 2, s.cfl, s.t_final)
    assert status == 0
    with Solver(s, "fp64") as g:
        g.upload(P.copy())
        for dt in dts:
            g.advance(dt)
        g.synchronize()
        out = g.download()
    if law == "rmhd":
        assert np.all(parity_error(s, out[s.interior()], ref[s.interior()]) <= 1e-12)
    else:
        assert np.array_equal(out[s.interior()].view(np.uint64), ref[s.interior()].view(np.uint64))


@pytest.mark.gpu
@pytest.mark.parametrize("n", [6, 31, 33, 64, 100, 513, 1024, 4096, 4097])
@pytest.mark.parametrize("bc,recon,riemann,rk", [("outflow", "plm", "hllc", 2), ("periodic", "pcm", "hlle", 1),
                                                 ("reflecting", "weno5", "hllc", 3)])
def test_plain_1d_loop_matches_single_steps(gpu_lib, n, bc, recon, riemann, rk):
    """The driver loop on one cluster against the same steps taken one call at
    a time by the step kernels: clock, step count and bits, in two runs and
    to an end time inside a launch."""
    s, P = _state("hydro", (n, 1, 1), recon, riemann, bc, rk, True)

    def steps(count, t_final=np.inf):
        with Solver(s, "fp64") as g:
            g.upload(P.copy())
            t, taken = 0.0, 0
            while taken < count and t < t_final:
                dt = min(g.courant() * s.cfl, t_final - t)
                g.advance(dt)
                t, taken = t + dt, taken + 1
            return g.download(), t, taken

    with Solver(s, "fp64") as g:
        g.upload(P.copy())
        taken = g.run(4) + g.run(3)
        a, t = g.download(), g.t
    b, tb, nb = steps(7)
    assert (t, taken) == (tb, nb)
    assert np.array_equal(a.view(np.uint64), b.view(np.uint64))
    end = 0.6 * t
    with Solver(s, "fp64") as g:
        g.upload(P.copy())
        taken = g.run(50, t_final=end)
        a, t = g.download(), g.t
    b, tb, nb = steps(50, end)
    assert (t, taken) == (tb, nb)
    assert np.array_equal(a.view(np.uint64), b.view(np.uint64))


# rows whose last block would be nearly empty (the launch indexes a whole
# slice), rows that fill their blocks (a block per row), and one past them
@pytest.mark.gpu
@pytest.mark.parametrize("law,shape", [("hydro", (120, 7, 5)), ("hydro", (121, 5, 6)), ("hydro", (33, 6, 7)),
                                       ("mhd", (128, 6, 6)), ("mhd", (129, 7, 5)), ("rmhd", (130, 9, 1))])
@pytest.mark.parametrize("precision", ["mixed", "mixed_fp64"])
def test_mixed_general_update_ragged_rows(gpu_lib, port, law, shape, precision):
    s, P = _state(law, shape, "plm", "hlle", "periodic", 2, False)
    ref = P.copy()
    status, _, dts = port.run(oracle_config(s), ref, 2, s.cfl, s.t_final)
    assert status == 0
    with Solver(s, precision) as g:
        g.upload(P.copy())
        for dt in dts:
            g.advance(dt)
        g.synchronize()
        out = g.download()
    # the mixed path's contract: 1e-5 of each field's L1 norm
    assert np.all(rel_l1_max(out[s.interior()], ref[s.interior()]) <= 1e-5)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,recon,rk,cooling", [((70, 33, 1), "plm", 2, -1.0), ((33, 40, 1), "weno5", 3, -1.0),
                                                    ((9, 10, 12), "pcm", 1, -1.0), ((17, 9, 11), "plm", 2, 0.1),
                                                    ((40, 1, 1), "weno5", 2, -1.0)])
def test_plain_mhd_in_a_medium_with_small_fields_matches_oracle(gpu_lib, port, shape, recon, rk, cooling):
    """A hot region in a medium at rest with a field along x, whose transverse
    fields and velocities are of 1e-100 to 1e-300 (and some subnormal or zero),
    as a wave leaves them ahead of it."""
    s = Scheme(law="mhd", recon=recon, riemann="hlle", bc="outflow", rk_order=rk, shape=shape, cfl=0.3,
               cooling_rate=cooling)
    rng = np.random.default_rng(sum(shape) + rk)
    P = W.empty_state(s)
    Q = np.zeros(shape + (P.shape[-1],))
    Q[..., 0] = 1.0
    Q[..., 4] = np.where(rng.random(shape) < 0.1, 10.0, 0.1)
    Q[..., 5] = 0.5
    for q in (2, 3, 6, 7):
        Q[..., q] = 10.0 ** -rng.uniform(100, 300, shape) * rng.choice([-1.0, 1.0], shape)
        Q[..., q] = np.where(rng.random(shape) < 0.1, rng.choice([0.0, -0.0, 3e-310, 1e-30], shape), Q[..., q])
    P[s.interior()] = Q
    P = W.apply_bc_numpy(s, P)
    ref = P.copy()
    status, _, dts = port.run(oracle_config(s), ref, 3, s.cfl, s.t_final)
    assert status == 0
    with Solver(s, "fp64") as g:
        g.upload(P.copy())
        for dt in dts:
            assert s.cfl * g.courant() == dt
            g.advance(dt)
        g.synchronize()
        out = g.download()
    assert np.array_equal(out[s.interior()].view(np.uint64), ref[s.interior()].view(np.uint64))


# tiles: one launch of fluxes a stage for all axes; face runs (hydro, PLM, HLLC
# from 2^17 zones) and magnetic HLLC: one per axis
@pytest.mark.gpu
@pytest.mark.parametrize("law,shape,recon,riemann,launches", [("hydro", (40, 30, 1), "plm", "hllc", 1),
                                                              ("hydro", (400, 400, 1), "plm", "hllc", 2),
                                                              ("hydro", (60, 50, 50), "plm", "hllc", 3),
                                                              ("mhd", (8, 9, 10), "pcm", "hllc", 3),
                                                              ("mhd", (24, 20, 1), "weno5", "hlle", 1)])
def test_kernel_timing_counts_every_plain_launch(gpu_lib, law, shape, recon, riemann, launches):
    s, P = _state(law, shape, recon, riemann, "periodic", 2, False)
    with Solver(s, "fp64") as g:
        g.upload(P.copy())
        dt = 0.1 * s.cfl * g.courant()
        g.set_kernel_timing(True)
        before = g.stats().kernel_launches
        g.advance(dt)
        g.advance(dt)
        enqueued = g.stats().kernel_launches - before
        ms, n = g.kernel_times()
        g.set_kernel_timing(False)
    assert n[0] == 2 * s.rk_order * launches and n[1] == 2 * s.rk_order, n
    assert n[0] + n[1] + 4 == enqueued      # and dt and the step count, once a step each
    assert ms[0] > 0.0 and ms[1] > 0.0
