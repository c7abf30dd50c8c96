"""Relativistic MHD states through the mixed path's host boundary: the upload
forms the conserved densities, the download recovers the primitives by a
Newton iteration that starts from the zone's FP32 primitives.

An FP64 accumulator holds the densities to FP64, so the recovery has to return
what was uploaded.  It stops at a step of 1e-12 in Z and W; with rho = D / W,
v = (S + b0 B / W) / (Z + B^2), |b0 B / W| and |S| at most Z + B^2, and
p = (Z / W^2 - D / W) (gamma - 1) / gamma with Z / W^2 = rho h and D / W = rho,
errors of 1e-12 in Z and W give at most 1e-12 of rho, 4e-12 of 1 in v and
3e-12 (h + 1) rho in p; rounding of the densities and of the iteration's residual
adds W^2 rho h 2^-50 to p and 2^-50 W^2 to v and rho."""
import numpy as np
import pytest

from helpers import oracle_config
from mara2_gb300 import workloads as W
from mara2_gb300.scheme import Scheme
from mara2_gb300.solver import Solver

G = 4.0 / 3


@pytest.mark.gpu
@pytest.mark.parametrize("w_max,p_min", [(1.5, 0.1), (6.0, 0.01), (20.0, 0.1)])
@pytest.mark.parametrize("small", [False, True])
def test_rmhd_download_returns_what_was_uploaded(gpu_lib, port, w_max, p_min, small):
    """small: some zones with fields of 1e-200, as a wave into a medium at rest
    leaves them, subnormal ones and zeros.  A zone that the oracle refuses (it
    finds no wave speeds in some fast ones) is put at rest; one that only the
    mixed path's upload refuses has to come back all the same."""
    shape = (40, 33, 1)
    s = Scheme(law="rmhd", recon="plm", riemann="hlle", bc="outflow", rk_order=2, shape=shape, gamma=G, cfl=0.3)
    rng = np.random.default_rng(int(10 * w_max) + small)
    P = W.empty_state(s)
    Q = np.zeros(shape + (8,))
    lorentz = 1.0 + (w_max - 1.0) * rng.random(shape)
    v = np.sqrt(1.0 - lorentz ** -2)
    n = rng.normal(size=shape + (3,))
    Q[..., 0] = rng.uniform(0.5, 2.0, shape)
    Q[..., 1:4] = n / np.linalg.norm(n, axis=-1, keepdims=True) * v[..., None]
    Q[..., 4] = p_min * 10.0 ** rng.uniform(0.0, 2.0, shape)
    Q[..., 5:8] = rng.uniform(-0.5, 0.5, shape + (3,))
    if small:
        for q in (2, 3, 5, 6, 7):
            pick = rng.random(shape) < 0.3
            Q[..., q] = np.where(pick, rng.choice([1e-200, -3e-150, 2e-110, 4e-310, 0.0], shape), Q[..., q])
    c = oracle_config(s)
    refused = np.array([port.from_primitive(c, z)[0] != 0 for z in Q.reshape(-1, 8)]).reshape(shape)
    assert np.mean(refused) < 0.5
    Q[refused, 1:4] = 0.0
    lorentz = 1.0 / np.sqrt(1.0 - np.sum(Q[..., 1:4] ** 2, axis=-1))
    P[s.interior()] = Q
    P = W.apply_bc_numpy(s, P)
    with Solver(s, "mixed_fp64") as g:
        g.upload(P.copy())
        out = g.download()[s.interior()]
    rho, p = Q[..., 0], Q[..., 4]
    h = 1.0 + G / (G - 1.0) * p / rho
    eps = 2.0 ** -50 * lorentz ** 2
    assert np.all(np.abs(out[..., 0] - rho) <= (1e-12 + eps) * rho)
    assert np.all(np.abs(out[..., 1:4] - Q[..., 1:4]) <= (4e-12 + eps)[..., None])
    assert np.all(np.abs(out[..., 4] - p) <= 3e-12 * (h + 1.0) * rho + eps * rho * h)
    assert np.array_equal(out[..., 5:8].view(np.uint64), Q[..., 5:8].view(np.uint64))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["mixed", "mixed_fp64"])
def test_zone_that_cannot_be_recovered_keeps_its_primitives(gpu_lib, precision):
    """A step far too long leaves densities without primitives: the step fails
    (code 16), and such a zone's primitives are those it had, in FP32."""
    shape = (24, 20, 1)
    s = Scheme(law="rmhd", recon="pcm", riemann="hlle", bc="outflow", rk_order=1, shape=shape, gamma=G, cfl=0.3)
    rng = np.random.default_rng(3)
    P = W.empty_state(s)
    Q = np.zeros(shape + (8,))
    Q[..., 0] = rng.uniform(0.5, 2.0, shape)
    Q[..., 1:4] = rng.uniform(-0.3, 0.3, shape + (3,))
    Q[..., 4] = rng.uniform(0.1, 2.0, shape)
    Q[..., 5:8] = rng.uniform(-0.5, 0.5, shape + (3,))
    P[s.interior()] = Q
    P = W.apply_bc_numpy(s, P)
    with Solver(s, precision) as g:
        g.upload(P.copy())
        g.advance(2.0)
        assert g.status() == 16
        st = g.stats()
        zone = tuple(st.first_zone)
        assert st.failures > 0
        out = g.download()[s.interior()]
    assert np.array_equal(out[zone].astype(np.float32), Q[zone].astype(np.float32))
    assert np.all(np.isfinite(out))


@pytest.mark.gpu
def test_rmhd_upload_of_small_fields_costs_what_others_do(gpu_lib):
    """Fields of 1e-200, as a plain run leaves them ahead of a wave, take the
    lean conversion too: by the general functions the upload takes six times
    as long (512^2: 1.54 against 0.25 ms), so a factor of three apart they are
    not the same conversion."""
    import time

    shape = (512, 512, 1)
    s = Scheme(law="rmhd", recon="plm", riemann="hlle", bc="outflow", rk_order=2, shape=shape, gamma=G, cfl=0.3)
    rng = np.random.default_rng(7)
    Q = np.zeros(shape + (8,))
    Q[..., 0] = rng.uniform(0.9, 1.1, shape)
    Q[..., 1:4] = rng.uniform(-0.1, 0.1, shape + (3,))
    Q[..., 4] = rng.uniform(0.9, 1.1, shape)
    Q[..., 5:8] = rng.uniform(-0.3, 0.3, shape + (3,))
    best = {}
    with Solver(s, "mixed") as g:
        for small in (False, True):
            if small:
                Q[..., 6] *= 1e-200
            P = W.empty_state(s)
            P[s.interior()] = Q
            P = W.apply_bc_numpy(s, P)
            for _ in range(8):
                t = time.perf_counter()
                g.upload(P)
                g.synchronize()
                best[small] = min(best.get(small, 1e9), time.perf_counter() - t)
    assert best[True] < 3.0 * best[False], best
