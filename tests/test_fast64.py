"""The plain path's forms with fewer FP64 operations (mara2_gb300/csrc/
fast64.cuh, fast64_rmhd.cuh, ieee64.cuh, ziv64.cuh), built for the host, bit for bit the general ones
(physics_fp64.cuh, crmath.cuh) and the host's own division, square root and product:
every law, reconstruction, solver, axis and smoothness indicator they cover,
on seeded operands - smooth states, exact zeros of either sign and equal
states, strong jumps, wide magnitudes, and any bit patterns (infinities, NaNs,
subnormals), which the forms must refuse or get right.  The hardware's seeds
of the division and square root enter within a few units in the last place,
so those are tested with seeds shifted both ways."""
import ctypes as C
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
HYDRO, MHD, RMHD, MHD_COOL = 0, 1, 2, 3
SMOOTH, ZEROS, JUMPS, WIDE, ANY, SMALL = range(6)
SMALL_MAGNETIC = 6


def _build(path, ulps, *flags):
    cxx = shutil.which("g++")
    if cxx is None or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    so = os.path.join(str(path), f"libfast64_{ulps}.so")
    subprocess.run([cxx, "-O2", "-ffp-contract=off", "-std=c++17", "-fPIC", "-shared", f"-DIEEE64_SEED_ULPS={ulps}", *flags,
                    "-I" + os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "fast64_probe.cpp"), "-o", so],
                   check=True)
    lib = C.CDLL(so)
    for f in ("probe_ieee",) if flags else ("probe_faces", "probe_zones", "probe_ieee", "probe_ziv"):
        getattr(lib, f).restype = C.c_long
    return lib


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return _build(tmp_path_factory.mktemp("fast64"), 0)


@pytest.mark.parametrize("ulps", [-2, 0, 2])
def test_integer_division_root_and_product_round_correctly(tmp_path, ulps):
    acc = C.c_long()
    n = 400000
    assert _build(tmp_path, ulps, "-DPROBE_IEEE_ONLY").probe_ieee(C.c_long(n), C.c_ulonglong(5), C.byref(acc)) == 0
    assert acc.value > 2.8 * n


CASES = [(HYDRO, r, s) for r in range(3) for s in range(2)] + [(law, r, 0) for law in (MHD, RMHD, MHD_COOL) for r in range(3)]


@pytest.mark.parametrize("law,recon,riemann", CASES)
def test_face_flux_has_the_general_forms_bits(lib, law, recon, riemann):
    n = 4000
    acc = C.c_long()
    for axis, gamma, theta in ((0, 5.0 / 3, 1.5), (1, 1.4, 1.0), (2, 4.0 / 3, 2.0)):
        for weno in (range(3) if recon == 2 else (2,)):
            for kind in range(6):
                bad = lib.probe_faces(C.c_long(n), C.c_ulonglong(100 * kind + axis), law, recon, riemann, axis, weno,
                                      C.c_double(gamma), C.c_double(theta), kind, C.byref(acc))
                assert bad == 0, (axis, weno, kind)
                if kind in (SMOOTH, ZEROS):
                    assert acc.value == n
                if kind == SMALL and law == RMHD:
                    assert acc.value > n / 2


@pytest.mark.parametrize("law", [HYDRO, MHD, RMHD, MHD_COOL])
def test_zone_conversions_and_wave_speeds_have_the_general_forms_bits(lib, law):
    n = 20000
    acc = C.c_long()
    for kind in range(6):
        assert lib.probe_zones(C.c_long(n), C.c_ulonglong(kind), law, C.c_double(5.0 / 3), kind, C.byref(acc)) == 0
        if kind in (SMOOTH, ZEROS, JUMPS):
            assert acc.value == n


def test_two_phase_functions_round_as_the_accurate_ones(lib):
    n = 200000
    acc = C.c_long()
    assert lib.probe_ziv(C.c_long(n), C.c_ulonglong(3), C.byref(acc)) == 0
    assert acc.value > 2.9 * n


# Density (and pressure) and velocity of five zones of ordinary magnitudes
# whose WENO5 value at the right edge of the middle one nearly vanishes
# (2^-153 and 2^-436), so that the density of kinetic energy there is subnormal.
EDGE_RHO = "0x1.845f67b9a7b48p-99 0x1.8f7b8e6bad8bcp-98 0x1.1ac7f23636d4bp-100 0x1.0e9e382c71194p-100 0x1.cb435c8e74616p-100"
EDGE_V = "-0x1.49592ff5d47c9p-328 -0x1.8b37d326fefbep-329 -0x1.077a8cc4a9fd4p-330 0x1.077a8cc4a9fd4p-330 0x1.8b37d326fefcp-329"


def test_weno_edges_that_nearly_vanish_are_refused_or_right(lib):
    rho, v = ([float.fromhex(x) for x in line.split()] for line in (EDGE_RHO, EDGE_V))
    Z = [(rho[min(s, 4)],) + 3 * (v[min(s, 4)],) + (rho[min(s, 4)],) for s in range(6)]
    flat = (C.c_double * 30)(*[x for z in Z for x in z])
    assert lib.probe_hydro_weno_face(flat, 2) <= 0
    # the same zones of magnitude one are taken
    flat = (C.c_double * 30)(*[x * 2.0 ** (330 if 0 < q < 4 else 100) for z in Z for q, x in enumerate(z)])
    assert lib.probe_hydro_weno_face(flat, 2) == 0


@pytest.mark.parametrize("kind", [SMALL, SMALL_MAGNETIC])
@pytest.mark.parametrize("law", [MHD, MHD_COOL])
@pytest.mark.parametrize("recon", range(3))
def test_small_fields_of_mhd_take_the_lean_forms(lib, law, recon, kind):
    """Ahead of a wave into a medium at rest, transverse fields and velocities
    fall to 1e-270 and stay: the lean forms have to take such faces and zones,
    with the general bits."""
    n = 6000
    acc = C.c_long()
    for axis in range(3):
        for weno in (range(3) if recon == 2 else (2,)):
            assert lib.probe_faces(C.c_long(n), C.c_ulonglong(7 + axis), law, recon, 0, axis, weno, C.c_double(5.0 / 3),
                                   C.c_double(1.5), kind, C.byref(acc)) == 0
            assert acc.value > 0.6 * n
    assert lib.probe_zones(C.c_long(20000), C.c_ulonglong(11), law, C.c_double(5.0 / 3), kind, C.byref(acc)) == 0
    assert acc.value > 0.6 * 20000


@pytest.mark.parametrize("law", [HYDRO, MHD, RMHD, MHD_COOL])
@pytest.mark.parametrize("gamma,theta", [(1.001, 1.5), (1.0 + 1e-6, 2.0), (5.0 / 3, 0.0)])
def test_nearly_isothermal_gases_and_unlimited_slopes_take_the_lean_forms(lib, law, gamma, theta):
    n = 3000
    acc = C.c_long()
    # (the relativistic law loses a third of these states' wave speeds to
    # rounding at gamma - 1 = 1e-6, by the general functions too)
    most = 0.9 if law != RMHD or gamma > 1.0001 else 0.0
    for recon in range(3):
        for axis in range(3):
            for kind in (SMOOTH, ZEROS, JUMPS, WIDE, ANY):
                for riemann in ((0, 1) if law == HYDRO else (0,)):
                    assert lib.probe_faces(C.c_long(n), C.c_ulonglong(50 * kind + axis), law, recon, riemann, axis, 2,
                                           C.c_double(gamma), C.c_double(theta), kind, C.byref(acc)) == 0
                    if kind == SMOOTH:
                        assert acc.value > most * n
    for kind in (SMOOTH, JUMPS, WIDE, ANY):
        assert lib.probe_zones(C.c_long(10000), C.c_ulonglong(kind), law, C.c_double(gamma), kind, C.byref(acc)) == 0
        if kind == SMOOTH:
            assert acc.value > most * 10000
