"""A kernel that is launched while its predecessor still runs (it begins with,
or later executes, griddepcontrol.wait) must not read that predecessor's data
through the read-only path: ld.global.nc, which __ldg and const __restrict__
pointers give, promises data that nothing writes while the kernel exists."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mara2_gb300", "csrc")
# read by kernels of the step, but written only before it: grid and tile tables
TABLES = {"grids", "tiles", "ntiles_p", "rot"}
WAITS = ("pdl_chain();", "pdl_wait();", "griddepcontrol.wait")


def _code(path):
    text = open(path).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _kernels(text):
    """(name, parameters, body) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void(?:\s+__launch_bounds__\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\))?\s*(\w+)\s*\(", text):
        i, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params, j = text[m.end():i - 1], text.index("{", i)
        k, depth = j + 1, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), params, text[j:k]


def test_kernels_of_a_chain_take_no_read_only_loads():
    waiting = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        text = _code(path)
        kernels = [k for k in _kernels(text) if any(w in k[2] for w in WAITS)]
        waiting += [name for name, _, _ in kernels]
        for name, params, _ in kernels:
            for p in params.split(","):
                read_only = re.search(r"\bconst\b[^*]*\*\s*__restrict__\s+(\w+)", p)
                assert not read_only or read_only.group(1) in TABLES, (os.path.basename(path), name, p.strip())
        assert not kernels or "__ldg" not in text, os.path.basename(path)
    assert {"flux_f_kernel", "update_f_kernel", "ct_emf_kernel", "hydro_tile_kernel", "flux_tile_kernel", "flux_run_kernel",
            "flux_general_kernel", "update_kernel", "courant_kernel", "k_advance_time"} <= set(waiting)
