"""Build and smoke entry points.

build(): compiles the CUDA library for sm_103a (mara2_gb300/build.py), the
oracle restatement (oracle/Makefile) and, where the reference's sources are
at hand, the reference's own hot-path translation units for the oracle
cross-check and the CPU baseline.  The sources are looked up in
$MARA_REF_SRC, else in the git-ignored baseline/_ref/src, which is filled
from the reference tree ($MARA_REF_TREE) on a machine that has it.

smoke(): one small plain-FP64 advance of a Sod shock tube on cuda:0 through
the C ABI, checked against the oracle.
"""
from __future__ import annotations

import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def build() -> None:
    from mara2_gb300 import build as B
    B.build()
    oracle_dir = os.path.join(ROOT, "oracle")
    subprocess.run(["make", "-s", "-C", oracle_dir], check=True)
    ref_src = os.environ.get("MARA_REF_SRC", os.path.join(ROOT, "baseline", "_ref", "src"))
    tree = os.environ.get("MARA_REF_TREE", "/root/reference")
    if tree and os.path.isdir(os.path.join(tree, "src")):
        subprocess.run(["make", "-s", "-C", oracle_dir, "stage", "REF_TREE=" + tree, "REF_DIR=" + ref_src],
                       check=True)
    if os.path.isfile(os.path.join(ref_src, "SolutionSchemes.cpp")):
        subprocess.run(["make", "-s", "-C", oracle_dir, "ref", "REF_DIR=" + ref_src], check=True)
    import mara2_gb300  # noqa: F401


def smoke() -> None:
    import numpy as np

    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    from mara2_gb300 import workloads as W
    from mara2_gb300.solver import Solver

    s, P = W.sod(128)
    c = O.make_config(law="hydro", recon="plm", riemann="hlle", bc="outflow", rk_order=2,
                      shape=s.shape, gamma=s.gamma, plm_theta=s.plm_theta)
    port = O.Oracle("port")
    ref = P.copy()
    status, _, dts = port.run(c, ref, 5, s.cfl, s.t_final)
    assert status == 0
    with Solver(s, "fp64", device=0) as g:
        g.upload(P.copy())
        for dt in dts:
            g.advance(dt)
        out = g.download()
    assert np.array_equal(out[s.interior()].view(np.uint64), ref[s.interior()].view(np.uint64)), \
        "GPU plain path differs from the oracle"
    print("smoke: ok (5 steps of a 128-cell Sod tube match the oracle bit for bit)")


if __name__ == "__main__":
    build()
    if "--smoke" in sys.argv:
        smoke()
