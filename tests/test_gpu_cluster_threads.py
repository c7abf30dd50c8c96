"""One-cluster driver loops of different sizes in several threads: each
handle has its own stream, but the dynamic shared memory limit belongs to the
kernel, so one thread's small grid must not lower it under another's launch."""
import threading

import numpy as np
import pytest

from mara2_gb300 import workloads as W
from mara2_gb300.scheme import Scheme
from mara2_gb300.solver import Solver


def _state(n):
    s = Scheme(shape=(n, 1, 1), recon="plm", riemann="hlle", bc="outflow", rk_order=2, cfl=0.3)
    rng = np.random.default_rng(n)
    P = W.empty_state(s)
    Q = P[s.interior()]
    Q[..., 0] = rng.uniform(0.9, 1.1, n)[:, None, None]
    Q[..., 1] = rng.uniform(-0.1, 0.1, n)[:, None, None]
    Q[..., 4] = rng.uniform(0.9, 1.1, n)[:, None, None]
    return s, W.apply_bc_numpy(s, P)


@pytest.mark.gpu
@pytest.mark.parametrize("precision,sizes", [("fp64", (4096, 128, 4096, 64)), ("mixed", (8192, 256, 8192, 128))])
def test_cluster_loops_of_different_sizes_in_threads(gpu_lib, precision, sizes):
    calls = 1500

    def steps(n):
        s, P = _state(n)
        with Solver(s, precision) as g:
            g.upload(P)
            for _ in range(calls):
                g.run(1)
            return g.download()

    expected = {n: steps(n) for n in set(sizes)}
    results = {}

    def work(k, n):
        try:
            results[k] = steps(n)
        except Exception as e:
            results[k] = e

    threads = [threading.Thread(target=work, args=(k, n)) for k, n in enumerate(sizes)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, n in enumerate(sizes):
        assert not isinstance(results[k], Exception), (n, results[k])
        assert np.array_equal(results[k].view(np.uint64), expected[n].view(np.uint64))
