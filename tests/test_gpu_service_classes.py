"""What the line-service kernel's jobs share: a kernel class, and the rows they publish."""
import time

import numpy as np
import pytest

from zinq_b200 import quantum_dynamics as qd

from test_gpu_service import small_line

pytestmark = pytest.mark.gpu


def served_ms(opts, precision):
    srv = qd.Server(stream_rows=False)
    best = 1e9
    for _ in range(4):
        t0 = time.perf_counter()
        tickets = [srv.submit(o, precision) for o in opts]
        for t in tickets:
            srv.wait(t)
        best = min(best, 1e3 * (time.perf_counter() - t0))
    assert srv.stats()["service_jobs"] == 4 * len(opts)
    srv.close()
    return best


def test_lines_of_two_lengths_are_served_side_by_side():
    # 1024 and 2048 points x 3 states, FP32 with energies: with what a job takes after its tables both come to
    # 208 KB.  In one class the shorter lines' jobs wait for the longer ones' (1.6 times the longer ones
    # alone); in two they run beside them.
    lines = {}
    for n in (1024, 2048):
        lines[n] = small_line(n, 3, 15.0, iters=300)
        lines[n]["write"] = {"population": "P", "norm": "N", "total_energy": "E"}
    alone = served_ms([lines[2048]] * 8, "fp32")
    both = served_ms([lines[2048], lines[1024]] * 8, "fp32")
    assert both <= 1.3 * alone, (both, alone)
