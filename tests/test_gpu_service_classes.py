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


@pytest.mark.parametrize("piece", [1, 4, 5])
def test_rows_are_published_when_the_piece_asked_for_is_complete(piece):
    # a ring of eight rows would publish counts that are multiples of eight only; a client that asks for smaller
    # pieces gets them at other counts too (some 300 polls in 20 ms of steps; one in eight, four or eight of the
    # counts are multiples of eight)
    srv = qd.Server(workers=1, stream_steps=piece)
    opt = small_line(1024, 1, 15.0, iters=3000)
    opt["write"] = {"population": "P"}  # one value a row: a ring of eight rows
    t = srv.submit(opt, "fp32")
    firsts, rows, t0, done = [], [], time.time(), False
    while not done:
        for e in srv.poll():
            done = done or e["kind"] == "done"
            if e["kind"] == "rows":
                firsts.append(e["first_row"])
                rows.append(e["rows"])
        assert time.time() - t0 < 60
        time.sleep(0.0005)
    r, _ = srv.wait(t)
    srv.close()
    assert any(f % 8 for f in firsts), firsts
    got = np.concatenate(rows)
    assert got.shape[0] == 3001
    np.testing.assert_array_equal(got[:, 3:4], r.observables[0].history["population"])
