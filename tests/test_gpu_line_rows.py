"""Rows of the resident 1-D kernel: momentum-space observables that leave psi in place, on every cluster size,
against the oracle at the plain form's bars (FP64 populations 1e-12, wavefunction relative L2 1e-10, other
observables 1e-10) and bit for bit over repeats."""
import numpy as np
import pytest

from oracle import qd_ref
from zinq_b200 import quantum_dynamics as qd

from test_gpu_parity import compare, tully

pytestmark = pytest.mark.gpu


# points per CTA of 32, 64 and 512: an odd number of radix-4 passes, so that the observation's transform
# ends in the buffer the next step's first pass writes
@pytest.mark.parametrize("cluster,npoint", [(2, 128), (2, 1024), (4, 256), (4, 2048), (8, 256), (8, 512)])
def test_momentum_rows_on_clusters(cluster, npoint, monkeypatch):
    monkeypatch.setenv("ZQD_LINE_CLUSTER", str(cluster))
    opt = tully("tully_1", False, npoint=npoint, iters=200)
    first, _, _ = compare(opt)
    for _ in range(4):
        again = qd.run(opt).observables[0]
        for k, v in first.observables[0].history.items():
            np.testing.assert_array_equal(again.history[k], v)
        np.testing.assert_array_equal(again.wavefunction, first.observables[0].wavefunction)


# rows that wait in shared memory and rows reduced at once in one run: steps that record more than the write
# options ask for (every 7th of 46, which no ring length divides) flush what waits before them, and the
# absorbed populations carry on across both
@pytest.mark.parametrize("cluster", [1, 16])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_logged_rows_between_waiting_rows(cluster, precision, monkeypatch, capfd):
    monkeypatch.setenv("ZQD_LINE_CLUSTER", str(cluster))
    opt = tully("tully_1", False, npoint=512, iters=46)
    opt["write"] = {"population": "P", "norm": "N"}
    opt["absorbing_potential"] = {"bounds": [[-12, 16]], "exponent": 0.3, "track_population": True}
    opt["log_interval"] = 7
    plain = qd.run(opt, precision=precision).observables[0]
    logged = qd.run(opt, precision=precision, log=True).observables[0]
    ref = qd_ref.run(opt)[0]
    tol = 1e-12 if precision == "fp64" else 1e-5
    for g in (plain, logged):
        assert g.history["population"].shape == ref.history["pop"].shape
        assert float(np.max(np.abs(g.history["population"] - ref.history["pop"]))) <= tol
        assert float(np.max(np.abs(g.history["norm"] - ref.history["norm"]))) <= max(tol, 1e-10)
    # the same run cut into pieces that end inside a ring
    cut = qd.Job(opt, precision=precision)
    while not cut.progress()[2]:
        cut.step(5)
    c = cut.result().observables[0]
    cut.close()
    np.testing.assert_array_equal(c.history["population"], plain.history["population"])
    np.testing.assert_array_equal(c.wavefunction, plain.wavefunction)


# two CTAs' registers fit an SM at 512 points x 2 states (two CTAs a job): 148 jobs are one wave of the 148 SMs, as
# 74 are.  One CTA per SM (shared memory taken for waiting rows) makes them two waves and the ratio 2; two side
# by side share the SM's pipes, which cost a wave 1.1 to 1.35 times one job's time, so the bar is 1.6.
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_waiting_rows_leave_the_ctas_of_an_sm_their_places(precision):
    opt = tully("tully_1", False, npoint=512, iters=300)
    opt["write"] = {"population": "P"}
    ms = {}
    for n in (74, 148):
        b = qd.Batch([opt] * n, precision=precision)
        ms[n] = min(b.run() for _ in range(5))
        b.close()
    assert ms[148] <= 1.6 * ms[74], ms
