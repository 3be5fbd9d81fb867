"""Small 2-D grids in real time (32 to 128 points per axis) run whole ranges of steps in one launch of one
cluster (nd_small_kernel).  Every grid length and state count of it, both precisions, against the
oracle at the parity bars of the other N-D tests (FP64 wavefunction relative L2 1e-10, populations
1e-12, other observables 1e-10; FP32 populations 1e-5), and runs cut into pieces against whole ones,
bit for bit (the observables row of a piece's last step is written by the piece itself)."""
import numpy as np
import pytest

from oracle import qd_ref
from zinq_b200 import quantum_dynamics as qd

from test_gpu_nd_lines import job

pytestmark = pytest.mark.gpu

SERIES = {"population": "pop", "position": "pos", "norm": "norm", "potential_energy": "epot", "acf": "acf"}


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("S", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [32, 64, 128])
def test_small_grids_against_the_oracle(n, S, precision):
    more = {} if S != 2 else {"adiabatic": True,
                              "absorbing_potential": {"bounds": [[-5, 5], [-5, 5]], "exponent": 0.05}}
    opt = job(2, n, S, 25, "population position norm potential_energy acf", **more)
    g = qd.run(opt, precision=precision).observables[0]
    r = qd_ref.run(opt)[0]
    tol = {"population": 1e-12} if precision == "fp64" else {"population": 1e-5}
    for k, name in SERIES.items():
        ref = np.asarray(r.history[name])
        err = float(np.max(np.abs(g.history[k].reshape(ref.shape) - ref)))
        assert err <= tol.get(k, 1e-10 if precision == "fp64" else 1e-4), (k, err)
    rel = float(np.linalg.norm(g.wavefunction - r.wavefunction) / np.linalg.norm(r.wavefunction))
    assert rel <= (1e-10 if precision == "fp64" else 1e-5), rel


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,S", [(32, 1), (64, 3), (128, 2)])
def test_pieces_give_the_bits_of_a_whole_run(n, S, precision):
    opt = job(2, n, S, 37, "population norm acf")
    whole = qd.Job(opt, precision=precision)
    whole.run()
    a = whole.result().observables[0]
    for piece in (1, 2, 16, 38):
        cut = qd.Job(opt, precision=precision)
        while not cut.progress()[2]:
            cut.step(piece)
        b = cut.result().observables[0]
        for k in a.history:
            np.testing.assert_array_equal(a.history[k], b.history[k])
        np.testing.assert_array_equal(a.wavefunction, b.wavefunction)
        assert a.ekin == b.ekin and a.norm == b.norm
        cut.close()
    whole.close()
