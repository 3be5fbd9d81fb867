"""Where an N-D step's sums are reduced: by an extra CTA of the next kinetic tile launch, by a launch of their own
where the next launch needs the outcome (stop_norm, tracked absorption) or a range of steps ends, by the
last CTA of a per-block launch on grids of at least 2^18 points.  Every such sequence against the oracle at the N-D parity
bars (FP64: series 1e-10, populations 1e-12, wavefunction relative L2 1e-10) and, cut into pieces that end a range
after one and after four steps, bit for bit the whole run."""
import numpy as np
import pytest

from zinq_b200 import quantum_dynamics as qd

from test_gpu_nd_lines import job
from test_gpu_parity import compare

pytestmark = pytest.mark.gpu


def sequences(d):
    cap = {"bounds": [[-1.5, 1.5]] * d, "exponent": 0.3, "track_population": True}
    return {"stop": {"absorbing_potential": dict(cap, stop_norm=0.97)}, "track": {"absorbing_potential": cap},
            "stop_untracked": {"absorbing_potential": dict(cap, track_population=False, stop_norm=0.97)},
            "imag2": {"imaginary": {"nstate": 2}}, "imag1": {"imaginary": {"nstate": 1}}, "td": {}, "plain": {}}


def options(d, n, S, iters, what, write):
    opt = job(d, n, S, iters, write, **sequences(d)[what])
    opt["time_step"] = 0.1
    opt["initial_conditions"]["momentum"] = [3.0] + [0.0] * (d - 1)
    if what == "td":
        opt["potential"]["custom"]["time_dependent"] = True
        opt["potential"]["custom"]["matrix"][0][0] += "+0.05*r1*sin(0.3*t)"
    return opt


@pytest.mark.parametrize("tma", ["1", "0"])
@pytest.mark.parametrize("what", ["stop", "stop_untracked", "track", "td", "imag1", "imag2", "plain"])
@pytest.mark.parametrize("d,n,S,write", [(2, 256, 2, "population norm"), (2, 512, 1, "population total_energy"),
                                         (3, 32, 2, "population"), (2, 16, 2, "norm total_energy")])
def test_sums_of_every_sequence(d, n, S, write, what, tma, monkeypatch):
    monkeypatch.setenv("ZQD_ND_TMA", tma)
    iters = 14
    opt = options(d, n, S, iters, what, write)
    whole, ref, _ = compare(opt)
    rows = len(ref[0].history["norm" if "norm" in write else "pop"])
    if what.startswith("stop") and n >= 32:
        assert 1 < rows <= iters  # the solve did stop
    for piece in (1, 4):
        cut = qd.Job(opt)
        while not cut.progress()[2]:
            cut.step(piece)
        res = cut.result()
        for a, b in zip(whole.observables, res.observables):
            for k in a.history:
                np.testing.assert_array_equal(a.history[k], b.history[k])
            np.testing.assert_array_equal(a.wavefunction, b.wavefunction)
            assert (a.norm, a.ekin, a.epot) == (b.norm, b.ekin, b.epot)
        cut.close()
