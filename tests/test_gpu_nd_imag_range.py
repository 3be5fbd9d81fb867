"""Imaginary time in FP32 on wells far below the zero of energy: a step multiplies the state by exp(-E dt).
The unnormalised state of one step, times the half step of the potential that opens the next, has to fit
FP32: exp(1.5 |E| dt) times the gain of the transforms it passes before it is normalised.  That is the last
axis only; a transform along every axis first would cost a factor of the packet's points along the others.

Values of E dt between the two limits, ln(3.4e38) = 88.7 = 1.5 |E| dt + ln(sum of |psi| along what is
transformed), psi the normalised Gaussian of unit width and dr = 12 / n: 3-D 64^3, ln 1.7 along a row and
6.9 over the grid, so 58.0 and 54.5 and the test at 56.5; 2-D 256^2, ln 3.4 and 7.4, so 56.9 and 54.2 and the
test at 55.5.  Shifting a potential by a constant changes only the factor, so the
observables equal the oracle's FP64 ones at the FP32 bars (populations, norm and positions 1e-5, the energy
1e-5 of the shift)."""
import numpy as np
import pytest

from oracle import qd_ref
from zinq_b200 import quantum_dynamics as qd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n,S,edt", [(2, 256, 1, 55.5), (2, 256, 2, 55.5), (3, 64, 1, 56.5)])
def test_fp32_relaxation_far_below_the_zero_of_energy(d, n, S, edt):
    dt = 0.05
    r2 = "+".join(f"r{j + 1}^2" for j in range(d))
    mat = [[f"0.5*({r2})-{edt / dt - 0.1 * i}" if i == j else f"0.05*exp(-({r2})/2)" for j in range(S)] for i in range(S)]
    opt = {"grid": {"bounds": [[-6, 6]] * d, "npoint": n},
           "initial_conditions": {"position": [0.0] * d, "momentum": [0.0] * d, "gamma": [1.0] * d,
                                  "state": 0, "adiabatic": False},
           "potential": {"custom": {"ndim": d, "matrix": mat}}, "mass": [1.0] * d, "iterations": 8, "time_step": dt,
           "adiabatic": False, "imaginary": {"nstate": 1},
           "write": {"population": "P", "norm": "N", "position": "X", "total_energy": "E"}}
    g = qd.run(opt, precision="fp32").observables[0]
    r = qd_ref.run(opt)[0]
    for k, name, tol in (("population", "pop", 1e-5), ("norm", "norm", 1e-5), ("position", "pos", 1e-5),
                         ("total_energy", "etot", 1e-5 * edt / dt)):
        err = float(np.max(np.abs(g.history[k] - r.history[name])))
        assert err <= tol, (k, err)
    assert abs(g.norm - 1) <= 1e-5 and np.all(np.isfinite(g.wavefunction))
