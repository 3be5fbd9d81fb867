"""Rows of the resident 1-D kernel: momentum-space observables that leave psi in place, on every cluster size,
against the oracle at the plain form's bars (FP64 populations 1e-12, wavefunction relative L2 1e-10, other
observables 1e-10) and bit for bit over repeats."""
import numpy as np
import pytest

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
