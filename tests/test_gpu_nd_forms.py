"""The N-D axis passes on grids that the one-cluster kernel of small 2-D grids does not take (2-D from 256
points per axis up, and 3-D), so that every launch of a step is an axis pass.

* Each form of the row kernel (populations, autocorrelation, everything, general) records the series
  the wide form records beside all others: FP64 1e-13 absolute, FP32 1e-7 (the sums are in FP64 in
  both, over different partitions of the same points).
* The narrow forms against the oracle at the N-D parity bars (FP64 populations 1e-12, autocorrelation and
  other observables 1e-10; FP32 populations 1e-5, autocorrelation 1e-4).
* Repeats are the same bit for bit; a TMA wait that runs out in the middle of a run fails the run.
* A tuned shape is accepted exactly where the passes' limits say so."""
import copy

import numpy as np
import pytest

from oracle import qd_ref
from zinq_b200 import _abi
from zinq_b200 import quantum_dynamics as qd

from test_gpu_nd import coupled_harmonic_2d
from test_gpu_nd_lines import job
from test_gpu_parity import compare
from test_gpu_tma import run_without_tma

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("d,n", [(2, 256), (3, 32)])
@pytest.mark.parametrize("S", [1, 2, 3])
def test_every_row_form_records_the_same_series(d, n, S, precision):
    tol = 1e-13 if precision == "fp64" else 1e-7
    iters = 12
    full = qd.run(job(d, n, S, iters, "population norm acf position total_energy"), precision=precision).observables[0]
    for write in ("population", "norm population", "acf", "acf norm", "wavefunction population"):
        part = qd.run(job(d, n, S, iters, write), precision=precision).observables[0]
        for k in write.split():
            if k != "wavefunction":
                assert float(np.max(np.abs(part.history[k] - full.history[k]))) <= tol, (write, k)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("d,n,S", [(2, 256, 2), (2, 256, 3), (2, 512, 1), (3, 32, 2), (3, 32, 3)])
@pytest.mark.parametrize("write", ["population", "acf"])
def test_narrow_row_forms_against_the_oracle(d, n, S, write, precision):
    opt = job(d, n, S, 8, write)
    g = qd.run(opt, precision=precision).observables[0]
    r = qd_ref.run(opt)[0]
    name, tol = {"population": ("pop", {"fp64": 1e-12, "fp32": 1e-5}), "acf": ("acf", {"fp64": 1e-10, "fp32": 1e-4})}[write]
    ref = np.asarray(r.history[name])
    assert float(np.max(np.abs(g.history[write].reshape(ref.shape) - ref))) <= tol[precision]
    rel = float(np.linalg.norm(g.wavefunction - r.wavefunction) / np.linalg.norm(r.wavefunction))
    assert rel <= (1e-10 if precision == "fp64" else 1e-5), rel


def pop_256(iters=60):
    opt = coupled_harmonic_2d(npoint=256, iters=iters)
    opt["write"] = {"population": "P"}
    return opt


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_populations_match_the_per_block_kernels_and_repeat(precision):
    opt = pop_256()
    a = qd.run(opt, precision=precision).observables[0]
    b = run_without_tma(opt, precision).observables[0]
    tol = 1e-12 if precision == "fp64" else 1e-6
    assert float(np.max(np.abs(a.history["population"] - b.history["population"]))) <= tol
    for _ in range(3):
        c = qd.run(opt, precision=precision).observables[0]
        np.testing.assert_array_equal(a.wavefunction, c.wavefunction)
        np.testing.assert_array_equal(a.history["population"], c.history["population"])


def test_a_wait_that_runs_out_between_steps_fails_the_run():
    # a job advanced step by step; before the second range the next TMA-staged launch (a tile pass of that
    # range) is made to withhold its loads, so its waits run out of a 100 us budget with nothing in flight
    j = qd.Job(pop_256(iters=6))
    j.step(3)
    _abi.check(_abi.load().zqd_testing_tma_withhold_load(1, 100.0))
    with pytest.raises(_abi.ZqdError) as err:
        j.step(3)
        j.result()
    assert err.value.status == -8 and "TMA" in str(err.value)
    j.close()
    opt = copy.deepcopy(pop_256(iters=6))  # the armed launch is used up: the next run is whole
    compare(opt)


def tuned_job(tmp_path, n, S, rows, tile, precision):
    table = tmp_path / "t.txt"
    table.write_text(f"2 {n} {S} {1 if precision == 'fp32' else 0} 0 0 0 0 {rows} {tile}\n")
    qd.tune_load(table)
    try:
        return qd.Job(job(2, n, S, 1, "population"), precision=precision)
    finally:
        qd.tune_clear()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("rows,tile", [(1, 2), (2, 8), (4, 4), (8, 8), (16, 16), (32, 16), (3, 0), (0, 3), (0, 16), (16, 0)])
@pytest.mark.parametrize("n,S", [(8, 1), (16, 1), (16, 2), (32, 4), (64, 2), (256, 1), (512, 3), (2048, 2)])
def test_tuned_shapes_are_accepted_within_the_limits(tmp_path, n, S, rows, tile, precision):
    # whole warps of eight points a thread, at most 512 threads (rows of three and four states 256), blocks of at
    # least 1024 bytes, tile rows of whole 16 bytes; grids below 32 points take the per-block kernels with any of these
    c = 16 if precision == "fp64" else 8
    warps = lambda points, most: points // 8 % 32 == 0 and points // 8 <= most  # noqa: E731
    row_ok = rows == 0 or (n % rows == 0 and rows * n * c >= 1024 and warps(S * rows * n, 512 if S <= 2 else 256))
    tile_ok = tile == 0 or (n % tile == 0 and tile * c % 16 == 0 and warps(tile * n, 512))
    if not (row_ok and tile_ok):
        with pytest.raises(_abi.ZqdError) as err:
            tuned_job(tmp_path, n, S, rows, tile, precision)
        assert err.value.status == -7
        return
    j = tuned_job(tmp_path, n, S, rows, tile, precision)
    sh = j.nd_shape()
    j.close()

    def widened(k, lines):  # to whole warps of sixteen points a thread
        while lines * k * n // 16 % 32:
            k *= 2
        return k

    if rows:
        assert sh["tma_row_block"] == (widened(rows, S) if n >= 32 else 0)
    if tile:
        assert sh["tma_tile_lines"] == (widened(tile, 1) if n >= 32 else 0)
