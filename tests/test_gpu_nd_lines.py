"""The TMA-staged axis passes over every line length they are built for (32 to 4096 points: one or two
exchange boundaries, first radix 8 or 16, lines within one warp up to 512 points and across warps
above), one to four states, both precisions, with the shapes the rules choose and the edges of what
they accept, against the oracle.  Bars: FP64 wavefunction relative L2 1e-10, populations 1e-12 and
energies 1e-10 of the oracle's (the parity bars of the other N-D tests); FP32 populations 1e-5.
A few steps: the transforms run twice per axis in each."""
import numpy as np
import pytest

from oracle import qd_ref
from zinq_b200 import _abi
from zinq_b200 import quantum_dynamics as qd

pytestmark = pytest.mark.gpu


def job(d, n, S, iters, write, **more):
    r2 = "+".join(f"r{j + 1}^2" for j in range(d))
    mat = [[f"0.5*({r2})+{0.1 * i}+{0.2 * (i + 1)}*r1" if i == j else f"0.05*exp(-({r2})/2)" for j in range(S)]
           for i in range(S)]
    opt = {"grid": {"bounds": [[-9, 9]] * d, "npoint": n},
           "initial_conditions": {"position": [-1.0] + [0.3] * (d - 1), "momentum": [0.7] + [0.0] * (d - 1),
                                  "gamma": [1.0] * d, "state": 0, "adiabatic": False},
           "potential": {"custom": {"ndim": d, "matrix": mat}}, "mass": [1.0] * d, "iterations": iters,
           "time_step": 0.02, "adiabatic": False, "write": {w: w for w in write.split()}}
    opt.update(more)
    return opt


def check(opt, precision):
    g = qd.run(opt, precision=precision).observables[0]
    r = qd_ref.run(opt)[0]
    pop_tol = 1e-12 if precision == "fp64" else 1e-5
    assert float(np.max(np.abs(g.pop - np.asarray(r.pop)))) <= pop_tol
    if "population" in g.history:
        assert float(np.max(np.abs(g.history["population"] - r.history["pop"]))) <= pop_tol
    rel = float(np.linalg.norm(g.wavefunction - r.wavefunction) / np.linalg.norm(r.wavefunction))
    assert rel <= (1e-10 if precision == "fp64" else 1e-5), rel
    if precision == "fp64":
        assert abs(g.ekin - r.ekin) <= 1e-10 * max(1.0, abs(r.ekin)) and abs(g.epot - r.epot) <= 1e-10 * max(1.0, abs(r.epot))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,S", [(32, 1), (32, 4), (64, 3), (128, 1), (128, 4), (256, 2), (512, 1), (512, 4), (1024, 1),
                                 (1024, 3), (1024, 4), (2048, 1), (2048, 2), (4096, 1)])
def test_2d_lines(n, S, precision):
    if n == 4096 and precision == "fp64":
        pytest.skip("FP64 lines of 4096 points are refused (shared memory)")
    iters = 6 if n <= 256 else 3 if n <= 1024 else 1
    check(job(2, n, S, iters, "population total_energy" if S > 1 else "population"), precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,S", [(32, 2), (64, 1), (64, 3), (128, 2), (256, 1)])
def test_3d_lines(n, S, precision):
    check(job(3, n, S, 2 if n <= 64 else 1, "population acf"), precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("rows,tile", [(1, 2), (4, 4), (8, 8), (32, 16)])
@pytest.mark.parametrize("n,S", [(64, 2), (256, 1), (512, 3)])
def test_shapes_at_the_edges_of_the_rules(tmp_path, n, S, rows, tile, precision):
    # a tuning table forces the shape (rounded up to whole warps of sixteen points a thread); one outside the
    # kernel's limits is refused when the job is created
    table = tmp_path / "t.txt"
    table.write_text(f"2 {n} {S} {1 if precision == 'fp32' else 0} 0 0 0 0 {rows} {tile}\n")
    qd.tune_load(table)
    try:
        try:
            j = qd.Job(job(2, n, S, 1, "population"), precision=precision)
        except _abi.ZqdError as e:
            assert e.status == -7
            return
        sh = j.nd_shape()
        j.close()
        whole = lambda k, lines: k if lines * k * n // 16 % 32 == 0 else whole(2 * k, lines)  # noqa: E731
        assert sh["tma_row_block"] == whole(rows, S) and sh["tma_tile_lines"] == whole(tile, 1)
        assert sh["tma_row_threads"] % 32 == 0 and sh["tma_tile_threads"] % 32 == 0
        check(job(2, n, S, 4, "population norm"), precision)
    finally:
        qd.tune_clear()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_row_forms_record_the_same_series(precision):
    # each form of the row kernel (populations, autocorrelation, everything, with absorption): the
    # series a narrow form records equals the one recorded beside all others
    tol = 1e-13 if precision == "fp64" else 1e-7
    for S in (1, 2):
        full = qd.run(job(2, 64, S, 20, "population norm acf position total_energy"), precision=precision).observables[0]
        for write in ("population", "norm population", "acf"):
            part = qd.run(job(2, 64, S, 20, write), precision=precision).observables[0]
            for k in write.split():
                assert float(np.max(np.abs(part.history[k] - full.history[k]))) <= tol, (S, k)
        cap = {"bounds": [[-5, 5], [-5, 5]], "exponent": 0.3, "track_population": True}
        check(job(2, 64, S, 20, "population norm", absorbing_potential=cap), precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("d,n,S", [(3, 128, 2), (2, 1024, 1)])
def test_many_items_per_cta_repeat_bit_for_bit(d, n, S, precision):
    # more tiles and row blocks than resident CTAs: a CTA's next load is issued while it still works on
    # the last one, into a stage every thread has finished reading
    j = qd.Job(job(d, n, S, 3, "population norm"), precision=precision)
    first = None
    for _ in range(10):
        j.run()
        o = j.result().observables[0]
        if first is None:
            first = o
        np.testing.assert_array_equal(o.wavefunction, first.wavefunction)
        np.testing.assert_array_equal(o.history["population"], first.history["population"])
    j.close()
