"""Performance cases of the wavepacket propagator: the work users give it, through its public entry points.

A case is a dict of plain values:
  entry      "run"    zinq_b200.quantum_dynamics.run on an options dict: tables, propagation and download in one call
             "job"    a Job whose tables the program keeps: Job.run and then Job.result (series and wavefunction)
             "rows"   a Job: Job.run and then Job.observables (the recorded rows, no wavefunction download)
             "batch"  a Batch of `jobs` jobs whose tables the program keeps: Batch.run and every result
             "serve"  a Server that the program keeps: submit a mix of `jobs` jobs, wait for all of them
             "fft"    the FFT entry point (zqd_fft_execute) with a kept plan, on a device tensor
  ndim, npoint, nstate, precision, steps   the grid, the electronic states, the form, the propagation steps
  potential  "harmonic" (coupled harmonic surfaces), "crossing" (tanh crossing), "anharmonic" (one 3-D well)
  write      the recorded time series, space-separated
  adiabatic, imaginary, absorb, spectrum   options of the run (0 / False: off)
All inputs come from the seed.  The FP32 form's outputs are returned as 32-bit floats, the type its
wavefunction has; everything else stays as the entry point returns it.
"""
import ctypes
import math
import random

import numpy as np
import torch

from zinq_b200 import _abi
from zinq_b200 import quantum_dynamics as qd


def _case(name, entry, ndim, npoint, nstate, precision, steps, potential, write, **more):
    c = {"name": name, "entry": entry, "ndim": ndim, "npoint": npoint, "nstate": nstate, "precision": precision,
         "steps": steps, "potential": potential, "write": write, "adiabatic": False, "imaginary": 0, "absorb": False,
         "spectrum": 0, "jobs": 1}
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: one short 1-D line, everything from options to results; latency and host overhead
        _case("line_small", "run", 1, 256, 1, "fp32", 100, "harmonic", "population position"),
        # the reference's basic use: a 1-D oscillator with energies recorded at every step (1024 points, FP64)
        _case("line_oscillator", "run", 1, 1024, 1, "fp64", 1000, "harmonic", "norm position total_energy"),
        # the headline workload: five momenta of the two-state avoided crossing on 8192 points, one batched launch
        _case("line_batch", "batch", 1, 8192, 2, "fp32", 2000, "crossing", "population", adiabatic=True, jobs=5),
        # three states with an absorbing boundary whose absorbed populations are tracked, ACF recorded
        _case("line_absorbing", "job", 1, 4096, 3, "fp64", 701, "harmonic", "population norm acf", absorb=True),
        # a small 2-D grid: many short steps, bound by what a step costs however little it does
        _case("grid2_small", "job", 2, 128, 2, "fp64", 500, "crossing", "population"),
        # three coupled 2-D surfaces with populations, norm and total energy at every step (512^2, FP64)
        _case("grid2_energy", "rows", 2, 512, 3, "fp64", 150, "harmonic", "population total_energy norm"),
        # what most of a serving stream is: 2-D FP32 jobs that record populations
        _case("grid2_fp32", "rows", 2, 512, 3, "fp32", 300, "harmonic", "population"),
        # imaginary-time relaxation of a 3-D well, the whole call with the relaxed state
        _case("grid3_relax", "run", 3, 128, 1, "fp64", 250, "anharmonic", "", imaginary=1),
        # 3-D real time, autocorrelation for a spectrum
        _case("grid3_acf", "rows", 3, 128, 1, "fp32", 300, "anharmonic", "acf", spectrum=1),
        # a grid whose wavefunction and tables do not fit in the last-level cache
        _case("grid2_wide", "rows", 2, 2048, 2, "fp64", 60, "harmonic", "population"),
        # a burst of uneven jobs through the server: 1-D and 2-D, one to three states, FP32
        _case("serve_burst", "serve", 2, 512, 3, "fp32", 300, "harmonic", "population", jobs=24),
        # the FFT entry point on a 3-D grid
        _case("fft_grid3", "fft", 3, 128, 1, "fp64", 1, "", "", direction=-1),
    ]


def draw(rng):
    kind = rng.choice(["line", "line", "batch", "grid2", "grid2", "grid3", "serve", "fft"])
    precision = rng.choice(["fp32", "fp64"])
    pow2 = lambda lo, hi: 1 << rng.randint(lo, hi)  # noqa: E731
    steps = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    name = ""
    if kind == "line":
        n, S = pow2(8, 14), rng.randint(1, 3)
        absorb = rng.random() < 0.25
        c = _case(name, rng.choice(["run", "job"]), 1, n, S, precision, steps(100, 1500),
                  rng.choice(["harmonic", "crossing"]),
                  rng.choice(["population", "population norm", "norm position total_energy", "position momentum"]),
                  adiabatic=rng.random() < 0.5, absorb=absorb)
    elif kind == "batch":
        n, S = pow2(9, 13), rng.randint(1, 3)
        c = _case(name, "batch", 1, n, S, precision, steps(100, 1500), rng.choice(["harmonic", "crossing"]),
                  "population", adiabatic=rng.random() < 0.5, jobs=rng.randint(2, 9))
    elif kind == "grid2":
        n, S = pow2(6, 11), rng.randint(1, 3)
        S = 1 + (S - 1) % 2 if n == 2048 else S
        most = max(20, min(600, 400 * 512 * 512 // (n * n)))
        c = _case(name, rng.choice(["rows", "job"]) if n <= 512 else "rows", 2, n, S, precision, steps(20, most),
                  rng.choice(["harmonic", "crossing"]),
                  rng.choice(["population", "population", "population norm position", "total_energy", "acf"]),
                  adiabatic=rng.random() < 0.3, absorb=rng.random() < 0.15)
    elif kind == "grid3":
        n = pow2(5, 7)
        S = rng.randint(1, 2)
        imag = S == 1 and rng.random() < 0.5
        c = _case(name, "rows", 3, n, S, precision, steps(20, 200), "anharmonic" if S == 1 else "harmonic",
                  "norm" if imag else rng.choice(["acf", "population", "norm total_energy"]), imaginary=1 if imag else 0)
    elif kind == "serve":
        c = _case(name, "serve", 2, pow2(7, 9), rng.randint(1, 3), precision, steps(50, 300), "harmonic", "population",
                  jobs=rng.randint(6, 24))
    else:
        d = rng.randint(1, 3)
        n = pow2(8, 13) if d == 1 else pow2(6, 11) if d == 2 else pow2(4, 8)
        c = _case(name, "fft", d, n, 1, precision, 1, "", "", direction=rng.choice([-1, 1]))
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------- inputs
def _matrix(potential, d, S, rng):
    """Diabatic potential expressions with constants from rng."""
    r2 = "+".join(f"r{j + 1}^2" for j in range(d))
    if potential == "anharmonic":
        a, b = rng.uniform(0.05, 0.15), rng.uniform(0.03, 0.07)
        return [[f"0.5*({r2})+{a:.17g}*(r1^2*r2-r2^3/3)+{b:.17g}*r3^4"]]
    mat = []
    if potential == "crossing":
        A, B, C = rng.uniform(0.008, 0.012), rng.uniform(1.4, 1.8), rng.uniform(0.004, 0.006)
        for i in range(S):
            mat.append([f"{A if i % 2 == 0 else -A:.17g}*tanh({B:.17g}*r1)+{0.05 * (i // 2):.17g}" if i == j else
                        f"{C:.17g}*exp(-({r2}))" for j in range(S)])
        return mat
    lin, c, k = rng.uniform(-1, 1, (S, d)), rng.uniform(0, 0.2, S), rng.uniform(0.03, 0.07)
    for i in range(S):
        tilt = "".join(f"+{lin[i, j]:.17g}*r{j + 1}" for j in range(d))
        mat.append([f"0.5*({r2}){tilt}+{c[i]:.17g}" if i == j else f"{k:.17g}*exp(-({r2})/2)" for j in range(S)])
    return mat


def _options(case, rng):
    """A quantum_dynamics options dict of the case, its physical parameters from rng."""
    d, S = case["ndim"], case["nstate"]
    mat = _matrix(case["potential"], d, S, rng)
    if case["potential"] == "crossing":  # a packet of mass 2000 that runs into the crossing at 0
        half, mass, dt = 24.0, 2000.0, 1.0 if d == 1 else 2.0
        p0 = float(rng.uniform(0.25, 0.6)) * min(50.0, math.pi * case["npoint"] / (2 * half))
        x0, mom, gamma = -float(rng.uniform(6, 10)), p0, max(0.25, p0 * p0 / 400.0)
    else:
        half, mass = {1: 12.0, 2: 12.0, 3: 8.0}[d], 1.0
        dt = 0.02 if d == 3 else 0.05
        x0, mom, gamma = -float(rng.uniform(1, 2)), float(rng.uniform(0, 1)), 1.0
        if d == 3:
            x0, mom = float(rng.uniform(0.5, 1)), 0.0
    # a packet on one adiabatic surface: where that surface's sign is well defined on the whole grid
    adia_start = bool(case["adiabatic"]) and S == 2 and case["potential"] == "crossing"
    opt = {"grid": {"bounds": [[-half, half]] * d, "npoint": case["npoint"]},
           "initial_conditions": {"position": [x0] + [0.25] * (d - 1), "momentum": [mom] + [0.0] * (d - 1),
                                  "gamma": [gamma] * d, "state": 0, "adiabatic": adia_start},
           "potential": {"custom": {"ndim": d, "matrix": mat}}, "mass": [mass] * d, "iterations": case["steps"],
           "time_step": dt, "adiabatic": bool(case["adiabatic"]), "write": {w: w for w in case["write"].split()}}
    if case["imaginary"]:
        opt["imaginary"] = {"nstate": case["imaginary"]}
    if case["absorb"]:
        opt["absorbing_potential"] = {"bounds": [[-0.6 * half, 0.6 * half]] * d, "exponent": 0.01,
                                      "track_population": True}
    if case["spectrum"]:
        opt["spectrum"] = {"padding": 0}
    return opt


def _mix(case, rng):
    """The server's jobs: sizes, states and lengths fixed by the case, parameters from rng."""
    pick = random.Random(case["jobs"] * 7919 + case["npoint"])
    opts = []
    for k in range(case["jobs"]):
        d = 1 + k % 2
        n = 1 << (pick.randint(8, 13) if d == 1 else pick.randint(6, case["npoint"].bit_length() - 1))
        sub = dict(case, ndim=d, npoint=n, nstate=1 + pick.randrange(case["nstate"]),
                   steps=pick.randint(case["steps"] // 3, case["steps"]),
                   potential=pick.choice(["harmonic", "crossing"]))
        opts.append(_options(sub, rng))
    return opts


def _all_options(case, seed):
    rng = np.random.default_rng(seed)
    if case["entry"] == "serve":
        return _mix(case, rng)
    return [_options(case, rng) for _ in range(case["jobs"])]


def _fft_input(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    kind = torch.float32 if case["precision"] == "fp32" else torch.float64
    x = torch.randn([case["npoint"]] * case["ndim"] + [2], generator=g, device="cuda", dtype=kind)
    return torch.view_as_complex(x)


def prepare(case, seed):
    entry, prec = case["entry"], case["precision"]
    state = {"case": case}
    if entry == "fft":
        lib = _abi.load()
        state["plan"] = ctypes.c_void_p()
        shape = (ctypes.c_int * case["ndim"])(*[case["npoint"]] * case["ndim"])
        _abi.check(lib.zqd_fft_plan_create(case["ndim"], shape, case["direction"], _abi.PRECISION[prec],
                                           ctypes.byref(state["plan"])))
        state["x"] = _fft_input(case, seed)
        state["y"] = torch.empty_like(state["x"])
        return state
    state["opts"] = _all_options(case, seed)
    if entry in ("job", "rows"):
        state["job"] = qd.Job(state["opts"][0], precision=prec)
    elif entry == "batch":
        state["batch"] = qd.Batch(state["opts"], precision=prec)
    elif entry == "serve":
        state["server"] = qd.Server(stream_rows=False)
    return state


# ------------------------------------------------------------------------------------------- one pass
def _typed(x, precision):
    """Outputs of the FP32 form in 32 bits (the type of its wavefunction)."""
    if precision != "fp32":
        return x
    return x.astype(np.complex64 if np.iscomplexobj(x) else np.float32)


def _outputs(result, precision, wavefunction):
    ob = result.observables[0]
    out = {k: _typed(v, precision) for k, v in ob.history.items()}
    out["final"] = _typed(np.concatenate([ob.pos, ob.mom, ob.pop, [ob.epot, ob.ekin, ob.norm]]), precision)
    if wavefunction:
        out["wavefunction"] = _typed(ob.wavefunction, precision)
    return out


def run(state):
    case = state["case"]
    entry, prec = case["entry"], case["precision"]
    if entry == "fft":
        state["y"].copy_(state["x"])
        _abi.check(_abi.load().zqd_fft_execute(state["plan"], ctypes.c_void_p(state["y"].data_ptr()),
                                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return state["y"]
    if entry == "run":
        return _outputs(qd.run(state["opts"][0], precision=prec), prec, True)
    if entry == "job":
        state["job"].run()
        return _outputs(state["job"].result(), prec, True)
    if entry == "rows":
        state["job"].run()
        return [_typed(rows, prec) for _, _, rows in state["job"].observables()]
    if entry == "batch":
        state["batch"].run()
        return [_outputs(state["batch"].result(i, want_wavefunction=True), prec, True) for i in range(case["jobs"])]
    tickets = [state["server"].submit(o, precision=prec) for o in state["opts"]]
    results = [state["server"].wait(t, want_wavefunction=True)[0] for t in tickets]
    # a job's populations and wavefunction
    return [[_typed(r.observables[0].history["population"], prec), _typed(r.observables[0].wavefunction, prec)]
            for r in results]


# ------------------------------------------------------------------------------------------- work
def _job_work(d, n, S, steps, precision, write):
    """What a propagation cannot do without.  Bytes: its tables and states once; on a grid whose state and
    propagator table exceed the last-level cache, per step two sweeps over the state (a transform along
    more than one axis needs two) and one over the table.  Operations: per step and state a forward and an
    inverse FFT, the two propagator products, the kinetic phase and the recorded sums."""
    N, c = float(n) ** d, 8 if precision == "fp32" else 16
    state, table = S * N * c, S * (S + 1) / 2 * N * c
    ffts = 3 if "energy" in write or "momentum" in write else 2
    flops = steps * N * (S * ffts * 5 * d * math.log2(n) + 2 * 8 * S * S + 8 * S + 6 * S)
    moved = 2 * state + table
    if d > 1 and state + table > 126e6:
        moved = steps * (4 * state + table)
    return moved, flops


def work(case):
    d, n, S, steps, prec = (case[k] for k in ("ndim", "npoint", "nstate", "steps", "precision"))
    if case["entry"] == "fft":
        N = float(n) ** d
        return {"bytes": 2 * N * (8 if prec == "fp32" else 16), "flops": 5 * N * d * math.log2(n)}
    if case["entry"] == "serve":
        jobs = [(len(o["mass"]), o["grid"]["npoint"], len(o["potential"]["custom"]["matrix"]), o["iterations"])
                for o in _mix(case, np.random.default_rng(0))]
    else:
        jobs = [(d, n, S, steps)] * case["jobs"]
    got = [_job_work(*j, prec, case["write"]) for j in jobs]
    return {"bytes": sum(g[0] for g in got), "flops": sum(g[1] for g in got)}


# ------------------------------------------------------------------------------------------- 64-bit results
def _values(expr, r):
    names = {f"r{j + 1}": v for j, v in enumerate(r)}
    names.update(tanh=torch.tanh, exp=torch.exp)
    v = eval(expr.replace("^", "**"), {"__builtins__": {}}, names)  # the expressions above only
    return v.expand(r[0].shape) if v.dim() else v.expand_as(r[0])


class _Grid:
    def __init__(self, opt):
        b, n = opt["grid"]["bounds"], opt["grid"]["npoint"]
        self.d, self.n, self.N = len(b), n, n ** len(b)
        dev = {"device": "cuda", "dtype": torch.float64}
        axis = [lo + torch.arange(n, **dev) * (hi - lo) / n for lo, hi in b]
        wave = [2 * math.pi / (hi - lo) * torch.fft.fftfreq(n, d=1.0 / n, **dev) for lo, hi in b]
        self.r = torch.meshgrid(*axis, indexing="ij")
        self.k = torch.meshgrid(*wave, indexing="ij")
        self.dr = math.prod((hi - lo) / n for lo, hi in b)
        self.dk = self.dr / self.N


def _eigen(V, d):
    """Eigenvalues and eigenvectors per point; along a 1-D grid each vector keeps the sign of its neighbour."""
    W, U = np.linalg.eigh(np.moveaxis(V.cpu().numpy().reshape(*V.shape[:2], -1), -1, 0), UPLO="U")
    if d == 1 and U.shape[1] > 1:
        ov = np.einsum("xkj,xkj->xj", U[1:], U[:-1])
        U[1:] *= np.cumprod(np.where(ov < 0, -1.0, 1.0), axis=0)[:, None, :]
    W, U = torch.from_numpy(W).cuda(), torch.from_numpy(U).cuda()
    S = V.shape[0]
    return W.T.reshape(S, *V.shape[2:]), U.permute(1, 2, 0).reshape(S, S, *V.shape[2:])


def _propagate(opt):
    """(rows, psi, final row) of the split-operator propagation of opt, in 64 bits."""
    g = _Grid(opt)
    mat = opt["potential"]["custom"]["matrix"]
    S, d, dt = len(mat), g.d, opt["time_step"]
    V = torch.stack([torch.stack([_values(e, g.r) for e in row]) for row in mat])
    W, U = _eigen(V, d)
    imag = "imaginary" in opt
    step = dt * (-1j if imag else 1.0)
    cap = torch.zeros_like(g.r[0])
    ab = opt.get("absorbing_potential")
    if ab:
        for x, (lo, hi) in zip(g.r, ab["bounds"]):
            cap += torch.exp(ab["exponent"] * torch.clamp(torch.maximum(lo - x, x - hi), min=0.0)) - 1
    decay = torch.exp(-0.5 * cap * abs(step))
    R = torch.einsum("im...,jm...,m...->ij...", U.to(torch.complex128), U.to(torch.complex128),
                     torch.exp(-0.5j * W * step)) * decay
    K = sum(k * k / (2 * m) for k, m in zip(g.k, opt["mass"]))
    phase = torch.exp(-1j * K * step)
    ic = opt["initial_conditions"]
    z = sum(-0.5 * ga * (x - q) ** 2 + 1j * p * (x - q)
            for x, q, p, ga in zip(g.r, ic["position"], ic["momentum"], ic["gamma"]))
    psi = torch.zeros((S,) + tuple(g.r[0].shape), device="cuda", dtype=torch.complex128)
    psi[ic["state"]] = torch.exp(z)
    psi /= math.sqrt(float((psi.abs() ** 2).sum()) * g.dr)
    if ic["adiabatic"]:
        psi = torch.stack([(U[i].to(psi.dtype) * psi).sum(0) for i in range(S)])
    psi0 = psi.clone()
    axes = tuple(range(1, d + 1))
    write, adia = set(opt["write"]), opt["adiabatic"]
    if "spectrum" in opt:
        write.add("acf")
    track = bool(ab and ab.get("track_population"))
    absorbed = torch.zeros(S, device="cuda", dtype=torch.float64)
    Uc = U.to(torch.complex128)

    def basis(x):
        return torch.stack([(Uc[:, i] * x).sum(0) for i in range(S)]) if adia and S > 1 else x

    def apply_r(x):
        return torch.stack([(R[i] * x).sum(0) for i in range(S)])

    def take(x):
        nonlocal absorbed
        if track:
            absorbed = absorbed + ((1 - decay * decay) * basis(x).abs() ** 2).flatten(1).sum(1) * g.dr

    def row(x, want):
        nan = torch.full((1,), math.nan, device="cuda", dtype=torch.float64)
        rho = (x.abs() ** 2).sum(0)
        out = [rho.sum().reshape(1) * g.dr if "norm" in want else nan]
        out += [(rho * q).sum().reshape(1) * g.dr if "position" in want else nan for q in g.r]
        energy = "total_energy" in want
        kin = energy or "kinetic_energy" in want
        if kin or "momentum" in want:
            rk = (torch.fft.fftn(x, dim=axes).abs() ** 2).sum(0)
        out += [(rk * q).sum().reshape(1) * g.dk if "momentum" in want else nan for q in g.k]
        out += [(basis(x).abs() ** 2).flatten(1).sum(1) * g.dr + absorbed if "population" in want else nan.expand(S)]
        if energy or "potential_energy" in want:
            out += [sum((x[i].conj() * V[i, j] * x[j]).real.sum() for i in range(S) for j in range(S)).reshape(1) * g.dr]
        else:
            out += [nan]
        out += [(rk * K).sum().reshape(1) * g.dk if kin else nan]
        if "acf" in want:
            a = (psi0.conj() * x).sum() * g.dr
            out += [a.real.reshape(1), a.imag.reshape(1)]
        else:
            out += [nan, nan]
        return torch.cat(out)

    rows = []
    for i in range(opt["iterations"] + 1):
        if i:
            take(psi)
            psi = torch.fft.ifftn(torch.fft.fftn(apply_r(psi), dim=axes) * phase, dim=axes)
            take(psi)
            psi = apply_r(psi)
        if imag:
            psi = psi / torch.sqrt((psi.abs() ** 2).sum() * g.dr)
        rows.append(row(psi, write))
    final = row(psi, {"norm", "position", "momentum", "population", "total_energy"})
    return torch.stack(rows).cpu().numpy(), psi.reshape(S, -1).cpu().numpy(), final.cpu().numpy()


def _exact_outputs(opt, wavefunction):
    rows, psi, fin = _propagate(opt)
    d, S = len(opt["mass"]), psi.shape[0]
    w, out = opt["write"], {}
    epot, ekin = rows[:, 1 + 2 * d + S:2 + 2 * d + S], rows[:, 2 + 2 * d + S:3 + 2 * d + S]
    if "norm" in w:
        out["norm"] = rows[:, :1]
    if "position" in w:
        out["position"] = rows[:, 1:1 + d]
    if "momentum" in w:
        out["momentum"] = rows[:, 1 + d:1 + 2 * d]
    if "population" in w:
        out["population"] = rows[:, 1 + 2 * d:1 + 2 * d + S]
    if "total_energy" in w:
        out["potential_energy"], out["kinetic_energy"], out["total_energy"] = epot, ekin, epot + ekin
    if "acf" in w:
        out["acf"] = rows[:, 3 + 2 * d + S] + 1j * rows[:, 4 + 2 * d + S]
    out["final"] = np.concatenate([fin[1:1 + 2 * d + S], fin[1 + 2 * d + S:3 + 2 * d + S], fin[:1]])
    if wavefunction:
        out["wavefunction"] = psi
    return out


def exact(case, seed):
    if case["entry"] == "fft":
        x = _fft_input(case, seed).to(torch.complex128)
        return torch.fft.fftn(x) if case["direction"] < 0 else torch.fft.ifftn(x)
    opts = _all_options(case, seed)
    if case["entry"] == "rows":
        return [_propagate(opts[0])[0]]
    if case["entry"] == "batch":
        return [_exact_outputs(o, True) for o in opts]
    if case["entry"] == "serve":
        got = [_propagate(o)[:2] for o in opts]
        return [[rows[:, 1 + 2 * len(o["mass"]):][:, :psi.shape[0]], psi] for o, (rows, psi) in zip(opts, got)]
    return _exact_outputs(opts[0], True)
