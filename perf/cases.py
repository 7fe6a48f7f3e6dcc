"""The work whose speed is measured: what users of this package have it do.

Single runs (``solver.create_instance(...).run()`` and its results), batched
ensembles advanced chunk by chunk, the prescreening sweep's solver call, and
the surrogate's inference and training step. Sizes are those of the presets,
the benchmark workloads and the tests in this repository.

A case is a dict of plain values:

``kind="run"``    one scenario through the solver factory; ``setup`` names the
                  medium, ``solver`` the solver, ``points`` and ``steps`` the
                  grid. FP32 solvers' results are returned as FP32 (their
                  own precision; the package hands them out in FP64 arrays).
``kind="chunk"``  an ensemble of ragged 2-level runs, advanced by ``steps``
                  steps per pass; the pass reads back the chunk's probe rows.
``kind="sweep"``  prescreen.SweepSpace.solve on ``points`` sweep points.
``kind="infer"``  surrogate.FNO.infer on a batch.
``kind="train"``  surrogate.FNO.train_step on a batch (the small learning
                  rate of the end of a cosine decay).
"""
import math

import numpy as np
import torch

from mbsolve_gb300 import ensemble as mb_ensemble
from mbsolve_gb300 import lib as mb
from mbsolve_gb300 import prescreen, setups, solvergpu, surrogate  # noqa: F401

HBAR, EPS0 = 1.05457266e-34, 8.854187817e-12
MU0 = math.pi * 4e-7
C0 = 1.0 / math.sqrt(MU0 * EPS0)
# steps an ensemble of kind "chunk" has before it ends
CHUNK_STEPS = 200000


def listed():
    return [
        # the reference's 0-D preset: one grid point, 10,000 steps, nothing
        # but the latency of a step
        dict(name="point_3lvl_fp64", kind="run", setup="song",
             solver="gpu-fdtd-3lvl-reg-cayley-fp64", points=1, steps=10000),
        # the plain 2-level workload (16,384 points), a stretch of its steps:
        # a single run that leaves most of the chip idle
        dict(name="run_2lvl_fp32", kind="run", setup="sit",
             solver="gpu-fdtd-2lvl-cvr-rodr-fp32", points=16384, steps=2000),
        # the reference's self-induced-transparency preset in double
        # precision, its solvers' default: three regions, full-grid records
        dict(name="sit_2lvl_fp64", kind="run", setup="ziolkowski",
             solver="gpu-fdtd-2lvl-cvr-rodr-fp64", points=32768, steps=10000),
        # the 6-level random medium (65,536 points), both propagators, FP32
        dict(name="run_6lvl_fp32", kind="run", setup="random",
             solver="gpu-fdtd-6lvl-cvr-rodr-fp32", points=65536, steps=500),
        dict(name="run_6lvl_cayley_fp32", kind="run", setup="random",
             solver="gpu-fdtd-6lvl-reg-cayley-fp32", points=65536, steps=200),
        # and its double-precision run, which the FP32 ones are judged by
        dict(name="run_6lvl_fp64", kind="run", setup="random",
             solver="gpu-fdtd-6lvl-cvr-rodr-fp64", points=65536, steps=100),
        # the 3-level Lambda medium, the longest grid (1,048,576 points)
        dict(name="lambda_3lvl_fp32", kind="run", setup="lambda",
             solver="gpu-fdtd-3lvl-reg-cayley-fp32", points=1048576,
             steps=200),
        # a quarter of the benchmark's batched ensemble, the chunk a sweep
        # advances between two reads of its probes
        dict(name="ensemble_2lvl_fp32", kind="chunk",
             solver="gpu-fdtd-2lvl-cvr-rodr-fp32", runs=1024, points=32768,
             steps=300),
        # training data and judging of a sweep: whole solver call on small
        # 6-level runs, host descriptions in, envelopes out
        dict(name="sweep_6lvl_fp32", kind="sweep", points=128,
             window=3e-12),
        # prescreening: the sweep's inference batch, and a handful of points
        dict(name="infer_4096", kind="infer", batch=4096, samples=1024,
             width=64, modes=32, layers=4),
        dict(name="infer_7", kind="infer", batch=7, samples=1024, width=64,
             modes=32, layers=4),
        # one training step of the surrogate at the training batch
        dict(name="train_64", kind="train", batch=64, samples=1024, width=64,
             modes=32, layers=4),
    ]


# cell-updates/s from which draw() chooses a number of steps (orders of
# magnitude only), by (algorithm, precision), for 2 to 6 levels
_RATES = {("cvr-rodr", "fp32"): (3e10, 2e10, 1.5e10, 1e10, 6e9),
          ("cvr-rodr", "fp64"): (1.2e9, 4e8, 2e8, 1.2e8, 8e7),
          ("reg-cayley", "fp32"): (2e10, 1.5e10, 6e9, 3e9, 1.5e9),
          ("reg-cayley", "fp64"): (1.5e9, 8e8, 4e8, 2e8, 1e8)}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["chunk", "infer", "train"])
    if kind == "run":
        prec = rng.choice(["fp32", "fp64"])
        if rng.random() < 0.1:
            return dict(kind="run", setup="vacuum",
                        solver="gpu-fdtd-noop-" + prec,
                        points=_log_int(rng, 100, 1 << 19),
                        steps=rng.randrange(100, 1500))
        algo = rng.choice(["cvr-rodr", "reg-cayley"])
        setup = rng.choice(["sit", "ziolkowski", "random", "random", "random",
                            "lambda", "song"])
        n = {"sit": 2, "ziolkowski": 2, "lambda": 3, "song": 3}.get(
            setup, rng.randrange(2, 7))
        pts = 1 if setup == "song" else _log_int(rng, 100, 1 << 19)
        while setup == "ziolkowski" and not _covers(pts, 150e-6):
            pts += 1
        steps = int(0.03 * _RATES[algo, prec][n - 2] / pts)
        steps = max(20, min(3000, steps)) - rng.randrange(10)
        return dict(kind="run", setup=setup, points=pts, steps=steps,
                    solver="gpu-fdtd-%dlvl-%s-%s" % (n, algo, prec))
    if kind == "chunk":
        return dict(kind="chunk", solver="gpu-fdtd-2lvl-cvr-rodr-fp32",
                    runs=_log_int(rng, 8, 600),
                    points=_log_int(rng, 2200, 32768),
                    steps=rng.randrange(150, 300))
    layers = rng.randrange(2, 5)
    samples = 64 * rng.randrange(3, 17)
    width = 8 * rng.randrange(2, 11)
    modes = 8 * rng.randrange(1, min(4, samples // 32) + 1)
    if kind == "infer":
        return dict(kind="infer", batch=_log_int(rng, 1, 2500),
                    samples=samples, width=width, modes=modes, layers=layers)
    return dict(kind="train", batch=8 * rng.randrange(1, 9), samples=samples,
                width=width, modes=modes, layers=layers)


# ------------------------------------------------------------------ inputs

class _profile(mb.ic_field_random):
    """An initial field given by its values at the grid points."""

    def __init__(self, values):
        super().__init__()
        self._cache[len(values)] = np.ascontiguousarray(values)


def _covers(n, length):
    """Whether the last of n grid points lies within `length` as rounded."""
    return (n - 1) * (length / (n - 1)) <= length


def _length(n, length):
    """The next length that covers n grid points."""
    while not _covers(n, length):
        length = math.nextafter(length, math.inf)
    return length


def _pulses(rng, n, length, amplitude, wavelength):
    """E and H of right- and left-going sech pulses, one per 50 um and at
    least three, as wide as a tenth of the device or 11 um."""
    x = np.arange(n) * (length / max(1, n - 1))
    e, h = np.zeros(n), np.zeros(n)
    count = max(3, int(length / 5e-5))
    for k in range(count):
        x0 = (k + rng.uniform(0.1, 0.9)) / count * length
        w = min(1.1e-5, 0.1 * length)
        a = amplitude * rng.uniform(0.5, 1.0) / np.cosh(
            np.clip((x - x0) / w, -300, 300))
        a = a * np.cos(2 * math.pi * (x - x0) / wavelength +
                       rng.uniform(0, 2 * math.pi))
        e += a
        h += rng.choice([-1.0, 1.0]) * a * math.sqrt(EPS0 / MU0)
    return e, h


def _levels(solver):
    return 0 if "noop" in solver else int(solver.split("-")[2][0])


def _describe(case, seed):
    """(device, scenario) of a case of kind "run"."""
    rng = np.random.default_rng([seed, 1])
    n, steps, N = case["points"], case["steps"], _levels(case["solver"])
    setup = case["setup"]
    spaced = setups.LENGTH_2LVL * (n - 1) / 16383.0
    if setup == "song":
        dt = 80e-15 / 9999
        dev, sce = setups.song2005(endtime=(steps - 1) * dt,
                                   num_timesteps=steps)
        # the preset's pulse, its centre between 0.7 and 12 fs
        return dev, _again(sce, [mb.sech_pulse(
            "sech", 0.0, mb.source.hard_source,
            3.5471e9 * rng.uniform(0.8, 1.2), 3.8118e14,
            17.248 - rng.uniform(13, 17), 1.76 / 5e-15, -math.pi / 2)])
    if setup == "ziolkowski":
        length = 150e-6
        dt = 0.5 * length / (n - 1) / C0
        dev, sce = setups.ziolkowski1995(n, (steps - 1.5) * dt)
        e, h = _pulses(rng, n, length, 2e9, C0 / 2e14)
        sce.set_ic_electric(_profile(e))
        sce.set_ic_magnetic(_profile(h))
        sce.add_record(mb.record("e_out", 0.0, 0.75 * length))
        return dev, sce
    if setup == "lambda":
        length = _length(n, spaced)
        dev, sce = setups.lambda_3lvl(n, steps, length)
        pops = [0.5, 0.2, 0.3]
    elif setup == "sit":
        length = _length(n, spaced)
        dev, sce = setups.sit_2lvl(
            n, steps, length=length, area=rng.uniform(0.5, 4) * math.pi,
            detuning=rng.uniform(-0.05, 0.05),
            t2=math.exp(rng.uniform(math.log(1e-13), math.log(1e-11))))
        pops = [0.9, 0.1]
    elif setup == "vacuum":
        dev = mb.device("vacuum")
        m = setups._material("Vacuum", None, 2.25)
        length = _length(n, spaced)
        dev.add_region(mb.region("Vacuum", m, 0.0, length))
        sce = mb.scenario(
            "vacuum", n, setups._courant_endtime(n, length, steps, 2.25),
            mb.ic_density_const(mb.qm_operator([])), mb.ic_field_const(0.0),
            mb.ic_field_const(0.0))
        sce.add_record(mb.record("e", 0.0, length))
    else:
        length = _length(n, 150e-6)
        dev, sce = setups.random_nlvl(N, n, steps, seed, length)
        pops = rng.dirichlet(np.ones(N))
    if setup == "random":
        e, h = _pulses(rng, n, length, 1e7, C0 / 5e12)
        e = e + 1e5
    else:
        e, h = _pulses(rng, n, length, setups.sech_area_amplitude(2 * math.pi),
                       C0 / 2e14)
    sce.set_ic_electric(_profile(e))
    sce.set_ic_magnetic(_profile(h))
    if setup != "vacuum":
        sce.set_ic_density(mb.ic_density_const(mb.qm_operator(list(pops))))
        sce.add_record(mb.record("d11", mb.record.density, 1, 1,
                                 0.6 * sce.get_endtime(), -1.0))
    # the whole field, at the start and after 60 % of the run
    sce.add_record(mb.record("e_all", 0.6 * sce.get_endtime()))
    sce.add_record(mb.record("h_mid", 0.0, 0.37 * length))
    return dev, sce


def _again(sce, sources):
    """The scenario with other sources."""
    new = mb.scenario(sce.get_name(), sce.get_num_gridpoints(),
                      sce.get_endtime(), sce.get_ic_density(),
                      sce.get_ic_electric(), sce.get_ic_magnetic(),
                      sce.get_num_timesteps())
    for r in sce.get_records():
        new.add_record(r)
    for s in sources:
        new.add_source(s)
    return new


def _describe_chunk(case, seed):
    """The runs of a case of kind "chunk": the benchmark ensemble's
    distributions, with pulses already inside the devices and three probes
    (the facet every step, two inside every fourth)."""
    rng = np.random.default_rng([seed, 2])
    runs = []
    for _ in range(case["runs"]):
        n = int(rng.integers(2048, case["points"] + 1))
        length = _length(n, setups.LENGTH_2LVL * (n - 1) / 16383.0)
        dev, sce = setups.sit_2lvl(
            n, CHUNK_STEPS, rng.uniform(0.5, 4) * math.pi,
            rng.uniform(-0.05, 0.05),
            math.exp(rng.uniform(math.log(1e-13), math.log(1e-11))), 1e-9,
            length)
        e, h = _pulses(rng, n, length,
                       setups.sech_area_amplitude(2 * math.pi), C0 / 2e14)
        sce.set_ic_electric(_profile(e))
        sce.set_ic_magnetic(_profile(h))
        dt = sce.get_endtime() / (CHUNK_STEPS - 1)
        for k in range(2):
            sce.add_record(mb.record("e_in%d" % k, 4.0 * dt,
                                     rng.uniform(0.05, 0.95) * length))
        runs.append((dev, sce))
    return runs


def _space(case):
    return prescreen.SweepSpace(seed=7000, window=case["window"])


def _shapes(case):
    return surrogate.Shapes(S=case["samples"], W=case["width"],
                            Mo=case["modes"], L=case["layers"], F=9)


def _network_inputs(case, seed):
    """Features like prescreen.SweepSpace.features' (input envelope, seven
    scaled parameters, grid coordinate), targets (the envelope delayed and
    attenuated) and weights, drawn on the GPU."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=dev).manual_seed(seed)
    B, S, W = case["batch"], case["samples"], case["width"]
    u = torch.rand(B, 10, generator=g, device=dev)
    t = torch.arange(S, device=dev)[None, :] / S
    X = torch.empty(B, S, 9, device=dev)
    width = 0.03 + 0.05 * u[:, 0:1]
    centre = 0.19 + 0.19 * u[:, 1:2]
    X[..., 0] = 1.0 / torch.cosh((t - centre) / width)
    X[..., 1:8] = (2 * u[:, None, 2:9] - 1)
    X[..., 8] = t
    target = (0.3 + 0.6 * u[:, 9:10]) / torch.cosh((t - centre - 0.02) / width)
    parts = []
    for name, shape in _shapes(case).param_spec():
        r = torch.rand(int(np.prod(shape)), generator=g, device=dev)
        if name.startswith(("wr", "wi")):
            # spectral weights of a network part-way through training
            r = (2 * r - 1) / W
        else:
            r = (2 * r - 1) / math.sqrt(shape[-1] if len(shape) > 1 else W)
        parts.append(r)
    return X, target, torch.cat(parts)


def prepare(case, seed):
    if case["kind"] == "run":
        dev, sce = _describe(case, seed)
        return {"case": case, "solver": mb.solver.create_instance(
            case["solver"], dev, sce)}
    if case["kind"] == "chunk":
        return {"case": case, "ensemble": mb_ensemble.ensemble(
            case["solver"], _describe_chunk(case, seed))}
    if case["kind"] == "sweep":
        space = _space(case)
        return {"case": case, "space": space,
                "points": space.sample(case["points"], seed)}
    X, target, theta = _network_inputs(case, seed)
    net = surrogate.FNO(_shapes(case))
    net.load_params(theta)
    return {"case": case, "net": net, "X": X, "target": target}


def run(state):
    case = state["case"]
    if case["kind"] == "run":
        s = state["solver"]
        s.run()
        kind = np.float32 if case["solver"].endswith("fp32") else np.float64
        return [r.get_data_real().astype(kind, copy=False)
                for r in s.get_results()]
    if case["kind"] == "chunk":
        e, steps = state["ensemble"], case["steps"]
        done = e.progress()[0]
        if done + steps > CHUNK_STEPS:
            raise RuntimeError("the ensemble has run to its end")
        e.advance(steps)
        row = -(-done // 4)
        return [e.probe_rows(0, done, steps).astype(np.float32)] + [
            e.probe_rows(k, row, steps // 4 - 1).astype(np.float32)
            for k in (1, 2)]
    if case["kind"] == "sweep":
        return state["space"].solve(state["points"])[0]
    if case["kind"] == "infer":
        return state["net"].infer(state["X"])
    net = state["net"]
    loss = net.train_step(state["X"], state["target"], lr=1e-6,
                          weight_decay=1e-4)
    return {"loss": loss, "grad": net.grad, "weights": net.theta}


# -------------------------------------------------------------------- work

def _update_flops(solver):
    """Floating-point operations of one grid point's time step."""
    N = _levels(solver)
    if N == 0:
        return 9
    if "cvr" in solver:
        # field update, plane rotations, one propagator product, current
        V = N * N - 1
        return 9 + 12 * (V // 2) + 2 * V * V + 3 * V
    # field update, A X = B with N right-hand sides, two N x N products (one
    # of them Hermitian), two dissipation half steps, current (complex: 8
    # operations per multiply-add)
    return int(9 + 8 * (4 * N ** 3 / 3 + 1.5 * N ** 3) +
               2 * (2 * N * N + N * (N - 1)) + 2 * N * N)


def work(case):
    if case["kind"] == "run":
        N, word = _levels(case["solver"]), 4 if "fp32" in case["solver"] else 8
        n, steps = case["points"], case["steps"]
        state = 3 + (N * N - 1 if "cvr" in case["solver"] else N * N)
        if case["setup"] == "song":
            rows = 4 * steps
        elif case["setup"] == "ziolkowski":
            # E and the inversion every 2.5 fs, E at one point every step
            dt = 0.5 * 150e-6 / (n - 1) / C0
            rows = steps + 2 * n * (1 + int(steps * dt / 2.5e-15))
        else:
            rows = 2 * steps + (2 if N == 0 else 4) * n
        return {"bytes": word * (2 * n * state + rows),
                "flops": n * steps * _update_flops(case["solver"])}
    if case["kind"] == "chunk":
        n = case["runs"] * (2048 + case["points"]) // 2
        return {"bytes": 4 * (2 * n * 6 + 3 * case["runs"] * case["steps"] // 2),
                "flops": n * case["steps"] * _update_flops(case["solver"])}
    if case["kind"] == "sweep":
        dt = 0.5 * 50e-6 / 223 / C0
        n, steps = case["points"] * 224, int(case["window"] / dt)
        return {"bytes": 4 * (2 * n * 38 + case["points"] * 1024),
                "flops": n * steps * _update_flops("gpu-fdtd-6lvl-cvr-")}
    B, S, W = case["batch"], case["samples"], case["width"]
    Mo, L = case["modes"], case["layers"]
    layer = 2 * S * W * 2 * Mo * 2 + 8 * Mo * W * W + 2 * S * W * W
    flops = B * (2 * S * W * 9 + L * layer + 2 * S * W * 128 + 2 * S * 128)
    n = _shapes(case).num_params()
    if case["kind"] == "infer":
        return {"bytes": 4 * (B * S * 10 + n), "flops": flops}
    # forward and backward; weights, gradient and two moments
    return {"bytes": 4 * (B * S * 10 + 7 * n), "flops": 3 * flops}


# ----------------------------------------------- results in 64-bit arithmetic

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _full(op, N):
    """Hermitian matrix of a qm_operator (upper triangle column-major)."""
    m = np.zeros((N, N), dtype=complex)
    d = op.get_main_diagonal()[:N]
    m[np.arange(len(d)), np.arange(len(d))] = d
    off = op.get_off_diagonal()
    q = 0
    for k in range(1, N):
        for j in range(k):
            if q < len(off):
                m[j, k], m[k, j] = off[q], np.conj(off[q])
            q += 1
    return m


def _grid(dev, sce):
    """n_x, dx, n_t, dt of the reference (Courant number 0.5)."""
    n = sce.get_num_gridpoints()
    if n == 1:
        n_t, dx = sce.get_num_timesteps(), 1e13
    else:
        dx = dev.get_length() / (n - 1)
        v = 1.0 / math.sqrt(MU0 * EPS0 * dev.get_minimum_permittivity())
        n_t = int(math.ceil(sce.get_endtime() / (0.5 * dx / v)) + 1)
    return n, dx, n_t, sce.get_endtime() / (n_t - 1)


def _relax(qm, rho):
    """Lindblad relaxation of a matrix."""
    S = np.array(qm.get_relaxation_superop().get_scattering_rates())
    g = qm.get_relaxation_superop().get_dephasing_rates()
    N = len(S)
    out = np.zeros((N, N), dtype=complex)
    out[np.arange(N), np.arange(N)] = S @ np.diag(rho)
    q = 0
    for k in range(1, N):
        for j in range(k):
            out[j, k], out[k, j] = g[q] * rho[j, k], g[q] * rho[k, j]
            q += 1
    return out


def _hermitian_basis(N):
    """Matrices of the real coordinates of a Hermitian matrix: the diagonal,
    then the real and the imaginary part of each upper entry."""
    pairs = [(j, k) for k in range(1, N) for j in range(k)]
    B = np.zeros((N * N, N, N), dtype=complex)
    for i in range(N):
        B[i, i, i] = 1.0
    for q, (j, k) in enumerate(pairs):
        B[N + 2 * q, j, k] = B[N + 2 * q, k, j] = 1.0
        B[N + 2 * q + 1, j, k], B[N + 2 * q + 1, k, j] = 1j, -1j
    return B, pairs


def _coordinates(m, pairs):
    N = m.shape[0]
    out = [m[i, i].real for i in range(N)]
    for j, k in pairs:
        out += [m[j, k].real, m[j, k].imag]
    return np.array(out)


class _rodrigues:
    """exp(L0 dt/2), the field's rotation exp(i mu e dt / hbar) and
    exp(L0 dt/2) on density matrices in the eigenbasis of the dipole
    operator: r [groups, N^2, points] real coordinates, one medium a group."""

    def __init__(self, qms, inits, dt, dev):
        N = qms[0].get_num_levels()
        B, pairs = _hermitian_basis(N)
        A, ang, cur, cur0, pops, r0 = [], [], [], [], [], []
        for qm, init in zip(qms, inits):
            H = _full(qm.get_hamiltonian(), N)
            mu = _full(qm.get_dipole_operator(), N)
            lam, Q = np.linalg.eigh(mu / np.abs(mu).max())
            lam = lam * np.abs(mu).max()

            def free(x):
                return -1j / HBAR * (H @ x - x @ H) + _relax(qm, x)
            gen = np.stack([_coordinates(
                Q.conj().T @ free(Q @ b @ Q.conj().T) @ Q, pairs)
                for b in B], axis=1)
            A.append(torch.linalg.matrix_exp(
                torch.tensor(gen * (dt / 2), dtype=torch.float64)))
            ang.append([(lam[j] - lam[k]) * dt / HBAR for j, k in pairs])
            cur.append([qm.get_carrier_density() * np.trace(
                mu @ free(Q @ b @ Q.conj().T)).real for b in B])
            pops.append([[(Q @ b @ Q.conj().T)[i, i].real for b in B]
                         for i in range(N)])
            # the coherence vector keeps only the last off-diagonal entry of
            # the initial matrix, as its first (the reference's indexing)
            rho = np.zeros((N, N), dtype=complex)
            d = init.get_main_diagonal()[:N]
            rho[np.arange(len(d)), np.arange(len(d))] = d
            off = init.get_off_diagonal()
            if off:
                rho[0, 1], rho[1, 0] = off[-1], np.conj(off[-1])
            r0.append(_coordinates(Q.conj().T @ rho @ Q, pairs))
        put = lambda v: torch.tensor(np.array(v), dtype=torch.float64, device=dev)  # noqa: E731
        self.N, self.P = N, len(pairs)
        self.A = torch.stack(A).to(dev)
        self.ang, self.cur, self.pops, self.r0 = put(ang), put(cur), put(pops), put(r0)

    def start(self, points):
        return self.r0[:, :, None].expand(-1, -1, points).contiguous()

    def _free(self, r):
        if self.N > 2 or len(self.A) == 1:
            return torch.matmul(self.A, r)
        return torch.stack([sum(self.A[:, i, j, None] * r[:, j]
                                for j in range(self.N ** 2))
                            for i in range(self.N ** 2)], dim=1)

    def step(self, r, e):
        r = self._free(r)
        N = self.N
        x = self.ang[:, :, None] * e[:, None, :]
        s, c = torch.sin(x), torch.cos(x)
        re, im = r[:, N::2], r[:, N + 1::2]
        turned = torch.empty_like(r)
        turned[:, :N] = r[:, :N]
        turned[:, N::2] = c * re - s * im
        turned[:, N + 1::2] = s * re + c * im
        return self._free(turned)

    def current(self, r):
        return torch.einsum("gv,gvl->gl", self.cur, r)

    def population(self, r, i):
        return torch.einsum("gv,gvl->gl", self.pops[:, i], r)


class _cayley:
    """Dissipation half step, (1 + iK)^-1 (1 - iK) with K = dt / (2 hbar)
    (H0 - mu e), dissipation half step: rho [N, N, points] of one medium."""

    def __init__(self, qm, init, dt, dev):
        N = qm.get_num_levels()
        put = lambda v: torch.tensor(np.array(v), dtype=torch.complex128, device=dev)  # noqa: E731
        H = _full(qm.get_hamiltonian(), N)
        mu = _full(qm.get_dipole_operator(), N)
        r = qm.get_relaxation_superop()
        self.N = N
        self.kH, self.kM = put(H * (dt / 2 / HBAR)), put(mu * (dt / 2 / HBAR))
        S = torch.tensor(r.get_scattering_rates(), dtype=torch.float64)
        self.D1 = torch.linalg.matrix_exp(S * (dt / 2)).to(dev)
        B, pairs = _hermitian_basis(N)
        D2 = np.ones((N, N))
        for q, (j, k) in enumerate(pairs):
            D2[j, k] = D2[k, j] = math.exp(r.get_dephasing_rates()[q] * dt / 2)
        self.D2 = put(D2)
        # the current's weights on the entries of rho
        w = np.zeros((N, N), dtype=complex)
        for a in range(N):
            for b in range(N):
                u = np.zeros((N, N), dtype=complex)
                u[a, b] = 1.0
                w[a, b] = qm.get_carrier_density() * np.trace(
                    (-1j / HBAR * (H @ u - u @ H) + _relax(qm, u)) @ mu)
        self.w = put(w)
        self.r0 = put(_full(init, N))

    def start(self, points):
        return self.r0[:, :, None].expand(-1, -1, points).contiguous()

    def _dissipate(self, rho):
        N = self.N
        out = rho * self.D2[:, :, None]
        i = torch.arange(N, device=rho.device)
        out[i, i] = (self.D1 @ rho[i, i].real).to(rho.dtype)
        return out

    @staticmethod
    def _mul(a, b):
        return sum(a[:, l, None, :] * b[None, l, :, :] for l in range(a.shape[1]))

    def step(self, rho, e):
        N = self.N
        e = e[0]
        rho = self._dissipate(rho)
        K = self.kH[:, :, None] - self.kM[:, :, None] * e
        eye = torch.eye(N, dtype=K.dtype, device=K.device)[:, :, None]
        A, U = eye + 1j * K, eye - 1j * K
        for k in range(N):
            for i in range(k + 1, N):
                f = A[i, k] / A[k, k]
                A[i] = A[i] - f * A[k]
                U[i] = U[i] - f * U[k]
        for k in range(N - 1, -1, -1):
            for i in range(k + 1, N):
                U[k] = U[k] - A[k, i] * U[i]
            U[k] = U[k] / A[k, k]
        rho = self._mul(self._mul(U, rho), U.conj().transpose(0, 1))
        return self._dissipate(rho)

    def current(self, rho):
        return torch.einsum("ab,abl->l", self.w, rho).real[None]

    def population(self, rho, i):
        return rho[i, i].real[None]


def _simulate(runs, solver, steps):
    """Records of `steps` steps of the runs in FP64: [record][run] arrays.
    Several runs have one medium each; one run may have several regions."""
    dev = _device()
    f64 = dict(dtype=torch.float64, device=dev)
    R = len(runs)
    grids = [_grid(d, s) for d, s in runs]
    L = max(g[0] for g in grids)
    a, b, c, gam, dxi = (torch.zeros(R, L, **f64) for _ in range(5))
    E, H = torch.zeros(R, L, **f64), torch.zeros(R, L, **f64)
    last = torch.tensor([g[0] - 1 for g in grids], device=dev)
    rows = torch.arange(R, device=dev)
    inside = torch.arange(L, device=dev)[None, :] <= last[:, None]
    segments = []
    for r, (d, s) in enumerate(runs):
        n, dx, n_t, dt = grids[r]
        for f, ic in ((E, s.get_ic_electric()), (H, s.get_ic_magnetic())):
            v = ic.values(n) if isinstance(ic, mb.ic_field_random) else \
                np.full(n, ic.initialize(0.0))
            f[r, :n] = torch.tensor(v, **f64)
        x = np.arange(n) * dx
        which = np.full(n, -1)
        regions = d.get_regions()
        for i in range(len(regions) - 1, -1, -1):
            which[(x >= regions[i].get_x_start()) &
                  (x <= regions[i].get_x_end())] = i
        for i, g in enumerate(regions):
            m = g.get_material()
            at = np.flatnonzero(which == i)
            if not len(at):
                continue
            lo, hi = int(at[0]), int(at[-1]) + 1
            eps = EPS0 * m.get_rel_permittivity()
            mu = MU0 * m.get_rel_permeability()
            loss = 2.0 * m.get_losses() * math.sqrt(eps / mu) * dt / (2 * eps)
            a[r, lo:hi] = (1 - loss) / (1 + loss)
            b[r, lo:hi] = dt / eps / (1 + loss)
            c[r, lo:hi] = dt / (mu * dx)
            gam[r, lo:hi] = m.get_overlap_factor()
            if m.get_qm() is not None and "noop" not in solver:
                segments.append((r, lo, hi, m.get_qm(), s.get_ic_density().initialize(0.0), dt))
        dxi[r] = 1.0 / dx
    # one group of all runs, or one per region
    models = []
    if R > 1:
        models.append((slice(0, L), _rodrigues(
            [g[3] for g in segments], [g[4] for g in segments], segments[0][5], dev)))
    else:
        for _, lo, hi, qm, init, dt in segments:
            models.append((slice(lo, hi), _rodrigues([qm], [init], dt, dev)
                           if "cvr" in solver else _cayley(qm, init, dt, dev)))
    rho = [m.start(at.stop - at.start) for at, m in models]
    P = torch.zeros(R, L, **f64)
    tables, records = [], []
    for r, (d, s) in enumerate(runs):
        n, dx, n_t, dt = grids[r]
        t = np.arange(steps) * dt
        for q in s.get_sources():
            with np.errstate(over="ignore"):
                v = q._ampl / np.cosh(q._beta * t - q._phase) * np.sin(
                    2 * math.pi * q._freq * t - q._phase_sin)
            tables.append((r, int(q.get_position() / dx), q.get_type(),
                           torch.tensor(v, **f64)))
        for k, q in enumerate(s.get_records()):
            if q.get_interval() <= dt:
                ratio, count = 1.0, n_t
            else:
                ratio = dt / q.get_interval()
                count = int(math.floor(s.get_endtime() / q.get_interval()) + 1)
            j = np.arange(steps)
            new = np.floor(ratio * j) != np.floor(ratio * (j - 1))
            new[0] = True
            row = np.floor(ratio * j).astype(int)
            due = {int(i): int(row[i]) for i in j[new] if row[i] < count}
            at = slice(0, n) if q.get_position() < 0 else \
                slice(int(round(q.get_position() / dx)), int(round(q.get_position() / dx)) + 1)
            out = torch.zeros(min(count, max(due.values()) + 1),
                              at.stop - at.start, **f64)
            records.append((k, r, q, due, at, out))
    # single-point field records are gathered together, every step
    kind = mb.record.type
    probes = [x for x in records if x[4].stop - x[4].start == 1 and
              x[2].get_type() in (kind.electric, kind.magnetic)]
    index = lambda v: torch.tensor(v, device=dev, dtype=torch.long)  # noqa: E731
    probe_at = index([x[1] for x in probes]), index([x[4].start for x in probes])
    electric = index([x[2].get_type() for x in probes]) == kind.electric
    trace = torch.zeros(steps, len(probes), **f64)
    due = {}
    for x in records:
        if not any(x is y for y in probes):
            for n, row in x[3].items():
                due.setdefault(n, []).append((x, row))
    hard = [q for q in tables if q[2] == mb.source.hard_source]
    soft = [q for q in tables if q[2] != mb.source.hard_source]
    hard, soft = [(index([q[0] for q in g]), index([q[1] for q in g]),
                   torch.stack([q[3] for q in g])) if g else None
                  for g in (hard, soft)]
    zero = torch.zeros(R, 1, **f64)

    def value(x):
        q, r, at = x[2], x[1], x[4]
        if q.get_type() == kind.electric:
            return E[r, at]
        if q.get_type() == kind.magnetic:
            return H[r, at]
        density = q.get_type() == kind.density
        # points without a medium hold the zero coherence vector
        out = torch.full((L,), 1.0 / _levels(solver) if density and
                         "cvr" in solver else 0.0, **f64)
        for (seg, m), y in zip(models, rho):
            v = m.population(y, q.get_row()) if density else \
                m.population(y, 1) - m.population(y, 0)
            out[seg] = v[r if R > 1 else 0]
        return out[at]

    be, bp = b * dxi, b * gam
    for n in range(steps):
        hn = torch.cat([H[:, 1:], zero], dim=1)
        hn[rows, last] = 0.0
        E = a * E + be * (hn - H) - bp * P
        if hard:
            E[hard[0], hard[1]] = hard[2][:, n]
        if soft:
            E.index_put_((soft[0], soft[1]), soft[2][:, n], accumulate=True)
        H = H + c * (E - torch.cat([zero, E[:, :-1]], dim=1))
        H[:, 0] = 0.0
        for i, (at, m) in enumerate(models):
            rho[i] = m.step(rho[i], E[:, at])
            P[:, at] = m.current(rho[i])
        if probes:
            trace[n] = torch.where(electric, E[probe_at], H[probe_at])
        for x, row in due.get(n, ()):
            x[5][row] = value(x)
    for i, x in enumerate(probes):
        x[5][list(x[3].values()), 0] = trace[list(x[3].keys()), i]
    out = {}
    for k, _, _, _, _, v in records:
        out.setdefault(k, []).append(v.reshape(-1))
    return [out[k] for k in sorted(out)]


def _network(case, X, target, theta):
    """Output, mean squared error and gradient of the network."""
    sh = _shapes(case)
    S, W, Mo, L = sh.S, sh.W, sh.Mo, sh.L
    X, target = X.double(), target.double()
    theta = theta.double().requires_grad_(case["kind"] == "train")
    p, o = {}, 0
    for name, shape in sh.param_spec():
        n = int(np.prod(shape))
        p[name] = theta[o:o + n].view(shape)
        o += n
    ang = 2 * math.pi * torch.arange(Mo, device=X.device)[:, None] * \
        torch.arange(S, device=X.device)[None, :] / S
    c, s = torch.cos(ang.double()), torch.sin(ang.double())
    twice = torch.full((Mo, 1), 2.0, dtype=torch.float64, device=X.device)
    twice[0] = 1.0
    gelu = torch.nn.functional.gelu

    def forward(X):
        v = X @ p["P"].T + p["bp"]
        for l in range(L):
            re = torch.einsum("ms,bsc->bmc", c / S, v)
            im = torch.einsum("ms,bsc->bmc", -s / S, v)
            wr, wi = p["wr%d" % l], p["wi%d" % l]
            yr = torch.einsum("bmc,mco->bmo", re, wr) - \
                torch.einsum("bmc,mco->bmo", im, wi)
            yi = torch.einsum("bmc,mco->bmo", re, wi) + \
                torch.einsum("bmc,mco->bmo", im, wr)
            v = torch.einsum("ms,bmo->bso", twice * c, yr) - \
                torch.einsum("ms,bmo->bso", twice * s, yi) + \
                v @ p["W%d" % l].T + p["bw%d" % l]
            if l < L - 1:
                v = gelu(v)
        return gelu(v @ p["Q1"].T + p["bq1"]) @ p["q2"] + p["bq2"]

    if case["kind"] == "infer":
        with torch.no_grad():
            return torch.cat([forward(x) for x in X.split(64)])
    loss = ((forward(X) - target) ** 2).mean()
    loss.backward()
    return loss.detach(), theta.grad


def _envelope(e, space):
    """Twice the mean of e exp(-2 pi i f t) over one carrier period around
    each of the window's samples."""
    t = torch.arange(e.shape[1], dtype=torch.float64, device=e.device) * \
        (space.record_every * space.dt)
    z = torch.cumsum(e * torch.exp(-2j * math.pi * space.f0 * t), dim=1)
    z = torch.cat([torch.zeros_like(z[:, :1]), z], dim=1)
    c = np.arange(space.samples) * (space.window / space.samples)
    step = space.record_every * space.dt
    lo = np.maximum(np.ceil((c - 0.5 / space.f0) / step), 0).astype(int)
    hi = np.minimum(np.floor((c + 0.5 / space.f0) / step), e.shape[1] - 1).astype(int)
    n = torch.tensor(np.maximum(hi - lo + 1, 1), device=e.device)
    return 2.0 * (z[:, hi + 1] - z[:, lo]).abs() / n


def exact(case, seed):
    if case["kind"] == "run":
        got = _simulate([_describe(case, seed)], case["solver"], case["steps"])
        return [v[0] for v in got]
    if case["kind"] == "chunk":
        steps = case["steps"]
        got = _simulate(_describe_chunk(case, seed), case["solver"], steps)
        return [torch.stack(got[0])[:, :steps]] + [
            torch.stack(v)[:, :steps // 4 - 1] for v in got[1:]]
    if case["kind"] == "sweep":
        space = _space(case)
        p = space.sample(case["points"], seed)
        got = _simulate([space.run(p, i) for i in range(case["points"])],
                        "gpu-fdtd-6lvl-cvr-rodr-fp32", space.n_t)
        e = torch.stack(got[0])
        return _envelope(e, space) / torch.tensor(
            p["amplitude"], dtype=torch.float64, device=e.device)[:, None]
    X, target, theta = _network_inputs(case, seed)
    if case["kind"] == "infer":
        return _network(case, X, target, theta)
    loss, grad = _network(case, X, target, theta)
    # the first Adam step at a learning rate of 1e-6: its size is the rate
    # wherever a gradient stands clear of zero
    g = grad + 1e-4 * theta.double()
    return {"loss": loss.reshape(1), "grad": grad,
            "weights": theta.double() - 1e-6 * g / (g.abs() + 1e-8)}
