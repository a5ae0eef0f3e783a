"""The work that users of this engine have it do, as cases to time.

A case is a plain dict; its "family" says which public entry points it goes
through:

  step        Context.propagate: one propagate_vector call for a few vectors,
              host arrays in and out (the smallest call)
  absorption  Context.absorption and absorption_fft: a linear spectrum from a
              loaded trajectory ("load": the trajectory is handed over from
              host memory in the same pass, as a program that runs once does)
  linear      Context.linear and absorption_fft: CD and LD spectra
  twodir      Context.twodir: the 2DIR and 2DUVvis families
  adjoint     absorption_model and backward_absorption: one step of a fit
  batch       Batch.run with every job's response and spectrum

The trajectories are the seeded synthetic ones of nise_2017_b200.synth with
the statistics of its workloads (amide-I-like chains and clusters around
1650 cm^-1, chromophore lattices around 15000 cm^-1).  The results of an FP32
context are returned in single precision, as its output files hold them; those
of an FP64 context in double.
"""
import ctypes
import math

import numpy as np
import torch

import nise_2017_b200 as nise
from nise_2017_b200 import synth

# 2 pi c in rad per (cm^-1 fs), with the constants of the reference's headers
ANGULAR = float(np.float32(2.99792458e-5)) * float(np.float32(2 * 3.14159265359))
LIGHT = float(np.float32(2.99792458e-5))
FIT_SCALE, FIT_LIFETIME = 1.05, 900.0


def listed():
    return [
        # one time step of the three polarisation vectors of a 16-site chain: the
        # reference's own per-vector call, launches and copies count
        {"name": "step_chain16", "family": "step", "n": 16, "nvec": 3, "prop": "Coupling", "precision": 32},
        # a whole small job from host memory: the 16-site chain of the first workload,
        # 10000 Full frames, 494 start points, Trotter
        {"name": "job_chain16", "family": "absorption", "geometry": "chain", "ham": "Full", "n": 16, "frames": 10000,
         "t1": 128, "sample": 20, "prop": "Coupling", "precision": 32, "load": True},
        # the reference's default propagation on a fluctuating Full Hamiltonian, a
        # protein-sized amide-I band: a propagator per frame
        {"name": "abs_full48_sparse", "family": "absorption", "geometry": "cluster", "ham": "Full", "n": 48,
         "frames": 2000, "t1": 128, "sample": 20, "prop": "Sparse", "precision": 32, "load": False},
        # the same above the size of a matrix that one SM's shared memory holds
        {"name": "abs_full200_sparse", "family": "absorption", "geometry": "cluster", "ham": "Full", "n": 200,
         "frames": 600, "t1": 96, "sample": 10, "prop": "Sparse", "precision": 32, "load": False},
        # the benchmark: exact propagation on the 1024-site lattice, 1995 start points
        {"name": "abs_lattice1024_sparse", "family": "absorption", "geometry": "lattice", "ham": "Coupling", "n": 1024,
         "frames": 100000, "t1": 256, "sample": 50, "prop": "Sparse", "precision": 32, "load": False},
        # Trotter on a lattice of the mixed batch (195 start points, an odd size)
        {"name": "abs_lattice547_trotter", "family": "absorption", "geometry": "lattice", "ham": "Coupling", "n": 547,
         "frames": 5000, "t1": 128, "sample": 25, "prop": "Coupling", "precision": 32, "load": False},
        # Runge-Kutta on a small odd-sized cluster with dense couplings
        {"name": "abs_full33_rk4", "family": "absorption", "geometry": "cluster", "ham": "Full", "n": 33,
         "frames": 1500, "t1": 64, "sample": 10, "prop": "RK4", "precision": 32, "load": False},
        # circular dichroism, a small difference of large terms: 3 N vectors per
        # start point in FP64
        {"name": "cd_full40_f64", "family": "linear", "tech": "CD", "n": 40, "frames": 900, "t1": 64, "sample": 40,
         "prop": "Sparse", "precision": 64},
        # the 2DIR workload: 64 oscillators, Trotter, ten of its start points
        {"name": "twodir_cluster64", "family": "twodir", "tech": "2DIR", "ham": "Coupling", "n": 64, "points": 10,
         "t1": 64, "t2": 0, "t3": 64, "sample": 100, "prop": "Coupling", "precision": 32},
        # 2DIR of a peptide with a waiting time and the default propagation
        {"name": "twodir_peptide12_sparse", "family": "twodir", "tech": "2DIR", "ham": "Full", "n": 12, "points": 24,
         "t1": 32, "t2": 10, "t3": 32, "sample": 20, "prop": "Sparse", "precision": 32},
        # forward and backward of a fit of site shifts, coupling scale and lifetime: the
        # adjoint workload's 256-site chain with a quarter of its trajectory
        {"name": "fit_chain256", "family": "adjoint", "n": 256, "frames": 5000, "t1": 128, "sample": 20,
         "prop": "Coupling"},
        # many trajectories of mixed sizes in one launch, Trotter and exact by turns
        {"name": "batch_mixed10", "family": "batch", "jobs": 10, "smallest": 8, "largest": 600, "frames": 2500,
         "t1": 128, "sample": 25},
    ]


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithm, odd ones among them."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    family = rng.choice(["step", "absorption", "absorption", "absorption", "linear", "twodir", "twodir", "adjoint",
                         "batch"])
    if family == "step":
        return {"family": family, "n": size(5, 150), "nvec": size(1, 200), "prop": rng.choice(["Coupling", "Sparse", "RK4"]),
                "precision": rng.choice([32, 32, 64])}
    if family == "absorption":
        kind = rng.choice(["chain", "full", "large", "lattice", "lattice", "rk4"])
        c = {"family": family, "geometry": "cluster", "ham": "Full", "n": 0, "frames": 0, "t1": size(48, 160), "sample": 0,
             "prop": "Sparse", "precision": 32, "load": rng.random() < 0.3}
        if kind == "chain":
            c.update(geometry="chain", n=size(5, 64), frames=size(1500, 12000), sample=size(8, 40), prop="Coupling",
                     precision=rng.choice([32, 32, 64]))
        elif kind == "full":
            c.update(n=size(6, 120), frames=size(400, 2000), sample=size(8, 40),
                     prop=rng.choice(["Sparse", "Sparse", "Diagonal", "Coupling"]), precision=rng.choice([32, 32, 64]))
        elif kind == "large":
            c.update(n=size(121, 300), frames=size(250, 500), sample=size(8, 25), t1=size(48, 96))
        elif kind == "lattice":
            c.update(geometry="lattice", ham="Coupling", n=size(64, 1024), frames=size(1500, 20000), sample=size(20, 60),
                     prop=rng.choice(["Sparse", "Diagonal", "Coupling"]))
        else:
            c.update(n=size(5, 64), frames=size(400, 1500), sample=size(8, 30), prop="RK4",
                     precision=rng.choice([32, 32, 64]))
        return c
    if family == "linear":
        return {"family": family, "tech": rng.choice(["CD", "LD"]), "n": size(6, 60), "frames": size(400, 1200),
                "t1": size(32, 96), "sample": size(20, 60), "prop": rng.choice(["Sparse", "Coupling"]),
                "precision": rng.choice([32, 64])}
    if family == "twodir":
        small = rng.random() < 0.6
        n = size(5, 24) if small else size(25, 64)
        return {"family": family, "tech": rng.choice(["2DIR", "2DIR", "2DIR", "2DUVvis"]),
                "ham": rng.choice(["Full", "Coupling"]), "n": n, "points": size(4, 24) if small else size(2, 8),
                "t1": size(16, 48), "t2": rng.choice([0, 0, 5, 20]), "t3": 0, "sample": size(10, 60),
                "prop": rng.choice(["Coupling", "Coupling", "Sparse"]) if n <= 16 else "Coupling", "precision": 32}
    if family == "adjoint":
        return {"family": family, "n": size(16, 256), "frames": size(800, 4000), "t1": size(48, 128),
                "sample": size(15, 40), "prop": "Coupling"}
    return {"family": family, "jobs": size(3, 10), "smallest": size(8, 24), "largest": size(100, 600),
            "frames": size(800, 2500), "t1": size(48, 128), "sample": size(20, 40)}


# ------------------------------------------------------------------ inputs
GEOMETRY = {"chain": synth.CHAIN, "cluster": synth.CLUSTER, "lattice": synth.LATTICE}


def _records(spec):
    """The trajectory's record images in host memory: energies, dipoles and, for static couplings, the coupling record."""
    n = spec.n_sites
    static = spec.ham_type == synth.COUPLING
    energy = np.empty(spec.frames * 4 * (1 + (n if static else n * (n + 1) // 2)), np.uint8)
    dipole = np.empty((spec.dipole_frames or spec.frames) * 4 * (1 + 3 * n), np.uint8)
    coupling = np.empty(4 * (1 + n * (n + 1) // 2), np.uint8) if static else None
    rc = synth.lib().nise_synth_fill(ctypes.byref(spec), energy.ctypes.data, dipole.ctypes.data,
                                     coupling.ctypes.data if static else None, None, None)
    if rc:
        raise RuntimeError("trajectory generator: %d" % rc)
    return energy, dipole, coupling


def _site_spec(geometry, ham, n, frames, seed, **more):
    """A synthetic trajectory with the statistics of the repository's workloads."""
    static = ham == "Coupling"
    d = {"n_sites": n, "frames": frames, "seed": seed + 1, "ham_type": synth.COUPLING if static else synth.FULL,
         "dipole_frames": 1 if static else 0, "mu_jitter": 0.0 if static else 0.05, "geometry": GEOMETRY[geometry]}
    if geometry == "lattice":
        return synth.c1_spec(**{**d, **more})
    if geometry == "cluster":
        return synth.c2_spec(**{**d, **more})
    return synth.c0_spec(**{**d, **more})


def _keywords(geometry, ham, n, frames, **more):
    base = {"lattice": synth.c1_keywords, "cluster": synth.c2_keywords, "chain": synth.c0_keywords}[geometry]
    return base(Singles=n, Length=frames, HamiltonianType=ham, **more)


def _precision(case):
    return nise.FP64 if case.get("precision") == 64 else nise.FP32


def _as_written(context, *arrays):
    """Responses and spectra in the type of the context's output files."""
    dtype = np.float32 if context.params.precision == nise.FP32 else np.float64
    return [a.astype(dtype) for a in arrays]


def _absorption_setup(case, seed):
    spec = _site_spec(case["geometry"], case["ham"], case["n"], case["frames"], seed)
    kw = _keywords(case["geometry"], case["ham"], case["n"], case["frames"], Technique="Absorption",
                   Propagation=case["prop"], RunTimes="%d 0 0" % case["t1"], Samplerate=case["sample"], Threshold=0)
    return spec, kw


def _linear_setup(case, seed):
    spec = _site_spec("cluster", "Full", case["n"], case["frames"], seed)
    kw = _keywords("cluster", "Full", case["n"], case["frames"], Technique=case["tech"], Propagation=case["prop"],
                   RunTimes="%d 0 0" % case["t1"], Samplerate=case["sample"], Threshold=0)
    return spec, kw


def _positions(case, seed):
    """CD's site positions per frame, in the dipole file's record layout."""
    rng = np.random.default_rng(seed + 17)
    n, frames = case["n"], case["frames"]
    rec = np.zeros((frames, 1 + 3 * n), np.float32)
    base = rng.uniform(0, 8.0 * n ** (1 / 3), size=(1, 3 * n))
    rec[:, 1:] = base + rng.normal(0, 0.05, size=(frames, 3 * n))
    return rec


def _twodir_setup(case, seed):
    t1, t2, t3 = case["t1"], case["t2"], case["t1"]  # the reference sets t3 to t1
    frames = t1 + t2 + t3 + 1 + (case["points"] - 1) * case["sample"] + 1
    spec = _site_spec("cluster", case["ham"], case["n"], frames, seed, dt_fs=2.0)
    kw = _keywords("cluster", case["ham"], case["n"], frames, Technique=case["tech"], Propagation=case["prop"],
                   RunTimes="%d %d %d" % (t1, t2, t3), Samplerate=case["sample"], EndPoint=case["points"], Threshold=0)
    return spec, kw


def _adjoint_setup(case, seed):
    spec = synth.c3_spec(n_sites=case["n"], frames=case["frames"], seed=seed + 1)
    kw = synth.c3_keywords(Singles=case["n"], Length=case["frames"], RunTimes="%d 0 0" % case["t1"],
                           Samplerate=case["sample"], Propagation=case["prop"])
    return spec, kw


def _adjoint_inputs(case, seed, rows):
    rng = np.random.default_rng(seed + 5)
    return rng.normal(0, 5.0, size=case["n"]), rng.normal(0, 1.0, size=rows), rng.normal(0, 1.0, size=rows)


def _batch_jobs(case, seed):
    """(spec, keywords) of every job: sizes evenly spread over their logarithm, Trotter and exact by turns."""
    jobs = []
    for i in range(case["jobs"]):
        n = round(case["smallest"] * (case["largest"] / case["smallest"]) ** (i / max(1, case["jobs"] - 1)))
        spec = _site_spec("lattice", "Coupling", n, case["frames"], seed * 100 + i)
        kw = _keywords("lattice", "Coupling", n, case["frames"], Technique="Absorption",
                       Propagation="Diagonal" if i % 2 else "Coupling", RunTimes="%d 0 0" % case["t1"],
                       Samplerate=case["sample"], FFT=1024)
        jobs.append((spec, kw))
    return jobs


def _step_inputs(case, seed):
    rng = np.random.default_rng(seed + 3)
    n, nvec = case["n"], case["nvec"]
    h = np.zeros((nvec, n * (n + 1) // 2), np.float32)
    iu = np.triu_indices(n)
    off = iu[0] != iu[1]
    near = (iu[1] - iu[0]) == 1
    h[:, ~off] = rng.normal(0, 20.0, size=(nvec, n))
    h[:, off] = rng.normal(0, 1.0, size=(nvec, int(off.sum())))
    h[:, near] += -8.0
    dtype = np.float64 if case["precision"] == 64 else np.float32
    return h, rng.normal(size=(nvec, n)).astype(dtype), rng.normal(size=(nvec, n)).astype(dtype)


def prepare(case, seed):
    family = case["family"]
    if family == "step":
        kw = synth.c0_keywords(Singles=case["n"], Propagation=case["prop"], Threshold=0)
        context = nise.Context(nise.params_from_keywords(kw, precision=_precision(case)))
        return {"case": case, "context": context, "inputs": _step_inputs(case, seed)}
    if family == "absorption":
        spec, kw = _absorption_setup(case, seed)
        context = nise.Context(nise.params_from_keywords(kw, precision=_precision(case)))
        records = _records(spec)
        if not case["load"]:
            context.set_trajectory(*records)
            records = None
        return {"case": case, "context": context, "records": records}
    if family == "linear":
        spec, kw = _linear_setup(case, seed)
        context = nise.Context(nise.params_from_keywords(kw, precision=_precision(case)))
        context.set_trajectory(*_records(spec))
        if case["tech"] == "CD":
            context.set_operators(position=_positions(case, seed))
        return {"case": case, "context": context}
    if family == "twodir":
        spec, kw = _twodir_setup(case, seed)
        context = nise.Context(nise.params_from_keywords(kw, precision=_precision(case)))
        context.set_trajectory(*_records(spec))
        return {"case": case, "context": context}
    if family == "adjoint":
        spec, kw = _adjoint_setup(case, seed)
        context = nise.Context(nise.params_from_keywords(kw))
        context.set_trajectory(*_records(spec))
        return {"case": case, "context": context, "inputs": _adjoint_inputs(case, seed, len(_axis(context.params)[0]))}
    contexts = []
    for spec, kw in _batch_jobs(case, seed):
        context = nise.Context(nise.params_from_keywords(kw))
        context.set_trajectory(*_records(spec))
        contexts.append(context)
    return {"case": case, "contexts": contexts, "batch": nise.Batch(contexts)}


def run(state):
    case = state["case"]
    family = case["family"]
    if family == "batch":
        batch = state["batch"]
        batch.run()
        out = []
        for i, context in enumerate(state["contexts"]):
            re, im, samples = batch.result(i)
            out.append(_as_written(context, re, im, *batch.spectrum(i)) + [samples])
        return out
    context = state["context"]
    if family == "step":
        return context.propagate(*state["inputs"])
    if family == "absorption":
        if state["records"] is not None:
            context.set_trajectory(*state["records"])
        re, im, samples = context.absorption()
        return _as_written(context, re, im, *context.absorption_fft(re, im, samples)) + [samples]
    if family == "linear":
        re, im, samples = context.linear()
        return _as_written(context, re, im, *context.absorption_fft(re[0], im[0], samples)) + [samples]
    if family == "twodir":
        response, samples = context.twodir()
        return _as_written(context, response) + [samples]
    shift, dre, dim = state["inputs"]
    w, sr, si = context.absorption_model(shift, FIT_SCALE, FIT_LIFETIME)
    g_shift, g_scale, g_lifetime = context.backward_absorption(shift, FIT_SCALE, FIT_LIFETIME, dre, dim)
    return [w, sr, si, g_shift, g_scale, g_lifetime]


# -------------------------------------------------------------------- work
def _points(frames, t1, sample):
    return (frames - t1 - 1) // sample + 1


def _job_work(geometry, ham, n, frames, t1, sample, prop, vectors, precision=32):
    """Bytes and operations of a linear-response job: every record read once, every vector stepped t1 - 1 times."""
    per_frame = 4.0 * (n if ham == "Coupling" else n * (n + 1) / 2 + 3 * n)
    # directed couplings per site: 2 in a chain, about 11 on the lattice (cut at 2 cm^-1), nearly all in a cluster
    nnz = n * {"chain": 2.0, "lattice": min(11.3, n - 1.0), "cluster": 0.95 * (n - 1.0)}[geometry]
    steps = float(_points(frames, t1, sample)) * vectors * (t1 - 1)
    if prop == "Coupling":  # five sub-steps of one 12-operation rotation per coupling and two phases per site
        flops = steps * 5 * (6.0 * nnz + 12.0 * n)
    elif prop == "RK4":  # five sub-steps of four products and the update
        flops = steps * 5 * (16.0 * nnz + 40.0 * n)
    else:  # five terms of the series of exp(-i H t)
        flops = steps * 5 * (4.0 * nnz + 10.0 * n)
    return {"bytes": frames * per_frame + 32.0 * t1, "flops": flops}


def work(case):
    family, n = case["family"], case["n"] if "n" in case else 0
    if family == "step":
        rsz = case["precision"] / 8
        per = {"Coupling": 5 * (6.0 * n * (n - 1) + 12.0 * n), "RK4": 5 * (16.0 * n * n + 40.0 * n),
               "Sparse": 5 * (4.0 * n * n + 10.0 * n)}[case["prop"]]
        return {"bytes": case["nvec"] * (4.0 * n * (n + 1) / 2 + 4 * rsz * n), "flops": case["nvec"] * per}
    if family == "absorption":
        return _job_work(case["geometry"], case["ham"], n, case["frames"], case["t1"], case["sample"], case["prop"], 3)
    if family == "linear":
        return _job_work("cluster", "Full", n, case["frames"], case["t1"], case["sample"], case["prop"],
                         3 * n if case["tech"] == "CD" else 3)
    if family == "twodir":
        t1, t3, pairs = case["t1"], case["t1"], n * (n + 1) / 2
        frames = t1 + case["t2"] + t3 + (case["points"] - 1) * case["sample"]
        vectors = case["points"] * (9.0 + 9.0 * t1) * (t3 - 1) * 5
        if case["prop"] == "Coupling":
            flops = vectors * (12.0 * 0.95 * n * (n - 1) / 2 * n + 12.0 * pairs)
        else:  # the sub-step U F U^T of a symmetric F
            flops = vectors * (2 * 8.0 * n ** 3)
        per_frame = 4.0 * (n if case["ham"] == "Coupling" else n * (n + 1) / 2 + 3 * n)
        return {"bytes": frames * per_frame + 8.0 * 12 * t1 * t3, "flops": flops}
    if family == "adjoint":  # the model, its recomputation and the backward sweep (about three steps each)
        w = _job_work("chain", "Full", n, case["frames"], case["t1"], case["sample"], "Coupling", 3)
        return {"bytes": w["bytes"], "flops": 5 * w["flops"]}
    total = {"bytes": 0.0, "flops": 0.0}
    for spec, kw in _batch_jobs(case, 0):
        w = _job_work("lattice", "Coupling", spec.n_sites, case["frames"], case["t1"], case["sample"],
                      kw["Propagation"], 3)
        total = {k: total[k] + w[k] for k in total}
    return total


# ------------------------------------------------- the same in 64 bits
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _hamiltonians(spec, kw, records):
    """diagonals [frames, n] and couplings ([n, n], or [frames, n, n]) in double, shifted and cut as the frame readers do."""
    n = spec.n_sites
    lo, hi = (float(x) for x in (kw["MinFrequencies"].split()[0], kw["MaxFrequencies"].split()[0]))
    shift, cut = np.float32((lo + hi) / 2), np.float32(kw["Couplingcut"])
    rec = records[0].view(np.float32).reshape(spec.frames, -1)[:, 1:]
    iu = np.triu_indices(n)

    def square(packed):
        m = np.zeros(packed.shape[:-1] + (n, n))
        m[..., iu[0], iu[1]] = np.where(np.abs(packed) < cut, 0, packed)
        m = m + np.swapaxes(m, -1, -2)
        m[..., range(n), range(n)] = 0
        return m

    if spec.ham_type == synth.COUPLING:
        return rec - shift, square(records[2].view(np.float32)[1:])
    diagonal = rec[:, iu[0] == iu[1]]
    return diagonal - shift, square(rec)


def _dipoles(spec, records):
    """[frames or 1, 3, n] in double."""
    return records[1].view(np.float32).reshape(-1, 1 + 3 * spec.n_sites)[:, 1:].reshape(-1, 3, spec.n_sites).astype(float)


class _System:
    """A trajectory on the device in double, and one time step of each propagation scheme for vectors [points, n, k]."""

    def __init__(self, spec, kw, records):
        dev = _device()
        diagonal, coupling = _hamiltonians(spec, kw, records)
        self.n, self.cut = spec.n_sites, float(np.float32(kw["Couplingcut"]))
        self.diagonal = torch.as_tensor(diagonal.astype(float), device=dev)
        self.static = coupling.ndim == 2
        self.coupling = torch.as_tensor(coupling, device=dev)
        self.dipole = torch.as_tensor(_dipoles(spec, records), device=dev)
        self.f = float(kw["Timestep"]) * ANGULAR
        self.ts, self.prop = int(kw["Trotter"]), kw["Propagation"]
        strength = np.abs(coupling) if self.static else np.abs(coupling).max(axis=0)
        self.pairs = [(int(a), int(b)) for a, b in np.argwhere(np.triu(strength, 1) > self.cut)]

    def mu(self, frames):
        """[points, n, 3] at the given frames."""
        d = self.dipole[frames] if self.dipole.shape[0] > 1 else self.dipole[:1].expand(len(frames), -1, -1)
        return d.transpose(1, 2)

    def matvec(self, frames, x):
        """H x for complex vectors x, the Hamiltonian of each point's own frame."""
        d = self.diagonal[frames][:, :, None]
        if self.static:
            s, n, k = x.shape
            flat = torch.view_as_real(x.transpose(0, 1).reshape(n, -1)).reshape(n, -1)
            y = torch.view_as_complex((self.coupling @ flat).reshape(n, s * k, 2)).reshape(n, s, k).transpose(0, 1)
        else:
            j = self.coupling[frames]
            y = torch.complex(j @ x.real, j @ x.imag)
        return d * x + y

    def step(self, frames, x):
        if self.prop == "Coupling":
            return self.trotter(frames, x)
        return self.rk4(frames, x) if self.prop == "RK4" else self.exact(frames, x)

    def exact(self, frames, x, f=None):
        """exp(-i H f) x by its Taylor series."""
        f = self.f if f is None else f
        j = self.coupling if self.static else self.coupling[frames]
        norm = f * float(self.diagonal[frames].abs().max() + j.abs().sum(-1).max())
        parts = max(1, math.ceil(norm / 2))
        for _ in range(parts):
            term, total, k, size = x, x, 0, 1.0
            while size > 1e-18:
                k += 1
                term = self.matvec(frames, term) * (-1j * f / parts / k)
                total = total + term
                size *= norm / parts / k
            x = total
        return x

    def rk4(self, frames, x):
        g = self.f / self.ts
        for _ in range(self.ts):
            term, y = x, x
            for k in (1, 2, 3, 4):
                term = self.matvec(frames, term) * (-1j * g / k)
                y = y + term
            x = y * (torch.linalg.vector_norm(x, dim=1, keepdim=True) / torch.linalg.vector_norm(y, dim=1, keepdim=True))
        return x

    def trotter(self, frames, x):
        g = self.f / self.ts
        phase = torch.exp(-0.5j * g * self.diagonal[frames])[:, :, None]
        rows = list(x.unbind(1))
        half = list(phase.unbind(1))
        turns = []
        for a, b in self.pairs:
            j = self.coupling[a, b] if self.static else self.coupling[frames, a, b][:, None]
            j = torch.where(j.abs() > self.cut, j, 0.0)
            si = -torch.sin(j * g)
            turns.append((torch.sqrt(1 - si * si), 1j * si))
        for _ in range(self.ts):
            rows = [r * h for r, h in zip(rows, half)]
            for (a, b), (co, si) in zip(self.pairs, turns):
                rows[a], rows[b] = co * rows[a] + si * rows[b], co * rows[b] + si * rows[a]
            rows = [r * h for r, h in zip(rows, half)]
        return torch.stack(rows, 1)


def _axis(params):
    """(rows of the transform, frequencies) of a 1D spectrum (the frequencies with the rounding of the context's precision)."""
    fft = max(params.fft, params.tmax1)
    shift = np.float32((np.float32(params.min1) + np.float32(params.max1)) / 2)
    f32 = params.precision == nise.FP32
    rows, freq = [], []
    for i in list(range(fft // 2, fft)) + list(range(fft // 2)):
        num = fft - i if i >= fft // 2 else -i
        if f32:
            w = -(np.float32(num) / np.float32(params.deltat) / np.float32(LIGHT) / np.float32(fft) - shift)
        else:
            w = -(num / float(np.float32(params.deltat)) / LIGHT / fft - float(shift))
        if params.min1 < w < params.max1:
            rows.append(i)
            freq.append(float(w))
    return rows, np.array(freq)


def _spectrum(params, re, im, samples):
    """The rows of the spectrum of a response (swapped parts, lifetime, first point halved, transform)."""
    fft = max(params.fft, params.tmax1)
    t = np.arange(params.tmax1) * float(params.deltat)
    z = (im + 1j * re) / samples
    if params.lifetime > 0:
        z = z * np.exp(-t / (2 * params.lifetime))
    z[0] *= 0.5
    out = np.fft.fft(z, fft) * (2.0 * params.deltat * LIGHT)
    rows, freq = _axis(params)
    return freq, out.imag[rows], out.real[rows]


def _params(kw, case):
    return nise.params_from_keywords(kw, precision=_precision(case))


def _trotter_cost(pairs, n, t1, sub=5):
    return (pairs + 2 * n / 8) * sub * t1


def _exact_absorption(spec, kw, records, params):
    s = _System(spec, kw, records)
    if s.prop == "Coupling" and _trotter_cost(len(s.pairs), s.n, params.tmax1) > 200000:
        return None
    points = _points(spec.frames, params.tmax1, params.sample)
    start = torch.arange(points, device=s.diagonal.device) * params.sample
    x = s.mu(start).to(torch.complex128)
    response = []
    for t in range(params.tmax1):
        response.append((s.mu(start + t) * x).sum())
        if t + 1 < params.tmax1:
            x = s.step(start + t, x)
    z = torch.stack(response).cpu().numpy()
    return [z.real.copy(), z.imag.copy(), *_spectrum(params, z.real, z.imag, points), None]


def _exact_linear(case, spec, kw, records, params, seed):
    s = _System(spec, kw, records)
    if s.prop == "Coupling" and _trotter_cost(len(s.pairs), s.n, params.tmax1) > 200000:
        return None
    points, n, dev = _points(spec.frames, params.tmax1, params.sample), s.n, s.diagonal.device
    start = torch.arange(points, device=dev) * params.sample
    mu0 = s.mu(start)
    cd = case["tech"] == "CD"
    x = torch.eye(n, dtype=torch.complex128, device=dev).expand(points, n, n) if cd else mu0.to(torch.complex128)
    if cd:
        place = torch.as_tensor(_positions(case, seed)[:, 1:].reshape(-1, 3, n), device=dev)
    response = []
    for t in range(params.tmax1):
        mu = s.mu(start + t)
        if cd:
            total = 0
            for a in range(3):
                for b in range(3):
                    if a == b:
                        continue
                    c = 3 - a - b
                    sign = 1.0 if (b - a + 3) % 3 == 2 else -1.0
                    r = place[start + t, c]  # the operator is a product of single-precision operands
                    weight = sign * (r[:, :, None] - r[:, None, :]) * mu[:, :, b].float()[:, :, None]
                    total = total + (weight.double() * mu0[:, :, a][:, None, :] * x).sum()
            response.append(total)
        else:
            each = (mu * x).sum((0, 1))
            response.append(each[2] - 0.5 * each[0] - 0.5 * each[1])
        if t + 1 < params.tmax1:
            x = s.step(start + t, x)
    z = torch.stack(response).cpu().numpy()
    return [z.real[None].copy(), z.imag[None].copy(), *_spectrum(params, z.real, z.imag, points), None]


POLARISATIONS = ([(a, a, a, a) for a in range(3)] + [(a, a, b, b) for a in range(3) for b in range(3) if a != b]
                 + [(a, b, a, b) for a in range(3) for b in range(3) if a != b]
                 + [(a, b, b, a) for a in range(3) for b in range(3) if a != b])
WEIGHTS = np.array([[6.0] * 3 + [2.0] * 18, [2.0] * 3 + [4.0] * 6 + [-1.0] * 12,
                    [0.0] * 9 + [2.5] * 6 + [-2.5] * 6]) / 30


def _doubles_step(s, kw, frames, f, uv):
    """One time step of two-exciton states f[points, vectors, n, n] (symmetric, |aa> on the diagonal)."""
    n, g, root = s.n, s.f / s.ts, math.sqrt(2.0)
    dev = f.device
    anharmonicity = 0.0 if uv else float(kw["Anharmonicity"])
    eye = torch.eye(n, device=dev, dtype=torch.float64)
    if s.prop != "Coupling":
        half = torch.exp(0.5j * g * anharmonicity * eye)
        u = s.exact(frames, torch.eye(n, dtype=torch.complex128, device=dev).expand(len(frames), n, n), g)[:, None]
        scale = torch.ones((n, n), dtype=torch.float64, device=dev) + (root - 1) * eye
        for _ in range(s.ts):
            f = f * half
            if uv:  # |ab> pairs with a != b only
                f = f * (1 - eye)
                f = (u @ f @ u.transpose(-1, -2)) * (1 - eye)
            else:
                f = (u @ (f * scale) @ u.transpose(-1, -2)) / scale
            f = f * half
        return f
    d = s.diagonal[frames]
    phase = torch.exp(-0.5j * g * (d[:, :, None] + d[:, None, :] - anharmonicity * eye))[:, None]
    rows = [(a, b) for a in range(n) for b in range(a, n)]
    index = torch.zeros((n, n), dtype=torch.long)
    for e, (a, b) in enumerate(rows):
        index[a, b] = index[b, a] = e
    index = index.to(dev)
    ia, ib = torch.tensor(rows, device=dev).T
    x = f[:, :, ia, ib]
    phase = phase[:, :, ia, ib]
    turns = []
    for a, b in s.pairs:
        j = s.coupling[a, b].expand(len(frames)) if s.static else s.coupling[frames, a, b]
        j = torch.where(j.abs() > s.cut, j, 0.0)[:, None]
        pair = []
        for angle in (j * g, j * g * float(np.float32(1.41421356237))):
            si = -torch.sin(angle)
            pair.append((torch.sqrt(1 - si * si), 1j * si))
        turns.append(pair)

    def turn(co, si, p, q):
        return co * p + si * q, co * q + si * p

    for _ in range(s.ts):
        x = x * phase
        for (a, b), (plain, wide) in zip(s.pairs, turns):
            others = torch.tensor([c for c in range(n) if c not in (a, b)], dtype=torch.long, device=dev)
            p, q = index[a][others], index[b][others]
            x[:, :, p], x[:, :, q] = turn(plain[0][..., None], plain[1][..., None], x[:, :, p], x[:, :, q])
            if not uv:
                aa, ab, bb = index[a, a], index[a, b], index[b, b]
                x[:, :, aa], x[:, :, ab] = turn(*wide, x[:, :, aa].clone(), x[:, :, ab].clone())
                x[:, :, ab], x[:, :, bb] = turn(*wide, x[:, :, ab].clone(), x[:, :, bb].clone())
        x = x * phase
    return x[:, :, index.reshape(-1)].reshape(f.shape)


def _exact_twodir(case, spec, kw, records):
    s = _System(spec, kw, records)
    if s.n > 16 or _trotter_cost(len(s.pairs), s.n, case["t1"]) * (case["prop"] == "Coupling") > 40000:
        return None
    n, t1s, t2s, t3s, points = s.n, case["t1"], case["t2"], case["t1"], case["points"]
    uv = case["tech"].endswith("UVvis")
    dev = s.diagonal.device
    tj = torch.arange(points, device=dev) * case["sample"] + t1s
    tk = tj + t2s
    # left[t1] of every component: the vector that starts at tj - t1 joins the others there
    x = s.mu(tj - (t1s - 1)).to(torch.complex128)
    for t1 in range(t1s - 1, 0, -1):
        x = torch.cat([s.mu(tj - (t1 - 1)).to(x.dtype), s.step(tj - t1, x)], 2)
    left = x.reshape(points, n, t1s, 3).transpose(1, 2)  # [points, t1, n, 3]
    gb1 = torch.einsum("stia,sib->stab", left, s.mu(tj).to(left.dtype))
    vectors = torch.cat([s.mu(tj).to(left.dtype), left.permute(0, 2, 1, 3).reshape(points, n, -1)], 2)
    for t in range(t2s):
        vectors = s.exact(tj + t, vectors)
    mu2 = s.mu(tk)
    third = s.mu(tk).to(left.dtype)
    # two-exciton states mu2 x v for every second component and vector
    root = float(np.float32(1.41421356237))
    eye = torch.eye(n, dtype=torch.float64, device=dev)
    v = vectors.transpose(1, 2)  # [points, 3 + 3 t1, n]
    outer = torch.einsum("sib,svj->sbvij", mu2.to(v.dtype), v)
    doubles = outer + outer.transpose(-1, -2)
    doubles = doubles * (1 - eye) + (0 if uv else 1) * eye * outer * root
    nv = v.shape[1]
    doubles = doubles.reshape(points, 3 * nv, n, n)
    v0 = v
    lifetime = float(kw["Lifetime"])
    out = torch.zeros((12, t3s, t1s), dtype=torch.float64, device=dev)
    for t3 in range(t3s):
        mu3 = s.mu(tk + t3)
        gb3 = torch.einsum("sia,sib->sab", third, mu3.to(third.dtype))
        vt = vectors.transpose(1, 2)
        at2 = torch.einsum("svi,sia->sva", v0, mu2.to(v0.dtype))
        at3 = torch.einsum("svi,sia->sva", vt, mu3.to(vt.dtype))
        g = torch.einsum("svij,sic->svcj", doubles * (1 - eye), mu3.to(v0.dtype))
        if not uv:
            g = g + root * torch.einsum("svjj,sjc->svcj", doubles, mu3.to(v0.dtype))
        g = g.reshape(points, 3, nv, 3, n)
        lw = torch.exp(-(torch.arange(t1s, device=dev) + t3) * float(kw["Timestep"]) / (2 * lifetime)) if lifetime > 0 else 1
        for m, (p0, p1, p2, p3) in enumerate(POLARISATIONS):
            left0 = slice(3 + p0, None, 3)
            # ground-state bleach
            a, b = gb1[:, :, p0, p1], gb3[:, p2, p3][:, None]
            one = -b * a.conj()
            two = -b * a
            # stimulated emission
            one = one - at3[:, p1, p3][:, None] * at2[:, left0, p2].conj()
            two = two - at2[:, p1, p2].conj()[:, None] * at3[:, left0, p3]
            # excited-state absorption
            one = one + torch.einsum("si,sti->st", g[:, p2, p1, p3], vt[:, left0].conj())
            two = two + torch.einsum("sti,si->st", g[:, p2, left0, p3], vt[:, p1].conj())
            for q in range(3):
                w = float(WEIGHTS[q, m]) * lw
                out[4 * q, t3] += w * one.imag.sum(0)
                out[4 * q + 1, t3] += w * one.real.sum(0)
                out[4 * q + 2, t3] += w * two.imag.sum(0)
                out[4 * q + 3, t3] += w * two.real.sum(0)
        if t3 + 1 < t3s:
            doubles = _doubles_step(s, kw, tk + t3, doubles, uv)
            vectors = s.step(tk + t3, vectors)
            third = s.step(tk + t3, third)
    return [out.cpu().numpy(), None]


def _exact_adjoint(case, seed):
    spec, kw = _adjoint_setup(case, seed)
    params = nise.params_from_keywords(kw, precision=nise.FP64)
    s = _System(spec, kw, _records(spec))
    if _trotter_cost(len(s.pairs), s.n, params.tmax1) > 25000:
        return None
    rows, freq = _axis(params)
    shift, dre, dim = _adjoint_inputs(case, seed, len(rows))
    dev = s.diagonal.device
    shift = torch.tensor(shift, device=dev, requires_grad=True)
    scale = torch.tensor(FIT_SCALE, dtype=torch.float64, device=dev, requires_grad=True)
    lifetime = torch.tensor(FIT_LIFETIME, dtype=torch.float64, device=dev, requires_grad=True)
    s.diagonal = s.diagonal + shift
    s.coupling, s.cut = s.coupling * scale, 0.0
    points = _points(spec.frames, params.tmax1, params.sample)
    start = torch.arange(points, device=dev) * params.sample
    x = s.mu(start).to(torch.complex128)
    response = []
    for t in range(params.tmax1):
        response.append((s.mu(start + t) * x).sum())
        if t + 1 < params.tmax1:
            x = s.step(start + t, x)
    z = torch.stack(response)
    t = torch.arange(params.tmax1, device=dev) * float(params.deltat)
    z = torch.complex(z.imag, z.real) / points * torch.exp(-t / (2 * lifetime))
    z = torch.cat([z[:1] * 0.5, z[1:]])
    out = torch.fft.fft(z, max(params.fft, params.tmax1)) * (2.0 * params.deltat * LIGHT)
    sr, si = out.imag[rows], out.real[rows]
    loss = (sr * torch.as_tensor(dre, device=dev)).sum() + (si * torch.as_tensor(dim, device=dev)).sum()
    loss.backward()
    return [freq, sr.detach().cpu().numpy(), si.detach().cpu().numpy(), shift.grad.cpu().numpy(), float(scale.grad),
            float(lifetime.grad)]


def _exact_step(case, seed):
    h, re, im = _step_inputs(case, seed)
    n, nvec = case["n"], case["nvec"]
    kw = synth.c0_keywords(Singles=n, Propagation=case["prop"], Threshold=0)
    s = _System.__new__(_System)
    iu = np.triu_indices(n)
    m = np.zeros((nvec, n, n))
    m[:, iu[0], iu[1]] = h
    m = m + np.swapaxes(m, 1, 2)
    diagonal = m[:, range(n), range(n)] / 2
    m[:, range(n), range(n)] = 0
    s.n, s.cut, s.static = n, float(np.float32(kw["Couplingcut"])), False
    if case["prop"] == "RK4":
        m[np.abs(m) <= s.cut] = 0
    s.diagonal, s.coupling = torch.as_tensor(diagonal), torch.as_tensor(m)
    s.f, s.ts, s.prop = float(kw["Timestep"]) * ANGULAR, int(kw["Trotter"]), case["prop"]
    s.pairs = [(a, b) for a in range(n) for b in range(a + 1, n)]
    x = torch.complex(torch.as_tensor(re.astype(float)), torch.as_tensor(im.astype(float)))[:, :, None]
    y = s.step(torch.arange(nvec), x)[:, :, 0]
    return y.real.numpy().copy(), y.imag.numpy().copy()


def exact(case, seed):
    family = case["family"]
    if family == "step":
        return _exact_step(case, seed)
    if family == "absorption":
        spec, kw = _absorption_setup(case, seed)
        return _exact_absorption(spec, kw, _records(spec), _params(kw, case))
    if family == "linear":
        spec, kw = _linear_setup(case, seed)
        return _exact_linear(case, spec, kw, _records(spec), _params(kw, case), seed)
    if family == "twodir":
        spec, kw = _twodir_setup(case, seed)
        return _exact_twodir(case, spec, kw, _records(spec))
    if family == "adjoint":
        return _exact_adjoint(case, seed)
    # the Trotter jobs of a batch have thousands of rotations in sequence: no values for those
    out = []
    for spec, kw in _batch_jobs(case, seed):
        params = nise.params_from_keywords(kw)
        value = _exact_absorption(spec, kw, _records(spec), params) if kw["Propagation"] == "Diagonal" else None
        out.append(value or [None] * 6)
    return out
