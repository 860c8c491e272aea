"""The work that programs have this package do, as measured cases.

Every case is one of seven kinds, each a call (or the few calls a program makes
together) of the public interface, over the sizes of the package's own
configurations, tests and benchmark:

``drop_in``     ``simulation_gpu.compute`` on a sheet: host inputs in, the
                histories out (plain FP64, or FP32 with the early exit)
``job``         a batch of shells through ``BatchedEngine``: the instances are
                added, advanced to their last step in a few launches, their
                histories gathered into the caller's order, and removed (what
                the server does with every request it admits)
``egm_fp64``    lead field of a new geometry, FP64 contraction with a Vm
                history, normalisation (the plain electrogram), on the device
``egm_bf16x3``  split of a new FP32 history, tensor-core contraction with a
                lead field kept in split form, normalisation
``electrodes``  electrode activation times and conduction velocity of a signal
``activation``  every activation of every voxel of an FP32 history
``lattice``     neighbour table and row order of a new geometry
"""
import ctypes
import functools
import math

import numpy as np
import torch

from pyheartsim_b200 import _lib, analysis, geometry_gpu, synthetic
from pyheartsim_b200.engine import BatchedEngine
from pyheartsim_b200.simulation import simulation_gpu, unipolar_electrogram_gpu

DELTA = 0.4                          # mm, the lattice constant of every configuration
DT_PHYS = {0: 0.05, 1: 0.02}         # ms, Mitchell-Schaeffer and Aliev-Panfilov
FOCAL = {0: (3, 2.0), 1: (8, 5.0)}   # focal stimulus: ball radius in voxels, duration in ms
LAUNCH_STEPS = 50                    # steps per launch of a job (the server's setting)
RADIUS_MM = 8.0                      # conduction velocity's neighbourhood


def listed():
    return [
        # the smallest call: a test-sized sheet through the drop-in, plain FP64; launches, barriers and host work count
        {"name": "sheet 40x40 plain fp64", "kind": "drop_in", "nx": 40, "ny": 40, "model": 0, "fast": False,
         "steps": 100},
        # the plain sheet configuration (200 x 200, corner stimulus) as the reference runs it
        {"name": "sheet 200x200 plain fp64", "kind": "drop_in", "nx": 200, "ny": 200, "model": 0, "fast": False,
         "steps": 60},
        # the same sheet in the fast form
        {"name": "sheet 200x200 fast fp32", "kind": "drop_in", "nx": 200, "ny": 200, "model": 0, "fast": True,
         "steps": 200},
        # the rotor shell (25/20/18 mm, wall 3), one Aliev-Panfilov instance alone on the GPU
        {"name": "rotor shell fast fp32", "kind": "job", "geometry": 1, "count": 1, "n_min": 91000, "n_max": 91001,
         "models": "ap", "fast": True, "fibres": False, "steps": 300},
        # the batched configuration: uneven scarred shells of both models
        {"name": "24 shells fast fp32", "kind": "job", "geometry": 2, "count": 24, "n_min": 50000, "n_max": 400000,
         "models": "mixed", "fast": True, "fibres": False, "steps": 300},
        # shells with a fibre field (anisotropic diffusion, edge terms)
        {"name": "4 fibre shells fast fp32", "kind": "job", "geometry": 3, "count": 4, "n_min": 60000,
         "n_max": 240000, "models": "mixed", "fast": True, "fibres": True, "steps": 300},
        # the median shell of the batch in the plain form
        {"name": "shell 157k plain fp64", "kind": "job", "geometry": 4, "count": 1, "n_min": 157000,
         "n_max": 157001, "models": "ms", "fast": False, "fibres": False, "steps": 30},
        # the rotor shell's electrogram: 64 electrodes, 1000 samples, plain FP64
        {"name": "electrogram fp64 91k x 64", "kind": "egm_fp64", "geometry": 1, "n": 91000, "n_e": 64, "T": 1000,
         "fibres": False},
        # the full electrogram: 2048 electrodes over half a million voxels
        {"name": "electrogram bf16x3 520k x 2048", "kind": "egm_bf16x3", "geometry": 5, "n": 520000, "n_e": 2048,
         "T": 1000},
        # analysis of a dense electrode array's signals
        {"name": "electrodes 2048 x 1000", "kind": "electrodes", "geometry": 5, "n_e": 2048, "T": 1000, "f64": True},
        # re-entry analysis of the rotor shell's 1 kHz history
        {"name": "activations 91k x 1000", "kind": "activation", "geometry": 1, "n": 91000, "S": 1000},
        # geometry preparation of the largest served request
        {"name": "lattice 1M", "kind": "lattice", "geometry": 6, "n": 1000000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["drop_in", "drop_in", "job", "job", "job", "egm_fp64", "egm_bf16x3", "electrodes",
                       "activation", "lattice"])
    geometry = rng.randrange(10, 10000)
    if kind == "drop_in":
        fast = rng.random() < 0.5
        return {"kind": kind, "nx": _log(rng, 30, 220), "ny": _log(rng, 30, 220), "model": rng.randrange(2),
                "fast": fast, "steps": rng.randrange(60, 200) if fast else rng.randrange(20, 60)}
    if kind == "job":
        fast = rng.random() < 0.75
        lo = _log(rng, 20000, 200000)
        return {"kind": kind, "geometry": geometry, "count": _log(rng, 1, 10) if fast else 1, "n_min": lo,
                "n_max": min(400000, int(lo * rng.uniform(1.0, 4.0)) + 1),
                "models": rng.choice(["ms", "ap", "mixed"]), "fast": fast, "fibres": rng.random() < 0.25,
                "steps": rng.randrange(100, 300) if fast else rng.randrange(10, 25)}
    if kind == "egm_fp64":
        return {"kind": kind, "geometry": geometry, "n": _log(rng, 20000, 200000), "n_e": _log(rng, 16, 256),
                "T": _log(rng, 100, 1000), "fibres": rng.random() < 0.5}
    if kind == "egm_bf16x3":
        return {"kind": kind, "geometry": geometry, "n": _log(rng, 40000, 500000), "n_e": _log(rng, 64, 2048),
                "T": _log(rng, 100, 1000)}
    if kind == "electrodes":
        return {"kind": kind, "geometry": geometry, "n_e": _log(rng, 64, 2048), "T": _log(rng, 200, 2000),
                "f64": rng.random() < 0.5}
    if kind == "activation":
        return {"kind": kind, "geometry": geometry, "n": _log(rng, 20000, 400000), "S": _log(rng, 200, 1000)}
    return {"kind": kind, "geometry": geometry, "n": _log(rng, 50000, 1000000)}


# ------------------------------------------------------------------ geometry
@functools.lru_cache(maxsize=64)
def _shell(n_target, geometry):
    """Integer coordinates (n, 3), ordered z, y, x, of an ellipsoidal shell
    (semi-axes in the ratio 25:20:18, wall of 3 voxels, four vein holes) of
    about ``n_target`` voxels; made on the GPU, kept on the host."""
    base = torch.tensor([25.0, 20.0, 18.0], dtype=torch.float64)
    rng = np.random.default_rng(geometry)
    dirs = rng.standard_normal((4, 3))
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    s = math.sqrt(n_target / 91000.0)
    a = (base * s).tolist()
    ax = [torch.arange(-math.ceil(v / DELTA) - 1, math.ceil(v / DELTA) + 2, device="cuda") for v in a]
    z, y, x = (g.double() * DELTA for g in torch.meshgrid(ax[2], ax[1], ax[0], indexing="ij"))
    r = ((x / a[0]) ** 2 + (y / a[1]) ** 2 + (z / a[2]) ** 2).sqrt()
    grad = ((x / a[0] ** 2) ** 2 + (y / a[1] ** 2) ** 2 + (z / a[2] ** 2) ** 2).sqrt()
    keep = (r <= 1.0) & ((1.0 - r) * r / grad.clamp(min=1e-12) < 3 * DELTA)
    for d in dirs:
        proj = x * d[0] + y * d[1] + z * d[2]
        perp2 = x * x + y * y + z * z - proj * proj
        keep &= ~((perp2 < (5.0 * s) ** 2) & (proj > 0))
    k, j, i = torch.nonzero(keep, as_tuple=True)
    return torch.stack([ax[0][i], ax[1][j], ax[2][k]], dim=1).cpu().numpy().astype(np.int64)


def _occupancy(ijk):
    """(dense grid of voxel ids with one empty cell of padding, grid coordinates)."""
    t = torch.as_tensor(ijk, device="cuda")
    g = t - t.min(dim=0).values + 1
    dims = (g.max(dim=0).values + 2).tolist()
    grid = torch.full(dims, -1, dtype=torch.int64, device="cuda")
    grid[g[:, 0], g[:, 1], g[:, 2]] = torch.arange(t.shape[0], device="cuda")
    return grid, g


_OFFSETS = ((1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0), (1, -1, 0),
            (-1, -1, 0), (0, 1, 1), (0, -1, 1), (0, 1, -1), (0, -1, -1), (1, 0, 1), (-1, 0, 1), (1, 0, -1), (-1, 0, -1))


def _neighbours(ijk, count):
    grid, g = _occupancy(ijk)
    return torch.stack([grid[g[:, 0] + o[0], g[:, 1] + o[1], g[:, 2] + o[2]] for o in _OFFSETS[:count]], dim=1)


def _scar(ijk, rng):
    """Conductivity scale: Gaussian-blob scar over up to 30 % of the voxels (0
    inside, 0.1 on the ring around it, 1 elsewhere)."""
    n = ijk.shape[0]
    t = torch.as_tensor(ijk, device="cuda").double()
    f = torch.zeros(n, dtype=torch.float64, device="cuda")
    for c in ijk[rng.integers(0, n, size=6)]:
        f += torch.exp(-((t - torch.as_tensor(c, device="cuda")) ** 2).sum(1) / 128.0)
    core = f >= torch.sort(f).values[min(n - 1, int((1.0 - rng.uniform(0.02, 0.3)) * n))]
    nb = _neighbours(ijk, 6)
    ring = (core[nb.clamp(min=0)] & (nb >= 0)).any(dim=1) & ~core
    return torch.where(core, 0.0, torch.where(ring, 0.1, 1.0)).double().cpu().numpy()


# ------------------------------------------------------------------ simulations
def _shells(case):
    """Geometry and model of each instance of a job."""
    rng = np.random.default_rng(case["geometry"])
    out = []
    for i in range(case["count"]):
        n = int(math.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]))))
        model = {"ms": 0, "ap": 1, "mixed": i % 2}[case["models"]]
        out.append((_shell(n, case["geometry"] * 100 + i), model))
    return out


def _job_inputs(case, seed):
    """Per instance: coordinates, conductivity scale, tensors, pacing sets."""
    for i, (ijk, model) in enumerate(_shells(case)):
        rng = np.random.default_rng([seed, i])
        scale = _scar(ijk, rng)
        radius, ms = FOCAL[model]
        healthy = np.flatnonzero(scale == 1.0)
        centre = ijk[healthy[rng.integers(0, healthy.size)]]
        s1 = np.flatnonzero(((ijk - centre) ** 2).sum(axis=1) <= radius * radius)
        # S2 on one side of the site, early enough to fall into the run
        s2 = np.flatnonzero(((ijk - centre - radius - 4) ** 2).sum(axis=1) <= radius * radius)
        flag = 1 if s2.size else 4
        dt = DT_PHYS[model]
        t_phys = case["steps"] * dt
        D0 = synthetic.fibre_tensors(ijk) if case["fibres"] else None
        sp, ap, par = synthetic.case_parameters(ijk.shape[0], model, dt, t_phys, s1, s2_ids=s2, flag=flag,
                                                s1_s2=0.4 * t_phys, c_scale=scale)
        yield dict(ijk=ijk, model=model, D0=D0, sp=sp, ap=ap, par=par, pacing=ms / sp["time_scale"],
                   s1=s1, s2=s2 if flag == 1 else np.zeros(0, np.int64))


def _sheet_inputs(case, seed):
    rng = np.random.default_rng(seed)
    ijk = synthetic.sheet(case["nx"], case["ny"])
    dt = DT_PHYS[case["model"]]
    x0, y0 = rng.integers(0, case["nx"] - 8), rng.integers(0, case["ny"] - 8)
    w = 5 if case["model"] == 0 else 8
    s1 = np.flatnonzero((ijk[:, 0] >= x0) & (ijk[:, 0] < x0 + w) & (ijk[:, 1] >= y0) & (ijk[:, 1] < y0 + w))
    scale = rng.uniform(0.8, 1.2, size=ijk.shape[0])
    sp, ap, par = synthetic.case_parameters(ijk.shape[0], case["model"], dt, case["steps"] * dt, s1, flag=4,
                                            c_scale=scale)
    pacing = (1.0 if case["model"] == 0 else 5.0) / sp["time_scale"]
    return dict(ijk=ijk, model=case["model"], D0=None, sp=sp, ap=ap, par=par, pacing=pacing, s1=s1,
                s2=np.zeros(0, np.int64))


class _State:
    def __init__(self, **kw):
        self.__dict__.update(kw)


def _p(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _prepare_drop_in(case, seed):
    d = _sheet_inputs(case, seed)
    n = d["ijk"].shape[0]
    nb = geometry_gpu.find_neighbor_voxel_ids(d["ijk"])
    P = geometry_gpu.heart_model_equation_parts(d["sp"], n, None, nb, d["par"])
    geom = {"neighbor_id_2d": nb, "Delta": DELTA, "voxel": d["ijk"] * DELTA}
    kw = dict(dtype=np.float32, fast=True, tol=1e-7) if case["fast"] else {}
    return _State(case=case, args=(n, P, geom, d["sp"], d["ap"]), kw=dict(kw, pacing_duration=d["pacing"]))


def _run_drop_in(s):
    return simulation_gpu.compute(*s.args, **s.kw)


def _prepare_job(case, seed):
    kw = dict(full_cycles=False, tol=1e-7, restart=20) if case["fast"] else dict(full_cycles=True, tol=1e-5, restart=50)
    insts = [geometry_gpu.compile_instance(d["ijk"] * DELTA, DELTA, d["par"], d["D0"], d["sp"], d["ap"], atol=1e-5,
                                           save_h=False, pacing_duration=d["pacing"], **kw)
             for d in _job_inputs(case, seed)]
    return _State(case=case, insts=insts, engine=BatchedEngine(_lib.PREC_F32 if case["fast"] else _lib.PREC_F64))


def _run_job(s):
    eng = s.engine
    stream = torch.cuda.current_stream()
    slots = [eng.add(x) for x in s.insts]
    for _ in range(-(-s.case["steps"] // LAUNCH_STEPS)):
        eng.advance(LAUNCH_STEPS, stream=stream, sync=True)
    out = [eng.history_device(k) for k in slots]
    for k in slots:
        eng.remove(k)
    return out


# ------------------------------------------------------------------ electrograms
def _wave(xyz, T, rng, dtype):
    """(T, n) Vm of a wave from a seeded site: upstroke of about 1 ms, plateau, recovery."""
    site = xyz[int(rng.integers(0, xyz.shape[0]))]
    at = (xyz - site).norm(dim=1) / 0.5 + 5.0
    dur = float(rng.uniform(120.0, 200.0))
    V = torch.empty((T, xyz.shape[0]), dtype=dtype, device="cuda")
    for t in range(T):
        V[t] = (torch.sigmoid((t - at) / 0.7) * (1.0 - torch.sigmoid((t - at - dur) / 12.0))).to(dtype)
    return V


def _egm_inputs(case, seed):
    ijk = _shell(case["n"], case["geometry"])
    rng = np.random.default_rng(seed)
    xyz = torch.as_tensor(ijk * DELTA, device="cuda")
    exyz = torch.as_tensor(synthetic.electrodes_off_surface(ijk, DELTA, case["n_e"], rng), device="cuda")
    c = torch.as_tensor(_scar(ijk, rng), device="cuda")
    D0 = None
    if case.get("fibres"):
        D0 = torch.as_tensor(synthetic.fibre_tensors(ijk).reshape(-1, 9), device="cuda")
    V = _wave(xyz, case["T"], rng, torch.float64 if case["kind"] == "egm_fp64" else torch.float32)
    return ijk, xyz, exyz, c, D0, V


@functools.lru_cache(maxsize=8)
def _gradient_terms(n, geometry):
    nb, _ = geometry_gpu.lattice_neighbors(_shell(n, geometry), order=False)
    return unipolar_electrogram_gpu.incoming_gradient_terms(nb.cpu().numpy())


def _leadfield(s):
    _lib.check(_lib.lib().phs_egm_leadfield_f64(s.n, s.n_e, _p(s.xyz), _p(s.exyz), _p(s.c), _p(s.D0), _p(s.ptr),
                                                _p(s.src), _p(s.dirs), 1.0 / (2.0 * DELTA), _p(s.Mt), _stream()),
               "phs_egm_leadfield_f64")


def _prepare_egm(case, seed):
    ijk, xyz, exyz, c, D0, V = _egm_inputs(case, seed)
    s = _State(case=case, n=ijk.shape[0], n_e=case["n_e"], T=case["T"], xyz=xyz, exyz=exyz, c=c, D0=D0, V=V)
    s.ptr, s.src, s.dirs = (torch.as_tensor(a, device="cuda") for a in _gradient_terms(case["n"], case["geometry"]))
    s.Mt = torch.empty((s.n_e, s.n), dtype=torch.float64, device="cuda")
    s.egm = torch.empty((s.T, s.n_e), dtype=V.dtype, device="cuda")
    if case["kind"] == "egm_bf16x3":
        # the lead field belongs to the geometry and the electrodes: built and split once
        s.Tp, s.Ep, s.Kp = -(-s.T // 128) * 128, -(-s.n_e // 128) * 128, -(-s.n // 64) * 64
        u16 = dict(dtype=torch.uint16, device="cuda")
        s.vh, s.vl = torch.empty((s.Tp, s.Kp), **u16), torch.empty((s.Tp, s.Kp), **u16)
        s.mh, s.ml = torch.empty((s.Ep, s.Kp), **u16), torch.empty((s.Ep, s.Kp), **u16)
        _leadfield(s)
        _lib.check(_lib.lib().phs_split_bf16(s.n_e, s.n, _p(s.Mt), s.n, 1, _p(s.mh), _p(s.ml), s.Ep, s.Kp,
                                             _stream()), "phs_split_bf16")
        s.Mt = None
        s.work = torch.empty(_lib.lib().phs_egm_bf16x3_workspace(s.Tp, s.Ep, s.Kp), dtype=torch.uint8, device="cuda")
    return s


def _run_egm_fp64(s):
    _leadfield(s)
    _lib.check(_lib.lib().phs_egm_contract_f64(s.T, s.n, s.n_e, _p(s.V), s.n, _p(s.Mt), _p(s.egm), _stream()),
               "phs_egm_contract_f64")
    _lib.check(_lib.lib().phs_egm_normalize(s.T, s.n_e, _p(s.egm), 1, _stream()), "phs_egm_normalize")
    return s.egm


def _run_egm_bf16x3(s):
    L = _lib.lib()
    _lib.check(L.phs_split_bf16(s.T, s.n, _p(s.V), s.n, 0, _p(s.vh), _p(s.vl), s.Tp, s.Kp, _stream()),
               "phs_split_bf16")
    _lib.check(L.phs_egm_contract_bf16x3(s.T, s.n_e, s.Tp, s.Ep, s.Kp, _p(s.vh), _p(s.vl), _p(s.mh), _p(s.ml),
                                         _p(s.egm), _p(s.work), _stream()), "phs_egm_contract_bf16x3")
    _lib.check(L.phs_egm_normalize(s.T, s.n_e, _p(s.egm), 0, _stream()), "phs_egm_normalize")
    return s.egm


# ------------------------------------------------------------------ analysis and geometry
def _electrode_inputs(case, seed):
    """Electrodes 2 mm off the rotor shell and their signals: a downstroke as a
    wave passes, over low noise."""
    rng = np.random.default_rng(seed)
    ijk = _shell(91000, case["geometry"])
    xyz = synthetic.electrodes_off_surface(ijk, DELTA, case["n_e"], rng)
    site = xyz[int(rng.integers(0, xyz.shape[0]))]
    at = np.linalg.norm(xyz - site, axis=1) / 0.4 * (case["T"] / 1000.0) + 20.0
    t = torch.arange(case["T"], dtype=torch.float64, device="cuda")[:, None]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    d = (t - torch.as_tensor(at, device="cuda")[None]) / 4.0
    sig = -d * torch.exp(-d * d) + 0.01 * torch.randn(d.shape, generator=gen, dtype=torch.float64, device="cuda")
    return xyz, sig if case["f64"] else sig.float()


def _prepare_electrodes(case, seed):
    xyz, sig = _electrode_inputs(case, seed)
    return _State(case=case, xyz=xyz, sig=sig)


def _run_electrodes(s):
    lat = analysis.electrode_lat_device(s.sig)
    vec, mag, mean = analysis.conduction_velocity(s.xyz, lat)
    return lat, vec, mag, mean


def _prepare_activation(case, seed):
    """An FP32 history of waves that pass every voxel again and again."""
    rng = np.random.default_rng(seed)
    xyz = torch.as_tensor(_shell(case["n"], case["geometry"]) * DELTA, device="cuda")
    site = xyz[int(rng.integers(0, xyz.shape[0]))]
    at = (xyz - site).norm(dim=1) / 0.5
    cycle = float(rng.uniform(140.0, 220.0))
    hist = torch.empty((case["S"], xyz.shape[0]), dtype=torch.float32, device="cuda")
    for t in range(case["S"]):
        ph = torch.remainder(t - at, cycle)
        hist[t] = (torch.where(t >= at, 1.0, 0.0) * (torch.tanh(ph) - torch.sigmoid((ph - 90.0) / 8.0))).float()
    n = xyz.shape[0]
    return _State(case=case, hist=hist, n=n, times=torch.full((n, 16), -1, dtype=torch.int32, device="cuda"),
                  counts=torch.zeros(n, dtype=torch.int32, device="cuda"))


def _run_activation(s):
    _lib.check(_lib.lib().phs_activation_times(s.case["S"], s.n, _p(s.hist), s.n, 0, 0.5, 16, _p(s.times),
                                               _p(s.counts), _stream()), "phs_activation_times")
    return s.times, s.counts


def _prepare_lattice(case, seed):
    """A shell's voxels in a seeded order."""
    ijk = torch.as_tensor(_shell(case["n"], case["geometry"]), device="cuda").to(torch.int32)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    # as a voxeliser leaves them: runs of the lattice order, the runs in any order
    runs = -(-ijk.shape[0] // 64)
    start = torch.randperm(runs, generator=gen, device="cuda")[:, None] * 64
    at = (start + torch.arange(64, device="cuda")[None]).reshape(-1)
    return _State(case=case, ijk=ijk[at[at < ijk.shape[0]]].contiguous())


def _run_lattice(s):
    return geometry_gpu.lattice_neighbors(s.ijk)


_PREPARE = {"drop_in": _prepare_drop_in, "job": _prepare_job, "egm_fp64": _prepare_egm, "egm_bf16x3": _prepare_egm,
            "electrodes": _prepare_electrodes, "activation": _prepare_activation, "lattice": _prepare_lattice}
_RUN = {"drop_in": _run_drop_in, "job": _run_job, "egm_fp64": _run_egm_fp64, "egm_bf16x3": _run_egm_bf16x3,
        "electrodes": _run_electrodes, "activation": _run_activation, "lattice": _run_lattice}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state.case["kind"]](state)


# ------------------------------------------------------------------ what a pass cannot do without
def _samples(steps, model):
    """(samples kept, steps between them): 1 kHz."""
    ts = 1 if model == 0 else 6
    dt = DT_PHYS[model] / ts
    t_final = steps * DT_PHYS[model] / ts
    n_steps, stride = int(np.round(t_final / dt)), int(1 / (dt * ts))
    return min(int(np.round(t_final * ts)), -(-n_steps // stride)), stride


def work(case):
    """Simulations: the per-voxel tables (six neighbours, coefficient, flags) in
    once, the state (two values) in and out every step, every history sample
    out; a step costs four evaluations of the reaction and one application of
    the seven-point operator.  The others: inputs in once, results out once."""
    kind = case["kind"]
    if kind in ("drop_in", "job"):
        size = 4 if case["fast"] else 8
        if kind == "drop_in":
            parts = [(case["nx"] * case["ny"], case["model"])]
        else:
            parts = [(ijk.shape[0], model) for ijk, model in _shells(case)]
        total, flops = 0.0, 0.0
        for n, model in parts:
            hist = _samples(case["steps"], model)[0] * size * (2 if kind == "drop_in" else 1)
            tables = 24 + size + 2 + ((48 + 12 * size) if case.get("fibres") else 0)
            total += n * (tables + 4.0 * size * case["steps"] + hist)
            flops += n * case["steps"] * (4 * 18 + 20 + (24 if case.get("fibres") else 0))
        return {"bytes": total, "flops": flops}
    if kind in ("egm_fp64", "egm_bf16x3"):
        n = _shell(case["n"], case["geometry"]).shape[0]
        T, n_e = case["T"], case["n_e"]
        if kind == "egm_fp64":
            terms = 6.0 * n
            by = 8.0 * T * n + n * (24 + 8 + (72 if case["fibres"] else 0)) + terms * 5 + 24.0 * n_e + 8.0 * T * n_e
            return {"bytes": by, "flops": 2.0 * T * n * n_e + 20.0 * n * n_e}
        return {"bytes": 4.0 * T * n + 4.0 * n_e * n + 4.0 * T * n_e, "flops": 6.0 * T * n * n_e}
    if kind == "electrodes":
        return {"bytes": (8.0 if case["f64"] else 4.0) * case["T"] * case["n_e"] + (24 + 4 + 32) * case["n_e"],
                "flops": 1.0 * case["T"] * case["n_e"] + 9.0 * case["n_e"] ** 2}
    n = _shell(case["n"], case["geometry"]).shape[0]
    if kind == "activation":
        return {"bytes": n * (4.0 * case["S"] + 4 * 16 + 4), "flops": 1.0 * n * case["S"]}
    return {"bytes": n * (12.0 + 72 + 4), "flops": 18.0 * n}


# ------------------------------------------------------------------ the same in 64 bits, plain torch and numpy
class _Operator:
    """L of an instance: face coefficients (cross terms folded in) and edge pairs."""

    def __init__(self, ijk, c, D0):
        aniso = D0 is not None
        nb = _neighbours(ijk, 18 if aniso else 6)
        have = nb >= 0
        self.nb = nb.clamp(min=0)
        n = nb.shape[0]
        scale = (c / (4 * DELTA ** 2))[:, None]
        D = torch.as_tensor(D0, device="cuda") if aniso else torch.eye(3, device="cuda").double().expand(n, 3, 3)
        d = have.double()
        P = torch.stack([4 * d[:, k] * D[:, k // 2, k // 2] for k in range(6)], dim=1)
        self.pairs = None
        if aniso:
            both = [d[:, 2 * i] * d[:, 2 * i + 1] for i in range(3)]
            for col in range(3):
                cross = sum(both[i] * (D[self.nb[:, 2 * i], i, col] - D[self.nb[:, 2 * i + 1], i, col])
                            for i in range(3))
                P[:, 2 * col] += both[col] * cross
                P[:, 2 * col + 1] -= both[col] * cross
            pairs = ((6, 8, 0, 1), (9, 7, 0, 1), (14, 16, 0, 2), (17, 15, 0, 2), (10, 12, 1, 2), (13, 11, 1, 2))
            need = ((6, 8), (7, 9), (14, 16), (15, 17), (10, 12), (11, 13))
            self.ecf = scale * torch.stack([2 * d[:, a] * d[:, b] * D[:, p[2], p[3]]
                                            for (a, b), p in zip(need, pairs)], dim=1)
            self.pairs = [(self.nb[:, p[0]], self.nb[:, p[1]]) for p in pairs]
        self.faces = self.nb[:, :6].contiguous()
        self.coef = scale * P
        self.bound = float(self.coef.abs().sum(dim=1).max())
        if aniso:
            self.bound += float(self.ecf.abs().sum(dim=1).max())

    def __call__(self, u):
        y = (self.coef * (u[self.faces] - u[:, None])).sum(dim=1)
        if self.pairs is not None:
            for k, (a, b) in enumerate(self.pairs):
                y += self.ecf[:, k] * (u[a] - u[b])
        return y


def _solve(L, h, b, x):
    """(I - h L) x = b by Chebyshev iteration to rounding level."""
    lo, hi = 1.0, 1.0 + 2.0 * h * L.bound
    mid, rad = (hi + lo) / 2, (hi - lo) / 2
    r = b - (x - h * L(x))
    goal = 4e-15 * float(b.norm()) + 1e-300
    d, alpha = None, 0.0
    for k in range(400):
        if k % 6 == 5 and float(r.norm()) <= goal:
            break
        beta = 0.0 if k == 0 else (0.5 * (rad * alpha) ** 2 if k == 1 else (rad * alpha / 2) ** 2)
        alpha = 1.0 / mid if k == 0 else 1.0 / (mid - beta / alpha)
        d = r.clone() if d is None else r + beta * d
        x = x + alpha * d
        r = b - (x - h * L(x))
    return x


def _reaction(model, u, h, J, p):
    if model == 0:
        du = h * u * u * (1 - u) / p["tau_in"] - u / p["tau_out"] + J
        return du, torch.where(u < p["v_gate"], (1 - h) / p["tau_open"], -h / p["tau_close"])
    du = -p["k"] * u * (u - p["a"]) * (u - 1) - u * h + J
    return du, (p["epsilon_0"] + p["mu1"] * h / (u + p["mu2"])) * (-h - p["k"] * u * (u - p["a"] - 1))


def _simulate64(d, steps, plain):
    """(u, h) histories and sample times.  ``plain``: a step whose start meets
    the reference's stopping test max(1e-5, 1e-5 |b|) keeps it."""
    model, sp = d["model"], d["sp"]
    n, ts, dt = d["ijk"].shape[0], sp["time_scale"], sp["dt"]
    p = synthetic.MS_PARAMS if model == 0 else synthetic.AP_PARAMS
    L = _Operator(d["ijk"], torch.as_tensor(d["par"]["c_voxel"], device="cuda"), d["D0"])
    u = torch.zeros(n, dtype=torch.float64, device="cuda")
    g = torch.full_like(u, 1.0 if model == 0 else 0.0)
    sets = [torch.zeros_like(u), torch.zeros_like(u)]
    for m, ids in zip(sets, (d["s1"], d["s2"])):
        m[torch.as_tensor(ids, device="cuda", dtype=torch.int64)] = 1.0
    t0 = [d["ap"]["s1_t"], d["ap"]["s1_t"] + d["ap"]["s1_s2_delta_t"]]
    if sp["arrhythmia_flag"] == 4:
        t0[1] = math.inf
    S, stride = _samples(steps, model)
    us, hs = [], []
    for k in range(int(np.round(sp["t_final"] / dt))):
        J = torch.zeros_like(u)
        for m, a in zip(sets, t0):
            if a <= k * dt <= a + d["pacing"]:
                J = torch.maximum(J, m)
        a1, b1 = _reaction(model, u, g, J, p)
        a2, b2 = _reaction(model, u + 0.5 * dt * a1, g + 0.5 * dt * b1, J, p)
        a3, b3 = _reaction(model, u + 0.5 * dt * a2, g + 0.5 * dt * b2, J, p)
        a4, b4 = _reaction(model, u + dt * a3, g + dt * b3, J, p)
        w = u + dt / 6 * (a1 + 2 * a2 + 2 * a3 + a4)
        g = g + dt / 6 * (b1 + 2 * b2 + 2 * b3 + b4)
        Lw = L(w)
        b = w + dt / 2 * Lw
        if plain and float((dt * Lw).norm()) <= max(1e-5, 1e-5 * float(b.norm())):
            u = w
        else:
            u = _solve(L, dt / 2, b, w)
        if k % stride == 0 and len(us) < S:
            us.append(u)
            hs.append(g)
    times = np.arange(len(us)) * stride * dt * ts
    return torch.stack(us), torch.stack(hs), times


def _leadfield64(xyz, exyz, c, D0, nb):
    """M (n_e, n): the gradient stencil carried over to the voxels it reads."""
    n, n_e = xyz.shape[0], exyz.shape[0]
    M = torch.zeros((n_e, n), dtype=torch.float64, device="cuda")
    for e in range(n_e):
        l = xyz - exyz[e]
        q = l if D0 is None else torch.einsum("vij,vi->vj", D0.view(-1, 3, 3), l)
        q = q * (c / l.norm(dim=1).clamp(min=1.0) ** 3 / (2 * DELTA))[:, None]
        for a in range(3):
            ok = (nb[:, 2 * a] >= 0) & (nb[:, 2 * a + 1] >= 0)
            M[e].index_add_(0, nb[ok, 2 * a], q[ok, a])
            M[e].index_add_(0, nb[ok, 2 * a + 1], -q[ok, a])
    return M


def _egm64(case, seed):
    ijk, xyz, exyz, c, D0, V = _egm_inputs(case, seed)
    nb = _neighbours(ijk, 6)
    parts = []
    for e in range(0, exyz.shape[0], 256):
        M = _leadfield64(xyz, exyz[e:e + 256], c, D0, nb)
        parts.append(torch.cat([V[t:t + 250].double() @ M.T for t in range(0, V.shape[0], 250)]))
    egm = torch.cat(parts, dim=1)
    return egm / (egm.max(dim=0).values - egm.min(dim=0).values).mean()


def _electrodes64(case, seed):
    xyz, sig = _electrode_inputs(case, seed)
    lat = torch.argmax(-(sig[1:] - sig[:-1]), dim=0).cpu().numpy()
    lat = (lat - lat.min()).astype(np.float64)
    vec = np.full((xyz.shape[0], 3), np.nan)
    mag = np.full(xyz.shape[0], np.nan)
    for i, x in enumerate(xyz):
        near = np.flatnonzero(((xyz - x) ** 2).sum(axis=1) <= RADIUS_MM ** 2)
        if near.size < 4:
            continue
        co = np.linalg.lstsq(np.c_[xyz[near], np.ones(near.size)], lat[near], rcond=None)[0][:3]
        if co @ co > 1e-8:
            vec[i] = co / (co @ co)
            mag[i] = 1.0 / np.sqrt(co @ co)
    return None, vec, mag, float(np.nanmean(mag))


def exact(case, seed):
    kind = case["kind"]
    if kind == "drop_in":
        u, h, t = _simulate64(_sheet_inputs(case, seed), case["steps"], not case["fast"])
        return u, h, t
    if kind == "job":
        return [_simulate64(d, case["steps"], not case["fast"])[0] for d in _job_inputs(case, seed)]
    if kind in ("egm_fp64", "egm_bf16x3"):
        return _egm64(case, seed)
    if kind == "electrodes":
        return _electrodes64(case, seed)
    return None                        # indices: whole numbers, compared as they are
