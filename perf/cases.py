"""The calls that users of the map engine make, as measurable cases.

A case is a plain dict.  `kind` names the public entry point:

  plan           Plan.run on a device-resident problem (repeated runs)
  compute        Context.compute, host arrays in, host maps out (the drop-in's call)
  batch          Batch.run and the download of every instance's maps
  compute_batch  compute_batch, many host problems in one call
  diff           Diff: coordinates in, maps out, dL/d(maps) in, gradients out
  vina           the same for several conformers and Vina-potential tables
  text           Context.format: map-file bodies of device-resident maps

Receptors are synthetic with the composition of the package's benchmark
(synth.py): atoms at 0.026 per cubic Angstrom in a sphere, types C 45%, A 10%,
N 10%, NA 3%, OA 15%, SA 2%, HD 15%, hydrogens 1 A from an N or OA parent, and
AD4.1 tables.  They are built here with numpy, because the inputs are made many
times.  `exact` restates every output in 64 bits with torch.
"""
import math

import numpy as np
import torch

from autogrid_b200.api import Batch, Context, Diff, Problem, compute_batch

A_DIV, NEINT, NDIEL, CUTOFF = 128, 1024, 8192, 8.0
REC_TYPES = ["C", "A", "N", "NA", "OA", "SA", "HD"]
HEAVY_SHARE = [0.45, 0.10, 0.10, 0.03, 0.15, 0.02]
LIGANDS = {8: ["A", "C", "HD", "N", "NA", "OA"],
           16: ["A", "C", "HD", "N", "NA", "OA", "SA", "S", "P", "F", "Cl", "Br", "I", "Fe"]}
# Rii, epsii, vol, solpar, Rij_hb, epsij_hb, hbond class (AD4.1 bound)
PARAMS = {
    "C": (4.00, 0.150, 33.5103, -0.00143, 0.0, 0.0, 0), "A": (4.00, 0.150, 33.5103, -0.00052, 0.0, 0.0, 0),
    "N": (3.50, 0.160, 22.4493, -0.00162, 0.0, 0.0, 0), "NA": (3.50, 0.160, 22.4493, -0.00162, 1.9, 5.0, 4),
    "OA": (3.20, 0.200, 17.1573, -0.00251, 1.9, 5.0, 5), "SA": (4.00, 0.200, 33.5103, -0.00214, 2.5, 1.0, 5),
    "HD": (2.00, 0.020, 0.0000, 0.00051, 0.0, 0.0, 2), "S": (4.00, 0.200, 33.5103, -0.00214, 0.0, 0.0, 0),
    "P": (4.20, 0.200, 38.7924, -0.00110, 0.0, 0.0, 0), "F": (3.09, 0.080, 15.4480, -0.00110, 0.0, 0.0, 0),
    "Cl": (4.09, 0.276, 35.8235, -0.00110, 0.0, 0.0, 0), "Br": (4.33, 0.389, 42.5661, -0.00110, 0.0, 0.0, 0),
    "I": (4.72, 0.550, 55.0585, -0.00110, 0.0, 0.0, 0), "Fe": (1.30, 0.010, 1.8400, -0.00110, 0.0, 0.0, 0),
}
COEFF_VDW, COEFF_HBOND, COEFF_ESTAT, COEFF_DESOLV, QSOLPAR = 0.1662, 0.1209, 0.1406, 0.1322, 0.01097
XS_RADIUS = {"C": 1.9, "A": 1.9, "N": 1.8, "NA": 1.8, "OA": 1.7, "SA": 2.0, "HD": 1.0}
VINA_LIGANDS = ["A", "C", "HD", "N", "NA", "OA", "SA", "S"]


def listed():
    return [
        # one small box over a small receptor, the tables resident: latency of a run
        dict(name="plan_1800_41cube_8maps", kind="plan", atoms=1800, n1x=41, n1y=41, n1z=41, maps=8, spacing=0.375),
        # uneven box, another spacing (coordinates that are no exact floats)
        dict(name="plan_5003_95x73x41_16maps", kind="plan", atoms=5003, n1x=95, n1y=73, n1z=41, maps=16, spacing=0.4),
        # the benchmark's large map set, resident
        dict(name="plan_10000_127cube_16maps", kind="plan", atoms=10000, n1x=127, n1y=127, n1z=127, maps=16, spacing=0.375),
        # the drop-in call on a small box, from host arrays to host maps
        dict(name="compute_1800_41cube_8maps", kind="compute", atoms=1800, n1x=41, n1y=41, n1z=41, maps=8, spacing=0.375,
             precision="fp32"),
        # the drop-in call on the large map set
        dict(name="compute_10000_127cube_16maps", kind="compute", atoms=10000, n1x=127, n1y=127, n1z=127, maps=16,
             spacing=0.375, precision="fp32"),
        # the drop-in call in double precision
        dict(name="compute_fp64_3000_61cube_8maps", kind="compute", atoms=3000, n1x=61, n1y=61, n1z=61, maps=8,
             spacing=0.375, precision="fp64"),
        # an ensemble of uneven boxes kept on the device, run and read back
        dict(name="batch_24_8maps", kind="batch", instances=24, lo_atoms=1000, hi_atoms=12000, lo_n=21, hi_n=101, maps=8),
        # the same kind of ensemble in one call from host arrays to host maps
        dict(name="compute_batch_24_8maps", kind="compute_batch", instances=24, lo_atoms=1000, hi_atoms=12000, lo_n=21,
             hi_n=101, maps=8),
        # one optimisation step over receptor coordinates and charges: forward and adjoint
        dict(name="diff_4000_61cube_8maps", kind="diff", atoms=4000, n1x=61, n1y=61, n1z=61, maps=8, spacing=0.375,
             precision="fp32"),
        # the same in double precision (gradient checks)
        dict(name="diff_fp64_1000_33cube_8maps", kind="diff", atoms=1000, n1x=33, n1y=33, n1z=33, maps=8, spacing=0.375,
             precision="fp64"),
        # forward and adjoint of eight conformers' Vina maps
        dict(name="vina_8x8000_101cube_8maps", kind="vina", atoms=8000, n1x=101, n1y=101, n1z=101, conformers=8,
             spacing=0.375),
        # map-file text of computed maps
        dict(name="text_101cube_8maps", kind="text", n1x=101, n1y=101, n1z=101, maps=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(v):
    return int(v) // 2 * 2 + 1


def _box(rng, lo, hi):
    mean = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return [max(11, min(_odd(hi), _odd(mean * math.exp(rng.uniform(-0.35, 0.35))))) for _ in range(3)]


def draw(rng):
    kind = rng.choice(["plan", "plan", "compute", "compute", "batch", "compute_batch", "diff", "vina", "text"])
    if kind == "text":
        n = _box(rng, 31, 127)
        return dict(kind=kind, n1x=n[0], n1y=n[1], n1z=n[2], maps=rng.choice([8, 16]))
    if kind in ("batch", "compute_batch"):
        return dict(kind=kind, instances=rng.randint(5, 24), lo_atoms=rng.randint(600, 1500), hi_atoms=rng.randint(3000, 9000),
                    lo_n=21, hi_n=_odd(rng.randint(41, 95)), maps=8)
    if kind == "vina":
        n = _box(rng, 31, 101)
        return dict(kind=kind, atoms=_log(rng, 1000, 8000), n1x=n[0], n1y=n[1], n1z=n[2], conformers=rng.randint(1, 7),
                    spacing=0.375)
    if kind == "diff":
        fp64 = rng.random() < 0.3
        n = _box(rng, 21, 37 if fp64 else 61)
        return dict(kind=kind, atoms=_log(rng, 600, 1500 if fp64 else 5000), n1x=n[0], n1y=n[1], n1z=n[2],
                    maps=8 if fp64 else rng.choice([8, 16]), spacing=0.375, precision="fp64" if fp64 else "fp32")
    fp64 = kind == "compute" and rng.random() < 0.25
    n = _box(rng, 25, 61 if fp64 else 121)
    case = dict(kind=kind, atoms=_log(rng, 800, 3000 if fp64 else 9500), n1x=n[0], n1y=n[1], n1z=n[2],
                maps=rng.choice([8, 16]), spacing=rng.choice([0.375, 0.375, 0.4, 0.5]))
    if kind == "compute":
        case["precision"] = "fp64" if fp64 else "fp32"
    if rng.random() < 0.15:
        case["dielectric"] = 40.0  # a constant dielectric
    return case


# ------------------------------------------------------------------ inputs --
def _unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


def receptor(n, seed):
    """Arrays of a synthetic receptor of n atoms, centred, in file order (each
    heavy atom followed by its hydrogens)."""
    rng = np.random.default_rng(seed)
    n_hd = int(round(0.15 * n))
    n_heavy = n - n_hd
    radius = 45.0 * (n / 10000.0) ** (1.0 / 3.0)
    step = (4.0 / 3.0 * math.pi * radius ** 3 / n_heavy) ** (1.0 / 3.0)
    k = np.arange(-int(radius / step) - 3, int(radius / step) + 4)
    grid = np.stack(np.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3) * step
    p = grid + rng.uniform(-0.5, 0.5, 3) * step + rng.uniform(-0.5, 0.5, grid.shape) * (step - 1.1)
    p = p[np.argsort((p * p).sum(1))[:n_heavy]]
    rng.shuffle(p)
    share = np.array(HEAVY_SHARE) / sum(HEAVY_SHARE)
    counts = np.floor(share * n_heavy).astype(int)
    counts[0] += n_heavy - counts.sum()
    types = np.repeat(np.arange(len(counts)), counts)
    rng.shuffle(types)
    pool = np.flatnonzero((types == REC_TYPES.index("N")) | (types == REC_TYPES.index("OA")))
    parent = rng.choice(pool, n_hd, replace=False)
    bond = _unit(rng.normal(size=(n_hd, 3)))
    order = np.argsort(np.concatenate([np.arange(n_heavy) * 2, parent * 2 + 1]), kind="stable")
    rec_type = np.concatenate([types, np.full(n_hd, REC_TYPES.index("HD"))])[order]
    coord = np.round(np.concatenate([p, p[parent] + bond])[order], 3)
    hbond = np.array([PARAMS[t][6] for t in REC_TYPES])[rec_type]
    rv = np.where((hbond >= 4)[:, None], _unit(rng.normal(size=(n, 3))), 0.0)
    hd = np.concatenate([np.zeros((n_heavy, 3)), bond])[order]
    rv = np.where((hbond == 2)[:, None], hd, rv)
    rv2 = _unit(np.cross(rng.normal(size=(n, 3)), np.where((hbond == 5)[:, None], rv, 1.0)))
    rv2 = np.where((hbond == 5)[:, None], rv2, 0.0)
    rexp = np.concatenate([np.zeros(n_heavy, int), np.where(types[parent] == REC_TYPES.index("N"), 2, 4)])[order]
    q = rng.normal(0.0, 0.25, n)
    return dict(coord=coord, charge=np.round(q - q.mean(), 3), rec_type=rec_type, hbond=hbond, rexp=rexp, rvector=rv,
                rvector2=rv2, vol=np.array([PARAMS[t][2] for t in REC_TYPES])[rec_type],
                solpar=np.array([PARAMS[t][3] for t in REC_TYPES])[rec_type], disorder=np.zeros(n, np.uint8))


_TABLES = {}


def _pair_table(lig, rec):
    """Smoothed 12-6 or 12-10 table of one (ligand type, receptor type)."""
    a, b = PARAMS[lig], PARAMS[rec]
    acc, don = (3, 4, 5), (1, 2)
    hb = (a[6] in acc and b[6] in don) or (a[6] in don and b[6] in acc)
    if hb:
        rij, eps = (a[4], a[5]) if a[6] in acc else (b[4], b[5])
        eps, xb = eps * COEFF_HBOND, 10
    else:
        rij, eps, xb = (a[0] + b[0]) / 2, math.sqrt(a[1] * b[1]) * COEFF_VDW, 6
    r = np.arange(1, NEINT) / A_DIV
    tab = np.full(NEINT, 100000.0, np.float32)
    c = eps / (12 - xb)
    tab[1:] = np.minimum(c * rij ** 12 * xb / r ** 12 - c * rij ** xb * 12 / r ** xb, 100000.0)
    tab[-1] = 0.0
    pad = np.pad(tab, 32, constant_values=100000.0)  # smooth 0.5 A: the lowest of 65 bins
    return np.lib.stride_tricks.sliding_window_view(pad, 65).min(1)


def _tables(maps):
    if maps not in _TABLES:
        r = np.arange(NDIEL) / A_DIV
        sol = COEFF_DESOLV * np.exp(-(r * r) / (2 * 3.6 ** 2))
        sol[0] = 0.0
        eps = -8.5525 + (78.4 + 8.5525) / (1 + 7.7839 * np.exp(-0.003627 * (78.4 + 8.5525) * r))
        eps[0] = 1.0
        vdw = np.stack([np.stack([_pair_table(m, t) for m in LIGANDS[maps]]) for t in REC_TYPES])
        _TABLES[maps] = vdw, sol, 332.0 / eps
    return _TABLES[maps]


def _problem(rec, maps, n1, spacing, dielectric=None):
    """AD4 maps: the ligand types of LIGANDS[maps], the e map and the d map."""
    vdw, sol, eps = _tables(maps)
    lig = LIGANDS[maps]
    return Problem(**rec, n1=n1, spacing=spacing, e_vdw_hb=vdw, sol_fn=sol, r_epsilon_fn=eps, n_rec_types=len(REC_TYPES),
                   n_atom_maps=len(lig), n_maps=len(lig) + 2, elec_map=len(lig), dsolv_map=len(lig) + 1,
                   map_is_covalent=[0] * len(lig), map_is_hbonder=[int(PARAMS[t][6] > 0) for t in lig],
                   map_hbond=[PARAMS[t][6] for t in lig], map_solpar_probe=[PARAMS[t][3] for t in lig],
                   map_vol_probe=[PARAMS[t][2] for t in lig], dddiel=int(dielectric is None),
                   invdielcal=332.0 / dielectric if dielectric else 0.0, coeff_estat=COEFF_ESTAT, solpar_q=QSOLPAR,
                   disorder_h=0, hydrogen_type=-1, separate_desolvation_maps=0, cov_half_width=1.0, cov_barrier=1000.0,
                   floating_grid=0, constriction_grid=0, constriction_cutoff=7.5, report_collisions=0)


def _vina_problem(rec, n1, spacing):
    """Maps of the Vina terms: plain sums, no e or d map."""
    if "vina" not in _TABLES:
        r = np.arange(1, NEINT) / A_DIV
        vdw = np.zeros((len(REC_TYPES), len(VINA_LIGANDS), NEINT), np.float32)
        for i, t in enumerate(REC_TYPES):
            for m, g in enumerate(VINA_LIGANDS):
                d = r - XS_RADIUS[t] - XS_RADIUS.get(g, 1.8)
                v = -0.035579 * np.exp(-(d / 0.5) ** 2) - 0.005156 * np.exp(-((d - 3.0) / 2.0) ** 2)
                v += np.where(d < 0, 0.840245 * d * d, 0.0)
                if t in "CA" and g in "CA":
                    v += -0.035069 * np.clip((0.5 - d), 0.0, 1.0)
                elif {t, g} & {"HD"} and {t, g} & {"OA", "NA", "SA"}:
                    v += -0.587439 * np.clip(-d / 0.7, 0.0, 1.0)
                vdw[i, m, 1:] = v
        _TABLES["vina"] = vdw
    k = len(VINA_LIGANDS)
    return Problem(**rec, n1=n1, spacing=spacing, e_vdw_hb=_TABLES["vina"], sol_fn=np.zeros(NDIEL),
                   r_epsilon_fn=np.zeros(NDIEL), n_rec_types=len(REC_TYPES), n_atom_maps=k, n_maps=k, elec_map=-1,
                   dsolv_map=-1, map_is_covalent=[0] * k, map_is_hbonder=[0] * k, map_hbond=[0] * k,
                   map_solpar_probe=[0.0] * k, map_vol_probe=[0.0] * k, dddiel=0, invdielcal=1.0, coeff_estat=0.0,
                   solpar_q=0.0, disorder_h=0, hydrogen_type=-1, separate_desolvation_maps=0, cov_half_width=1.0,
                   cov_barrier=1000.0, floating_grid=0, constriction_grid=0, constriction_cutoff=7.5, report_collisions=0)


def _n1(case):
    return case["n1x"], case["n1y"], case["n1z"]


def _ensemble(case):
    """(atoms, box) of each instance: atoms log-uniform, box sides uniform.  They
    are the case's own; the seed makes the receptors."""
    rng = np.random.default_rng([7, case["instances"], case["lo_atoms"], case["hi_atoms"], case["hi_n"]])
    sizes = []
    for _ in range(case["instances"]):
        n = int(round(math.exp(rng.uniform(math.log(case["lo_atoms"]), math.log(case["hi_atoms"])))))
        sizes.append((n, tuple(_odd(v) for v in rng.integers(case["lo_n"], case["hi_n"] + 1, 3))))
    return sizes


def _problems(case, seed):
    return [_problem(receptor(n, [seed, i]), case["maps"], box, 0.375) for i, (n, box) in enumerate(_ensemble(case))]


def _single(case, seed):
    return _problem(receptor(case["atoms"], seed), case["maps"], _n1(case), case["spacing"], case.get("dielectric"))


def _pinned(shape, dtype=torch.float32):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _conformers(case, seed, rec):
    """Base structure plus N(0, 0.3 A) per atom, in the float32 of a user's parameters."""
    rng = np.random.default_rng([seed, 5])
    return (rec["coord"] + rng.normal(0.0, 0.3, (case["conformers"],) + rec["coord"].shape)).astype(np.float32)


def _weights(shape, seed, dtype):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype)


class _HostText:
    """The text of a format call, in the context's own buffer."""

    def __init__(self, ctx, text):
        self.ctx = ctx
        self.__array_interface__ = dict(shape=(text.total,), typestr="|u1", version=3, data=(text.ptr, True))


class _DeviceMaps:
    """A Plan's device maps as an array that torch can wrap."""

    def __init__(self, plan):
        self.plan = plan
        self.__cuda_array_interface__ = dict(shape=plan.problem.map_shape, typestr="<f4", version=3,
                                             data=(plan.device_maps_ptr(), False))


def prepare(case, seed):
    kind, ctx = case["kind"], Context(0)
    if kind == "plan":
        plan = ctx.plan(_single(case, seed))
        return dict(kind=kind, plan=plan, maps=torch.as_tensor(_DeviceMaps(plan), device="cuda"))
    if kind == "compute":
        prob = _single(case, seed)
        out = _pinned(prob.map_shape, torch.float64 if case["precision"] == "fp64" else torch.float32)
        return dict(kind=kind, ctx=ctx, prob=prob, out=out, precision=case["precision"])
    if kind in ("batch", "compute_batch"):
        probs = _problems(case, seed)
        outs = [_pinned(p.map_shape) for p in probs]
        return dict(kind=kind, ctx=ctx, probs=probs, outs=outs, batch=Batch(ctx, probs) if kind == "batch" else None)
    if kind in ("diff", "vina"):
        rec = receptor(case["atoms"], seed)
        if kind == "vina":
            prob, k, dtype = _vina_problem(rec, _n1(case), case["spacing"]), case["conformers"], torch.float32
            coord = _conformers(case, seed, rec)
            coord = coord[0] if k == 1 else coord
        else:
            prob, k = _problem(rec, case["maps"], _n1(case), case["spacing"]), 1
            dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
            coord = rec["coord"].astype(np.float32)
        d = Diff(ctx, prob, "fp64" if dtype == torch.float64 else "fp32", conformers=k)
        charge = np.broadcast_to(rec["charge"], coord.shape[:-1]).copy()
        return dict(kind=kind, diff=d, dtype=dtype, coord=torch.from_numpy(coord).to("cuda", dtype),
                    charge=torch.from_numpy(charge).to("cuda", dtype),
                    maps=torch.empty(d.shape, dtype=dtype, device="cuda"), grad=_weights(d.shape, seed, dtype))
    # text: affinity-like values, most of them small, some in clashes, some zero;
    # the seed orders the points (the length of the text stays the same)
    prob = _problem(receptor(64, seed), case["maps"], _n1(case), 0.375)
    g = torch.Generator(device="cuda").manual_seed(0)
    shape = (prob.n_out, prob.points)
    v = torch.randn(shape, generator=g, device="cuda") * 0.4
    u = torch.rand(shape, generator=g, device="cuda")
    v = torch.where(u > 0.75, torch.exp(v.abs() * 12.0).clamp(max=3.0e5), v)
    v = torch.where(u < 0.02, torch.zeros_like(v), v)
    order = torch.randperm(prob.points, generator=g.manual_seed(seed), device="cuda")
    return dict(kind=kind, ctx=ctx, prob=prob, maps=v[:, order].contiguous())


def run(state):
    kind = state["kind"]
    if kind == "plan":
        state["plan"].run()
        return state["maps"]
    if kind == "compute":
        return state["ctx"].compute(state["prob"], state["precision"], out=state["out"])
    if kind == "batch":
        state["batch"].run()
        return [state["batch"].download(i, o) for i, o in enumerate(state["outs"])]
    if kind == "compute_batch":
        return compute_batch(state["ctx"], state["probs"], state["outs"])
    if kind in ("diff", "vina"):
        # one step of an optimisation loop: the engine takes FP64 device arrays
        d, coord, charge = state["diff"], state["coord"].double(), state["charge"].double()
        torch.cuda.current_stream().synchronize()  # the engine works on a stream of its own
        d.set_atoms_device(coord.data_ptr(), charge.data_ptr())
        d.forward(device_out=state["maps"].data_ptr())
        g, gq = torch.empty_like(coord), torch.empty_like(charge)
        d.backward_device(state["grad"].data_ptr(), g.data_ptr(), gq.data_ptr())
        if kind == "vina":  # these maps do not depend on the charges
            return dict(maps=state["maps"], coord=g.to(state["dtype"]))
        return dict(maps=state["maps"], coord=g.to(state["dtype"]), charge=gq.to(state["dtype"]))
    mt = state["ctx"].format(state["prob"], state["maps"].data_ptr(), 4)
    return dict(text=np.asarray(_HostText(state["ctx"], mt)), map_bytes=mt.map_bytes.astype(np.int64), emin=mt.emin, emax=mt.emax)


def _pair_work(atoms, points, maps, elem):
    """Map values: 12 operations per far pair (distance, 1/r, table value), 25
    plus 3 per map for the pairs within 8 A (56 per point at 0.026 atoms per
    cubic Angstrom, fewer outside the receptor)."""
    near = 40.0 * points
    return dict(bytes=80.0 * atoms + elem * points * maps, flops=12.0 * atoms * points + near * (25.0 + 3.0 * maps))


def work(case):
    kind = case["kind"]
    if kind in ("batch", "compute_batch"):
        parts = [_pair_work(n, b[0] * b[1] * b[2], case["maps"], 4) for n, b in _ensemble(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    points = case["n1x"] * case["n1y"] * case["n1z"]
    if kind == "text":
        return dict(bytes=points * case["maps"] * 11.0, flops=0.0)
    elem = 8 if case.get("precision") == "fp64" else 4
    if kind == "vina":
        k = case["conformers"]
        w = _pair_work(0, points, 8, elem)
        return dict(bytes=k * (2 * w["bytes"] + 48.0 * case["atoms"]), flops=3.0 * k * w["flops"])
    w = _pair_work(case["atoms"], points, case["maps"], elem)
    if kind == "diff":
        return dict(bytes=2 * w["bytes"], flops=3 * w["flops"])
    return w


# ------------------------------------------------------------- exact values --
class _Exact:
    """The maps of a problem (and the gradient of sum(weights * maps)) in 64
    bits: nearest-bin tables, or linearly interpolated ones (`linear`)."""

    def __init__(self, prob, linear=False, coord=None):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda v: torch.as_tensor(np.asarray(v, np.float64), device=self.dev)  # noqa: E731
        a, s = prob.arrays, prob.scalars
        self.s, self.linear, self.n1 = s, linear, prob.n1
        self.coord = t(a["coord"] if coord is None else coord).reshape(-1, 3)
        self.q, self.rv, self.rv2 = t(a["charge"]), t(a["rvector"]).reshape(-1, 3), t(a["rvector2"]).reshape(-1, 3)
        self.vol, self.solpar = t(a["vol"]), t(a["solpar"])
        self.type = torch.as_tensor(a["rec_type"].astype(np.int64), device=self.dev)
        self.hb = torch.as_tensor(a["hbond"].astype(np.int64), device=self.dev)
        self.rexp = torch.as_tensor(a["rexp"].astype(np.int64), device=self.dev)
        self.n_atoms, self.nam = prob.n_atoms, int(s["n_atom_maps"])
        # [type * NEINT + bin][map]
        self.vdw = t(a["e_vdw_hb"].reshape(-1, self.nam, NEINT)).permute(0, 2, 1).reshape(-1, self.nam).contiguous()
        self.step = torch.zeros_like(self.vdw).reshape(-1, NEINT, self.nam)
        self.step[:, :-1] = self.vdw.reshape(-1, NEINT, self.nam).diff(dim=1)
        self.step = self.step.reshape(-1, self.nam)
        self.sol, self.dsol = t(a["sol_fn"][:NEINT]), t(a["sol_fn"][:NEINT + 1]).diff()
        eps = t(a["r_epsilon_fn"]) if s["dddiel"] else torch.full((NDIEL,), float(s["invdielcal"]), dtype=torch.float64,
                                                                  device=self.dev)
        self.eps = eps * s["coeff_estat"]
        self.deps = torch.cat([self.eps.diff(), self.eps.new_zeros(1)])
        self.axes = [(torch.arange(n, device=self.dev, dtype=torch.float64) - (n - 1) // 2) * s["spacing"] for n in prob.n1]
        z, y, x = torch.meshgrid(self.axes[2], self.axes[1], self.axes[0], indexing="ij")
        self.pts = torch.stack([x, y, z], -1).reshape(-1, 3)
        self.hbonder = [m for m in range(self.nam) if a["map_is_hbonder"][m]]
        self.map_hbond = a["map_hbond"]
        self.sp, self.vp = t(a["map_solpar_probe"]), t(a["map_vol_probe"])
        self.ch = self._closest_h() if self.hbonder else None

    def _closest_h(self):
        h = torch.nonzero((self.hb == 1) | (self.hb == 2)).reshape(-1)
        out = []
        step = max(1, 2 ** 25 // max(1, h.numel()))
        for p in self.pts.split(step):
            r2 = sum((self.coord[h, d][None] - p[:, d, None]) ** 2 for d in range(3))
            out.append(h[r2.argmin(1)])
        return torch.cat(out)

    def emap(self, weight=None):
        """The e map; with weight, dL/d(coord) and dL/dq instead."""
        grad = weight is not None
        out = None if grad else torch.zeros(len(self.pts), dtype=torch.float64, device=self.dev)
        gx, gq = torch.zeros_like(self.coord), torch.zeros_like(self.q)
        step = max(1, 2 ** 24 // len(self.pts))
        for a0 in range(0, self.n_atoms, step):
            a = slice(a0, a0 + step)
            d = [self.coord[a, i][:, None] - self.pts[None, :, i] for i in range(3)]
            if self.linear:
                r = (d[0] ** 2 + d[1] ** 2 + d[2] ** 2).sqrt().clamp(min=1e-6)
                b = (r * A_DIV).long().clamp(max=NDIEL - 1)
                slope = self.deps[b]
                T = self.eps[b] + (r * A_DIV - b) * slope
            else:
                r = torch.hypot(d[0], torch.hypot(d[1], d[2])).clamp(min=1e-6)
                T = self.eps[(r * A_DIV).long().clamp(max=NDIEL - 1)]
            inv = 1.0 / r.clamp(min=0.5)
            if not grad:
                out += (self.q[a][:, None] * T * inv).sum(0)
                continue
            gq[a] = (T * inv * weight).sum(1)
            dF = torch.where(r > 0.5, (slope * A_DIV - T * inv) * inv, slope * A_DIV * inv)
            k = weight * dF / r * self.q[a][:, None]
            for i in range(3):
                gx[a, i] = (k * d[i]).sum(1)
        return (gx, gq) if grad else out

    def _pairs(self, a0, step):
        """(atom, point) index of the pairs within the cutoff."""
        at = torch.arange(a0, min(self.n_atoms, a0 + step), device=self.dev)
        reach = int(CUTOFF / self.s["spacing"]) + 2
        off = torch.arange(-reach, reach + 1, device=self.dev)
        idx, d2 = [], []
        for i in range(3):
            k = torch.round(self.coord[at, i] / self.s["spacing"]).long()[:, None] + off + (self.n1[i] - 1) // 2
            ok = (k >= 0) & (k < self.n1[i])
            d = (self.coord[at, i][:, None] - (k - (self.n1[i] - 1) // 2) * self.s["spacing"]) ** 2
            idx.append(k)
            d2.append(torch.where(ok, d, torch.full_like(d, 1e9)))
        yz = d2[2][:, :, None] + d2[1][:, None, :]
        j, kz, ky = torch.nonzero(yz <= CUTOFF ** 2 + 0.01, as_tuple=True)
        full = yz[j, kz, ky][:, None] + d2[0][j]
        m, kx = torch.nonzero(full <= CUTOFF ** 2 + 0.01, as_tuple=True)
        j, kz, ky = j[m], kz[m], ky[m]
        return at[j], (idx[2][j, kz] * self.n1[1] + idx[1][j, ky]) * self.n1[0] + idx[0][j, kx]

    def _angles(self, at, pt, dn, rv, rv2):
        """racc, rdon, Hramp of the pairs."""
        racc, rdon, ramp = (torch.ones(len(at), dtype=torch.float64, device=self.dev) for _ in range(3))
        if not self.hbonder:
            return racc, rdon, ramp
        hb = self.hb[at]
        i = torch.nonzero(hb == 2).reshape(-1)
        c = -(dn[i] * rv[at[i]]).sum(1)
        pos = c.clamp(min=0.0)
        e = self.rexp[at[i]]
        racc = racc.index_put((i,), torch.where(e == 2, pos ** 2, torch.where(e == 4, pos ** 4, pos)))
        h = self.ch[pt[i]]
        use = (h != at[i]) & ((c > 0) | self.linear)
        i, h = i[use], h[use]
        ct = (rv[h] * rv[at[i]]).sum(1).clamp(-1.0, 1.0)
        ramp = ramp.index_put((i,), 0.5 - 0.5 * torch.cos(torch.acos(ct) * (120.0 / 90.0)))
        i = torch.nonzero(hb == 4).reshape(-1)
        rdon = rdon.index_put((i,), (-(dn[i] * rv[at[i]]).sum(1)).clamp(min=0.0) ** 2)
        i = torch.nonzero(hb == 5).reshape(-1)
        n, v, w = dn[i], rv[at[i]], rv2[at[i]]
        c = -(n * v).sum(1)
        t0 = (n * w).sum(1).clamp(-1.0, 1.0)
        ct0 = (1.0 - t0 * t0).clamp(min=1e-30).sqrt()
        cr = torch.linalg.cross(n, w)
        ti = (cr * v).sum(1) / (cr * cr).sum(1).clamp(min=1e-6).sqrt()
        ti = ti.clamp(-1.0, 1.0)
        s2 = 2.0 * ti.abs() * (1.0 - ti * ti).clamp(min=1e-30).sqrt()
        front = (0.9 + 0.1 * s2) * ct0
        back = 562.25 * (0.116978 - c * c) ** 3 * ct0
        if self.linear:
            back = back * (1.0 + s2 / 9.0)
        zero = torch.zeros_like(c)
        return racc, rdon.index_put((i,), torch.where(c >= 0, front, torch.where(c >= -0.34202, back, zero))), ramp

    def _terms(self, at, pt, coord, q, rv, rv2):
        """Value of each pair in every map [pairs, maps], the d map's, and the
        pairs that enter by the H-bond minimum and maximum."""
        d = coord[at] - self.pts[pt]
        r = (d * d).sum(1).sqrt().clamp(min=1e-6)
        dn = d / r[:, None]
        x = r * A_DIV
        b = x.detach().long().clamp(max=NEINT - 1)
        row = self.type[at] * NEINT + b
        T, sol = self.vdw[row], self.sol[b]
        w = torch.ones_like(r)
        if self.linear:
            f = x - b
            T = T + f[:, None] * self.step[row]
            sol = sol + f * self.dsol[b]
            w = (NEINT - x).clamp(max=1.0)
        racc, rdon, ramp = self._angles(at, pt, dn, rv, rv2)
        hb = self.hb[at]
        cols, ext = list(T.unbind(1)), {}
        for m in self.hbonder:
            mh, Tm = int(self.map_hbond[m]), T[:, m]
            rs = (Tm / 100.0).clamp(0.0, 1.0)
            donor = (hb == 1) | (hb == 2)
            if mh in (3, 5):
                cols[m] = torch.where(donor, Tm * ramp * (racc + (1 - racc) * rs), Tm)
            else:
                mine = donor if mh == 4 else hb > 2
                f = racc if mh == 4 else rdon
                ext[m] = (mine, w * Tm * (f + (1 - f) * rs))
                cols[m] = torch.where(mine, torch.zeros_like(Tm), Tm)
        solv = self.solpar[at] + self.s["solpar_q"] * q[at].abs()
        ws = (w * sol)[:, None]
        E = w[:, None] * torch.stack(cols, 1) + ws * (self.sp * self.vol[at][:, None] + self.vp * solv[:, None])
        return E, w * sol * self.vol[at] * self.s["solpar_q"], ext

    def _chunks(self):
        reach = CUTOFF / self.s["spacing"]
        per_atom = max(1.0, min(float(len(self.pts)), 4.2 * reach ** 3))
        step = max(1, int(1.5e6 / per_atom))
        for a0 in range(0, self.n_atoms, step):
            at, pt = self._pairs(a0, step)
            if len(at):
                d = self.coord[at] - self.pts[pt]
                near = (d * d).sum(1).sqrt() <= CUTOFF
                yield at[near], pt[near]

    def maps(self):
        """[n_maps, points]; keeps the H-bond extremes for grad()."""
        P = len(self.pts)
        out = torch.zeros((int(self.s["n_maps"]), P), dtype=torch.float64, device=self.dev)
        ext = [m for m in self.hbonder if int(self.map_hbond[m]) in (1, 2, 4)]
        self.lo = {m: torch.full((P,), 999999.0, dtype=torch.float64, device=self.dev) for m in ext}
        self.hi = {m: torch.full((P,), -999999.0, dtype=torch.float64, device=self.dev) for m in ext}
        for at, pt in self._chunks():
            E, dm, mm = self._terms(at, pt, self.coord, self.q, self.rv, self.rv2)
            for m in range(self.nam):
                out[m].index_add_(0, pt, E[:, m])
            if self.s["dsolv_map"] >= 0:
                out[self.s["dsolv_map"]].index_add_(0, pt, dm)
            for m, (mine, v) in mm.items():
                self.lo[m].scatter_reduce_(0, pt[mine], v[mine], "amin")
                self.hi[m].scatter_reduce_(0, pt[mine], v[mine], "amax")
        for m in ext:
            some = self.hi[m] > -999999.0
            out[m] += torch.where(some, self.lo[m] + self.hi[m].clamp(min=0.0), torch.zeros_like(self.lo[m]))
        if self.s["elec_map"] >= 0:
            out[self.s["elec_map"]] = self.emap()
        return out

    def grad(self, weight):
        """Gradients of sum(weight * maps) (after maps())."""
        w = weight.to(self.dev, torch.float64).reshape(int(self.s["n_maps"]), -1)
        total = [torch.zeros_like(v) for v in (self.coord, self.q, self.rv, self.rv2)]
        for at, pt in self._chunks():
            var = [v.clone().requires_grad_(True) for v in (self.coord, self.q, self.rv, self.rv2)]
            E, dm, mm = self._terms(at, pt, *var)
            L = sum((E[:, m] * w[m][pt]).sum() for m in range(self.nam))
            if self.s["dsolv_map"] >= 0:
                L = L + (dm * w[self.s["dsolv_map"]][pt]).sum()
            for m, (mine, v) in mm.items():
                hit = (v == self.lo[m][pt]).double() + ((v == self.hi[m][pt]) & (v > 0)).double()
                L = L + (v * (hit * mine * w[m][pt]).detach()).sum()
            for acc, g in zip(total, torch.autograd.grad(L, var, allow_unused=True)):
                if g is not None:
                    acc += g
        if self.s["elec_map"] >= 0:
            gx, gq = self.emap(w[self.s["elec_map"]])
            total[0] += gx
            total[1] += gq
        return total


def exact(case, seed):
    kind = case["kind"]
    if kind == "text":
        return None  # bytes, and extremes of the inputs themselves
    if kind in ("plan", "compute"):
        prob = _single(case, seed)
        return _Exact(prob).maps().reshape(prob.map_shape)
    if kind in ("batch", "compute_batch"):
        # the larger instances would take too long together
        return [_Exact(p).maps().reshape(p.map_shape) if p.points * p.n_atoms < 1.0e9 else None
                for p in _problems(case, seed)]
    rec = receptor(case["atoms"], seed)
    if kind == "diff":
        prob = _problem(rec, case["maps"], _n1(case), case["spacing"])
        dtype = torch.float64 if case["precision"] == "fp64" else torch.float32
        ex = _Exact(prob, linear=True, coord=rec["coord"].astype(np.float32))
        ex.q = torch.from_numpy(rec["charge"]).to(dtype).double().to(ex.dev)
        maps = ex.maps()
        g = ex.grad(_weights(prob.map_shape, seed, dtype))
        return dict(maps=maps.reshape(prob.map_shape), coord=g[0], charge=g[1])
    prob, k = _vina_problem(rec, _n1(case), case["spacing"]), case["conformers"]
    coord, shape = _conformers(case, seed, rec), (k,) + prob.map_shape
    weight = _weights(prob.map_shape if k == 1 else shape, seed, torch.float32).reshape(shape)
    maps, grads = [], []
    for c in range(k):
        ex = _Exact(prob, linear=True, coord=coord[c])
        maps.append(ex.maps().reshape(prob.map_shape))
        grads.append(ex.grad(weight[c])[0])
    if k == 1:
        return dict(maps=maps[0], coord=grads[0])
    return dict(maps=torch.stack(maps), coord=torch.stack(grads))
