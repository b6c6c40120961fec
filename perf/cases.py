"""Workloads of the library as programs run them, for timing and for comparing results.

Every case goes through the package's public Python entry points: the one-shot profile and the histogram
managers on host arrays, device-resident structures and batches, the SimpleCalculator and the rigid-body
server, the fitter and the hydration generator.  The structures are the seeded globules, hydration shells and
shell assemblies of ausaxs_b200.synth at the sizes of the benchmark configurations (500 to 500,000 atoms).

``exact`` evaluates the same quantities in 64 bits with plain torch from the mathematics: all pair distances,
their histogram by form-factor pair, the mean distance of every bin, and the Debye sum over the bins.
"""
import math

import numpy as np
import torch

import ausaxs_b200 as ab
from ausaxs_b200 import _capi, hist, synth

RHO_WATER = 0.334  # e / A^3
VOLUME_PER_ATOM = 18.0  # A^3, a protein-like specific volume


def listed():
    return [
        # the smallest call: a peptide-sized model scored inside a host program's loop, launch latency only
        {"name": "profile_500", "kind": "profile", "manager": "ffavg", "atoms": 500, "waters": 100, "width": 0.25,
         "nq": 100, "qmax": 0.5, "precision": 1},
        # the ordinary SAXS model (5,000 atoms, 200 q) kept on the device and evaluated again and again
        {"name": "structure_5k", "kind": "structure", "manager": "ffavg", "atoms": 5000, "waters": 1000, "width": 0.25,
         "nq": 200, "qmax": 0.5, "precision": 2},
        # the reference's own usage, molecule -> calculate_all() -> debye_transform() on its default q axis,
        # with explicit excluded volumes and an odd size
        {"name": "histogram_2711", "kind": "histogram", "manager": "ffexplicit", "atoms": 2711, "waters": 533,
         "width": 0.25, "nq": 0, "qmax": 0.5, "precision": 1},
        # the Simple (weighted) model of a mid-size complex
        {"name": "weighted_20k", "kind": "structure", "manager": "mt", "atoms": 20011, "waters": 4003, "width": 0.25,
         "nq": 200, "qmax": 0.5, "precision": 2},
        # wide-angle profile with fine bins and given excluded-volume dummies, host arrays in, I(q) out
        {"name": "grid_10k", "kind": "profile", "manager": "ffgrid", "atoms": 10007, "waters": 2001, "width": 0.1,
         "nq": 1000, "qmax": 1.0, "precision": 2},
        # the benchmark's wide-angle structure, its dummies kept on the device
        {"name": "grid_50k", "kind": "structure", "manager": "ffgrid", "atoms": 50000, "waters": 10000, "width": 0.1,
         "nq": 1000, "qmax": 1.0, "precision": 2},
        # the largest single structure: a 60-fold icosahedral shell
        {"name": "shell_500k", "kind": "structure", "manager": "ffavg", "atoms": 499980, "waters": 60000, "width": 0.1,
         "nq": 2000, "qmax": 1.0, "precision": 2},
        # an ensemble of models of uneven size, scored together from one captured graph
        {"name": "batch_32", "kind": "batch", "structures": 32, "nmin": 500, "nmax": 50000, "width": 0.25, "nq": 400,
         "qmax": 0.8, "precision": 2},
        # one step of rigid-body refinement and its rejection: a body moved and moved back, I(q) and fit for each
        {"name": "serve_8_bodies", "kind": "serve", "bodies": 8, "nmin": 3000, "nmax": 20000, "nq": 400, "qmax": 0.5},
        # symmetric assembly through the calculator: scaled self and cross jobs of a body and its copies
        {"name": "calculator_12mer", "kind": "calculator", "atoms": 4001, "copies": 12, "waters": 800, "width": 0.25},
        # fit of the hydration contrast to a measured curve, from an existing histogram
        {"name": "fit_5k", "kind": "fit", "atoms": 5000, "waters": 1000, "width": 0.25, "nq": 200, "qmax": 0.5},
        # hydration shell regenerated after a conformational change
        {"name": "hydrate_12k", "kind": "hydrate", "atoms": 12000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["profile", "structure", "structure", "structure", "histogram", "batch", "serve", "calculator",
                       "fit", "hydrate"])
    if kind in ("profile", "structure", "histogram"):
        if kind == "histogram":
            manager = rng.choice(["ffavg", "ffexplicit", "mt"])
        else:
            manager = rng.choice(["ffavg", "ffavg", "ffexplicit", "mt", "ffgrid"])
        hi = {"histogram": 10000, "profile": 20000, "structure": 60000}[kind]
        n = _log_int(rng, 500, min(hi, 20000) if manager == "ffgrid" else hi)
        width = 0.1 if manager == "ffgrid" else rng.choice([0.25, 0.25, 0.1])
        return {"kind": kind, "manager": manager, "atoms": n, "waters": int(n * rng.uniform(0.05, 0.25)), "width": width,
                "nq": 0 if kind == "histogram" else rng.randint(50, 1000), "qmax": rng.choice([0.5, 0.8, 1.0]),
                "precision": rng.choice([1, 2, 2])}
    if kind == "batch":
        return {"kind": "batch", "structures": rng.randint(3, 32), "nmin": 500, "nmax": _log_int(rng, 2000, 30000),
                "width": rng.choice([0.25, 0.25, 0.1]), "nq": rng.randint(100, 500), "qmax": 0.8,
                "precision": rng.choice([1, 2])}
    if kind == "serve":
        return {"kind": "serve", "bodies": rng.randint(2, 8), "nmin": 1000, "nmax": _log_int(rng, 3000, 20000),
                "nq": rng.randint(100, 500), "qmax": 0.5}
    if kind == "calculator":
        return {"kind": "calculator", "atoms": _log_int(rng, 300, 8333), "copies": rng.randint(2, 12),
                "waters": rng.randint(50, 1500), "width": rng.choice([0.25, 0.1])}
    if kind == "fit":
        n = _log_int(rng, 500, 12000)
        return {"kind": "fit", "atoms": n, "waters": int(n * rng.uniform(0.1, 0.25)), "width": 0.25,
                "nq": rng.randint(60, 500), "qmax": 0.5}
    return {"kind": "hydrate", "atoms": _log_int(rng, 500, 50000)}


# ---- inputs ---------------------------------------------------------------------------------------------------


def _shell(seed, n, n_waters):
    """A 60-fold icosahedral shell: one subunit with its waters, turned into place."""
    sub, ff = synth.globule(seed, n // 60, r_in=120.0, r_out=150.0, cone_cos=1.0 - 1.0 / 36.0)
    w = synth.waters(seed + 1, sub, ff, n_waters // 60)
    R = synth.icosahedral_rotations()
    return (np.concatenate([sub @ r.T for r in R]), np.tile(ff, len(R)), np.concatenate([w @ r.T for r in R]))


def _molecule(seed, n, n_waters, grid=False):
    if n > 200000:
        xyz, ff, w = _shell(seed, n, n_waters)
    else:
        xyz, ff = synth.globule(seed, n)
        w = synth.waters(seed + 1, xyz, ff, n_waters)
    x = synth.exv_grid(xyz, ff) if grid else None
    return ab.Molecule(atoms=xyz, ff_types=ff, weights=synth.ff_charge(ff), waters=w,
                       water_weights=np.full(len(w), synth.ff_charge([synth.FF_WATER])[0]), exv=x,
                       volume=VOLUME_PER_ATOM * n)


def _case_molecule(case, seed):
    return _molecule(97 * seed + 1, case["atoms"], case["waters"], case.get("manager") == "ffgrid")


def _batch_molecules(case, seed):
    rng = np.random.default_rng(seed)
    ns = np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["structures"]))
    ns[0], ns[-1] = case["nmin"], case["nmax"]
    return [_molecule(1009 * seed + 31 * i + 7, int(n), int(round(0.2 * n))) for i, n in enumerate(ns)]


def _q(case):
    return np.linspace(0.005, case["qmax"], case["nq"])


def _manager(case, molecule):
    kind = case.get("manager", "ffavg")
    if kind == "ffgrid":
        return ab.HistogramManagerMTFFGrid(molecule, case["width"], 8000)
    cls = {"ffavg": ab.HistogramManagerMTFFAvg, "ffexplicit": ab.HistogramManagerMTFFExplicit,
           "mt": ab.HistogramManagerMT}[kind]
    return cls(molecule, True, case["width"], 8000)


def _params(case):
    return _capi.DebyeParams(1.0, 1.0, 1.0, 0.0, 0.0, 1.0, case["precision"], 1e-5)


def _assembly_move(case, seed):
    """The assembly, the moved body, and the rotation about its centroid plus shift (at most 5 degrees, about 2 A)."""
    asm = synth.assembly(seed + 40, case["bodies"], case["nmin"], case["nmax"])
    rng = np.random.default_rng(seed)
    body = int(rng.integers(case["bodies"]))
    R = synth.random_rotation(rng, 5.0)
    c = asm.bodies[body].mean(axis=0)
    t = rng.standard_normal(3)
    t *= rng.uniform(0.2, 2.0) / np.linalg.norm(t)
    return asm, body, R, c - R @ c + t


def _calculator_sets(case, seed):
    """A body, its copies under a cyclic symmetry, and the body's waters: float32 records {x, y, z, w}."""
    xyz, ff = synth.globule(97 * seed + 1, case["atoms"])
    w = synth.waters(97 * seed + 2, xyz, ff, case["waters"])
    weights = synth.ff_charge(ff)
    radius = 1.2 * (np.abs(xyz).max() + 2.0) / math.sin(math.pi / case["copies"])
    shift = np.array([radius, 0.0, 0.0])
    copies = []
    for k in range(case["copies"]):
        a = 2 * math.pi * k / case["copies"]
        R = np.array([[math.cos(a), -math.sin(a), 0], [math.sin(a), math.cos(a), 0], [0, 0, 1.0]])
        copies.append(hist.pack((xyz + shift) @ R.T, weights, False))
    return copies, hist.pack(w + shift, np.full(len(w), synth.ff_charge([synth.FF_WATER])[0]), False)


def _calculator_jobs(case):
    """(first set, second set or None, scaling, merge id): the body's own pairs, one representative per class of
    equivalent pairs of copies, the waters against every copy, and the waters' own pairs."""
    n = case["copies"]
    jobs = [(0, None, n, 0)]
    for k in range(1, n // 2 + 1):
        jobs.append((0, k, n // 2 if 2 * k == n else n, 0))
    jobs += [("w", k, n, 1) for k in range(n)]
    jobs.append(("w", None, n, 2))
    return jobs


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind}
    if kind in ("profile", "histogram"):
        st["manager"] = _manager(case, _case_molecule(case, seed))
        st["q"] = _q(case) if case["nq"] else None
        st["precision"] = case["precision"]
        if kind == "histogram":
            st["tot"], st["d_axis"] = np.zeros(8000), np.zeros(8000)
    elif kind == "structure":
        m = _case_molecule(case, seed)
        man = _manager(case, m)
        a, w = m.compact_w() if case["manager"] == "mt" else m.compact_ff()[:2]
        x = m.compact_ff()[2] if case["manager"] == "ffgrid" else None
        st["cfg"] = man.config()
        st["structure"] = _capi.Structure(_capi.default_context(), a, w, x, ff_typed=case["manager"] != "mt")
        st["q"] = torch.from_numpy(_q(case)).cuda()
        st["I"] = torch.zeros(case["nq"], dtype=torch.float64, device="cuda")
        st["params"] = _params(case)
    elif kind == "batch":
        st["batch"] = hist.BatchedProfiles(_batch_molecules(case, seed), bin_width=case["width"])
        st["q"] = _q(case)
        st["precision"] = case["precision"]
    elif kind == "serve":
        asm, body, R, t = _assembly_move(case, seed)
        server = _capi.Server(0)
        q = _q(case)
        cfg = _capi.HistConfig(_capi.MANAGER_FFAVG, 1, 0.25, 8000, VOLUME_PER_ATOM * RHO_WATER)
        params = _capi.DebyeParams(1.0, 1.0, 1.0, 0.0, 0.0, 1.0, 1, 1e-5)
        target = 1e6 * np.exp(-((20.0 * q) ** 2) / 3) + 1e3
        st["id"], _ = server.admit(cfg, [hist.pack(b, f, True) for b, f in zip(asm.bodies, asm.ff)],
                                   [np.zeros((0, 4), np.float32) for _ in asm.bodies], q, params, target=target,
                                   target_err=0.01 * target)
        st["server"], st["body"] = server, body
        st["move"], st["back"] = (R, t), (R.T, -R.T @ t)
    elif kind == "calculator":
        st["copies"], st["waters"] = _calculator_sets(case, seed)
        st["jobs"] = _calculator_jobs(case)
        st["width"] = case["width"]
    elif kind == "fit":
        model = ab.HistogramManagerMTFFAvg(_case_molecule(case, seed), True, case["width"], 8000).calculate_all()
        q = _q(case)
        model.apply_water_scaling_factor(1.0 + 0.05 * (seed % 17))
        _, I = model.debye_transform(q)
        model.apply_water_scaling_factor(1.0)
        noise = np.random.default_rng(seed).standard_normal(len(q))
        st["fitter"] = ab.SmartFitter((q, I * (1 + 0.01 * noise), 0.01 * I), model)
    else:
        xyz, ff = synth.globule(97 * seed + 1, case["atoms"])
        st["axes"] = _capi.hydrate_axes(xyz)
        st["atoms"] = torch.from_numpy(np.ascontiguousarray(xyz)).cuda()
        st["ff"] = torch.from_numpy(ff).cuda()
        st["waters"] = torch.zeros((case["atoms"] + 1024, 3), dtype=torch.float64, device="cuda")
    return st


def run(st):
    kind = st["kind"]
    if kind == "profile":
        return ab.profile(st["manager"], st["q"], precision=st["precision"])
    if kind == "histogram":
        h = st["manager"].calculate_all()
        _, I = h.debye_transform(st["q"])
        # the histogram's length is the structure's largest distance; these go into arrays of one length
        st["tot"][:h.max_bin] = h.get_counts()
        st["d_axis"][:h.max_bin] = h.get_d_axis()
        return {"I": I, "tot": st["tot"], "d_axis": st["d_axis"], "pairs": h.pairs}
    if kind == "structure":
        st["structure"].profile_device(st["cfg"], st["q"], len(st["q"]), st["params"], st["I"])
        return st["I"]
    if kind == "batch":
        return st["batch"].debye_transform(st["q"], precision=st["precision"])
    if kind == "serve":
        s, i = st["server"], st["id"]
        out = {}
        for name in ("move", "back"):
            out[name], out[name + "_fit"] = s.wait(s.submit(i, st["body"], *st[name]), i)
        return out
    if kind == "calculator":
        calc = ab.Calculator(_capi.default_context(), st["width"], 8000)
        points = lambda s: st["waters"] if s == "w" else st["copies"][s]
        for a, b, scaling, merge in st["jobs"]:
            if b is None:
                calc.enqueue_calculate_self(points(a), scaling, merge)
            else:
                calc.enqueue_calculate_cross(points(a), points(b), scaling, merge)
        out = calc.run()
        calc.close()
        return [out[k][i] for k in ("self", "cross") for i in sorted(out[k])]
    if kind == "fit":
        r = st["fitter"].fit("cw")
        return {"parameters": np.array(r.get_parameter_values()), "chi2": r.chi2, "I_fit": r.I_fit}
    n, _ = _capi.hydrate_device(_capi.default_context(), st["atoms"], st["ff"], len(st["ff"]), st["axes"], st["waters"],
                                len(st["waters"]))
    return {"waters": st["waters"], "n": n}


# ---- what a pass cannot do without --------------------------------------------------------------------------------


def _pairs(case):
    n, w = case.get("atoms", 0), case.get("waters", 0)
    kind = case["kind"]
    if kind in ("profile", "structure", "histogram", "fit"):
        p = n * (n - 1) / 2 + n * w + w * (w - 1) / 2
        # dummies of a 1 A grid (about 7.4 per atom) against atoms and waters; their own pairs lie on a lattice and
        # need no distance each
        return p + (7.4 * n * (n + w) if case.get("manager") == "ffgrid" else 0)
    if kind == "batch":
        lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
        mean_square = (math.exp(2 * hi) - math.exp(2 * lo)) / (2 * (hi - lo)) if hi > lo else math.exp(2 * lo)
        return case["structures"] * mean_square * 1.2 * 1.2 / 2
    if kind == "serve":
        mean = (case["nmin"] + case["nmax"]) / 2.5
        return 2 * mean * mean * (case["bodies"] - 0.5)
    if kind == "calculator":
        c = case["copies"]
        return n * n * (0.5 + c // 2) + w * n * c + w * w / 2
    return 0


def work(case):
    kind = case["kind"]
    if kind == "hydrate":
        # 26 candidates per atom, each with 79 probe cells of a byte and a mark; atoms in, waters out
        return {"bytes": case["atoms"] * 28.0 + case["atoms"] * 0.05 * 24, "flops": case["atoms"] * 26.0 * 79}
    nq = case.get("nq") or 100
    width = case.get("width", 0.25)
    atoms = case.get("atoms") or case.get("bodies", 1) * case.get("nmax", 0) // 2
    diameter = 300.0 if atoms > 200000 else 2 * 23.2 * (max(atoms, 1) / 5000.0) ** (1 / 3) + 7
    rows, bins = (3 if case.get("manager") == "mt" else 27), diameter / width
    points = atoms + case.get("waters", 0) + (7.4 * atoms if case.get("manager") == "ffgrid" else 0)
    transforms = 1
    if kind == "batch":
        transforms = case["structures"]
        points = transforms * 1.2 * (case["nmax"] - case["nmin"]) / max(1e-9, math.log(case["nmax"] / case["nmin"]))
        bins = 300
    if kind == "calculator":
        return {"bytes": 16.0 * (points * case["copies"] + case["waters"]) + 3 * 3 * 8000 * 8, "flops": 10 * _pairs(case)}
    if kind == "fit":
        return {"bytes": 8.0 * (rows * bins + 4 * nq), "flops": 2.0 * rows * bins * nq}
    out = 8.0 * nq * transforms + (245 * 8 * bins if kind == "histogram" else 0)
    if kind == "serve":
        out, transforms = 2 * out, 2
    return {"bytes": 16.0 * points + 8.0 * nq + out, "flops": 10 * _pairs(case) + 2.0 * rows * bins * nq * transforms}


# ---- the same in 64 bits ------------------------------------------------------------------------------------------

# five-Gaussian form factors (a, b in s = q / 4 pi units, c) and displaced volumes (A^3) of the types used here
FORM_FACTORS = {
    1: ((0.456221, 3.219608, 0.812773, 2.666928, 1.380927), (21.503498, 13.397134, 34.547137, 5.826620, 0.412902), 0.463202),
    3: ((2.657506, 1.078079, 1.490909, -4.241070, 0.713791), (14.780758, 0.776775, 42.086843, -0.000294, 0.239535), 4.297983),
    7: ((11.893780, 3.277479, 1.858092, 0.858927, 0.912985), (0.000158, 10.232723, 30.344690, 0.656065, 0.217287), -11.804902),
    11: ((2.960427, 2.508818, 0.637853, 0.722838, 1.142756), (14.182259, 5.936858, 0.112726, 34.958481, 0.390240), 0.027014),
    12: ((6.362157, 5.154568, 1.473732, 1.635073, 1.209372), (1.514347, 22.092528, 0.061373, 55.445176, 0.646925), 0.154722),
}
VOLUMES = {1: 20.911, 3: 12.352, 7: 0.027, 11: 14.238, 12: 15.413}


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _form_factor(t, q):
    a, b, c = FORM_FACTORS[t]
    return sum(x * torch.exp(-y / (16 * math.pi ** 2) * q * q) for x, y in zip(a, b)) + c


def _volume_factor(v, q):
    return v * RHO_WATER * torch.exp(-(v ** (2 / 3) / (4 * math.pi)) * q * q)


def _points(xyz):
    """The coordinates a record holds (float32), in 64 bits."""
    return torch.from_numpy(np.ascontiguousarray(xyz, np.float64)).to(torch.float32).to(_device(), torch.float64)


def _pair_histogram(A, rows_a, B, rows_b, n_rows, width, bins, own, weights=None):
    """Counts [n_rows, bins], sums of distances [bins] and of weight products [bins] over the pairs of A and B (own:
    the pairs i < j of A); the row of a pair is rows_a[i] + rows_b[j]."""
    dev = A.device
    counts = torch.zeros(n_rows * bins, dtype=torch.float64, device=dev)
    dsum = torch.zeros(bins, dtype=torch.float64, device=dev)
    wsum = torch.zeros(bins, dtype=torch.float64, device=dev)
    step = max(1, (1 << 25) // max(1, len(B)))
    for i0 in range(0, len(A), step):
        a = A[i0:i0 + step]
        j0 = i0 + 1 if own else 0
        b = B[j0:]
        if not len(b):
            continue
        d = ((a[:, None, 0] - b[None, :, 0]).square_() + (a[:, None, 1] - b[None, :, 1]).square_()
             + (a[:, None, 2] - b[None, :, 2]).square_()).sqrt_()
        k = torch.round(d / width).to(torch.int64)
        keep = None
        if own:
            i = torch.arange(i0, i0 + len(a), device=dev)
            keep = torch.arange(j0, j0 + len(b), device=dev)[None, :] > i[:, None]
        pick = (lambda v: v[keep]) if own else (lambda v: v.reshape(-1))
        kk, dd = pick(k), pick(d)
        dsum += torch.bincount(kk, dd, minlength=bins)
        row = pick((rows_a[i0:i0 + step, None] + rows_b[None, j0:]) * bins + k) if n_rows > 1 else kk
        counts += torch.bincount(row, minlength=n_rows * bins)
        if weights is not None:
            wsum += torch.bincount(kk, pick(weights[0][i0:i0 + step, None] * weights[1][None, j0:]), minlength=bins)
    return counts.reshape(n_rows, bins), dsum, wsum


def _bins(points, width):
    p = torch.cat(points)
    return int(((p.max(0).values - p.min(0).values).norm() / width).item()) + 12


def _axis(dsum, n, width):
    b = torch.arange(len(n), dtype=torch.float64, device=n.device) * width
    return torch.where(n > 0, dsum / n.clamp(min=1), b)


def _sinc(axis, q):
    x = axis[:, None] * q[None, :]
    return torch.where(x < 1e-3, 1 - x * x / 6 + x ** 4 / 120, torch.sin(x) / x.clamp(min=1e-300))


def _cut(n):
    """Bins up to the last one in use, at least ten."""
    used = torch.nonzero(n[10:])
    return 10 if not len(used) else int(used[-1]) + 11


def _intensity(manager, atoms, ff, waters, q, width, z_exv=0.0, dummies=None, weights=None):
    """I(q) and the histograms it is made of."""
    dev = _device()
    A, W = _points(atoms), _points(waters)
    X = None if dummies is None else _points(dummies)
    bins = _bins([p for p in (A, W, X) if p is not None and len(p)], width)
    q = torch.from_numpy(np.asarray(q, np.float64)).to(dev)
    zero_w = torch.zeros(len(W), dtype=torch.int64, device=dev)
    one = lambda t: torch.from_numpy(np.asarray(t, np.float64).astype(np.float32)).to(dev, torch.float64)
    if manager == "mt":
        wa, ww = one(weights[0]), one(weights[1])
        zero_a = torch.zeros(len(A), dtype=torch.int64, device=dev)
        caa, daa, saa = _pair_histogram(A, zero_a, A, zero_a, 1, width, bins, True, (wa, wa))
        caw, daw, saw = _pair_histogram(W, zero_w, A, zero_a, 1, width, bins, False, (ww, wa))
        cww, dww, sww = _pair_histogram(W, zero_w, W, zero_w, 1, width, bins, True, (ww, ww))
        aa, aw, ww_ = 2 * saa, 2 * saw, 2 * sww
        aa[0] += (wa * wa).sum()
        ww_[0] += (ww * ww).sum()
        axis = _axis(daa + daw + dww, (caa + caw + cww)[0], width)
        axis[0] = 0
        I = torch.exp(-q * q) * ((aa + aw + ww_) @ _sinc(axis, q))
        return I, {"tot": aa + aw + ww_, "d_axis": axis}
    types = sorted(set(int(t) for t in np.unique(ff)))
    T = len(types)
    t = torch.from_numpy(np.searchsorted(types, ff)).to(dev)
    caa, daa, _ = _pair_histogram(A, t * T, A, t, T * T, width, bins, True)
    caw, daw, _ = _pair_histogram(A, t, W, zero_w, T, width, bins, False)
    cww, dww, _ = _pair_histogram(W, zero_w, W, zero_w, 1, width, bins, True)
    caa, cww = caa.reshape(T, T, bins), cww[0]
    number = torch.bincount(t, minlength=T).to(torch.float64)
    n = 2 * caa.sum((0, 1)) + caw.sum(0) + 2 * cww
    n[0] += len(A) + len(W)
    axis = _axis(2 * daa + daw + 2 * dww, n, width)
    axis[0] = 0
    S = _sinc(axis, q)
    aa = 2 * caa
    for k in range(T):
        aa[k, k, 0] += number[k]
    ww = 2 * cww
    ww[0] += len(W)
    f = [_form_factor(k, q) for k in types]
    fw = _form_factor(1, q)
    I = sum(f[a] * f[b] * (aa[a, b] @ S) for a in range(T) for b in range(T))
    I = I + sum(2 * f[a] * fw * (caw[a] @ S) for a in range(T)) + fw * fw * (ww @ S)
    rows = {"tot": n, "d_axis": axis}
    if manager == "ffavg":
        fx = torch.exp(-(1.62 ** 2 / 2) * q * q)
        ax = 2 * caa.sum(1) * z_exv
        xx = 2 * caa.sum((0, 1))
        xx[0] += len(A)
        I = I - sum(2 * f[a] * fx * (ax[a] @ S) for a in range(T)) + fx * fx * (z_exv ** 2 * xx @ S)
        I = I - 2 * fx * fw * (z_exv * caw.sum(0) @ S)
    elif manager == "ffexplicit":
        x = [_volume_factor(VOLUMES[k], q) for k in types]
        xw = _volume_factor(VOLUMES[1], q)
        for a in range(T):
            for b in range(T):
                I = I + (x[a] * x[b] - f[a] * x[b] - f[b] * x[a]) * (aa[a, b] @ S)
            I = I - (fw * x[a] + f[a] * xw) * (caw[a] @ S)
    else:
        zero_x = torch.zeros(len(X), dtype=torch.int64, device=dev)
        cax, dax, _ = _pair_histogram(A, t, X, zero_x, T, width, bins, False)
        cwx, dwx, _ = _pair_histogram(W, zero_w, X, zero_x, 1, width, bins, False)
        cxx, dxx, _ = _pair_histogram(X, zero_x, X, zero_x, 1, width, bins, True)
        Sx = _sinc(_axis(dax + dwx, cax.sum(0) + cwx[0], width), q)
        xx = 2 * cxx[0]
        xx[0] += len(X)
        Sxx = _sinc(_axis(2 * dxx, xx, width), q)
        fx = _volume_factor(1.0, q)
        I = I - sum(2 * f[a] * fx * (cax[a] @ Sx) for a in range(T)) - 2 * fx * fw * (cwx[0] @ Sx) + fx * fx * (xx @ Sxx)
    return I, rows


def exact(case, seed):
    kind = case["kind"]
    pairs = _pairs(case)
    if case.get("manager") == "ffgrid":
        pairs += (7.4 * case["atoms"]) ** 2 / 2
    # a search's path, the order in which waters are accepted: nothing a formula gives; beyond 8e9 pairs it takes long
    if kind in ("fit", "hydrate") or pairs > 8e9:
        return None
    if kind == "batch":
        out = []
        for m in _batch_molecules(case, seed):
            out.append(_intensity("ffavg", m.atoms, m.ff_types, m.waters, _q(case), case["width"],
                                  m.volume * RHO_WATER / len(m.atoms))[0].cpu())
        return torch.stack(out)
    if kind == "serve":
        asm, body, R, t = _assembly_move(case, seed)
        q, none = _q(case), np.zeros((0, 3))
        ff = np.concatenate(asm.ff)
        out = {"move_fit": None, "back_fit": None}
        # a body is kept as its float32 records and moved in 64 bits
        kept = [np.asarray(b, np.float32).astype(np.float64) for b in asm.bodies]
        for name in ("move", "back"):
            bodies = list(kept)
            if name == "move":
                bodies[body] = kept[body] @ R.T + t
            out[name] = _intensity("ffavg", np.concatenate(bodies), ff, none, q, 0.25, VOLUME_PER_ATOM * RHO_WATER)[0].cpu()
        return out
    if kind == "calculator":
        copies, w = _calculator_sets(case, seed)
        dev = _device()
        sets = {"w": torch.from_numpy(w).to(dev, torch.float64)}
        sets.update({k: torch.from_numpy(c).to(dev, torch.float64) for k, c in enumerate(copies)})
        zero = {k: torch.zeros(len(v), dtype=torch.int64, device=dev) for k, v in sets.items()}
        bins, out = 8000, {}
        for a, b, scaling, merge in _calculator_jobs(case):
            own = b is None
            c = a if own else b
            r = out.setdefault((0 if own else 1, merge), [torch.zeros(bins, dtype=torch.float64, device=dev) for _ in range(3)])
            n, d, v = _pair_histogram(sets[a], zero[a], sets[c], zero[c], 1, case["width"], bins, own,
                                      (sets[a][:, 3], sets[c][:, 3]))
            for x, y in zip(r, (v, n[0], d)):
                x += 2 * scaling * y
            if own:
                square = (sets[a][:, 3] ** 2).sum() * scaling
                r[0][0] += square
                r[1][0] += torch.floor(square)
        return [tuple(x.cpu() for x in out[k]) for k in sorted(out)]
    m = _case_molecule(case, seed)
    q = hist.default_q_axis() if not case["nq"] else _q(case)
    I, rows = _intensity(case["manager"], m.atoms, m.ff_types, m.waters, q, case["width"],
                         m.volume * RHO_WATER / len(m.atoms), m.exv, (m.weights, m.water_weights))
    if kind != "histogram":
        return I.cpu()
    m = _cut(rows["tot"])
    out = {"I": I.cpu(), "pairs": None}
    for name in ("tot", "d_axis"):
        out[name] = torch.zeros(8000, dtype=torch.float64)
        out[name][:m] = rows[name][:m].cpu()
    return out
