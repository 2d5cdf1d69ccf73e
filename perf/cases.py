"""The work that a user of this framework has it do, as cases to be timed.

Six calls make up the framework's use, and each has cases over its range:

  forces      the forces of a term on lists in force, at new positions: an
              outer program (its own integrator, a sampler) drives the term
  evaluate    a configuration never seen before: the neighbor build, forces,
              energies and virials (analysis of stored frames, minimizers,
              Monte Carlo)
  md          a trajectory frame's worth of MD steps through `Simulation`,
              from a state that the program holds
  gradient    force matching: the forces of a batch of frames through
              `mdir_b200.torch.forces`, and the gradient of the loss in every
              sigma, epsilon and charge
  energies    energies of frames through `mdir_b200.torch.evaluate` and their
              gradient in the parameters and the positions
  batch       many uneven solvated systems at once through `BatchEvaluator`

Inputs are liquids, not lattices: water boxes are brought near equilibrium by
a short deterministic dynamics here (torch, no code of the framework), large
ones by tiling a smaller equilibrated one, as programs that set up boxes do.
`exact` restates the sums in 64 bits with plain torch."""

import functools
import math

import numpy as np
import torch

from mdir_b200 import (Ensemble, Execution, FrameEvaluator, InitialState, Integrator,
                       NonbondedTerm, Schedule, Simulation, System, compile)
from mdir_b200 import torch as mtorch
from mdir_b200.batch import BatchEvaluator

F_COUL = float.fromhex("0x1.15def44ac2182p+7")  # kJ mol^-1 nm e^-2
KB = 0.0083144626181532
DENSITY = 33.4  # waters a nm^3
ROH, THETA = 0.09572, math.radians(104.52)
RHH = 2.0 * ROH * math.sin(THETA / 2.0)
Q_O, Q_H, SIG_O, EPS_O = -0.834, 0.417, 0.315061, 0.6364
M_O, M_H = 15.9994, 1.008
CUTOFF = 0.9
DEV = "cuda"


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # The smallest call: LJ forces of the argon box at new positions, all
        # launches and latency.
        {"name": "forces-argon-864", "kind": "forces", "argon": 6, "skin": 0.1, "switch": 2},
        # A term driven from outside at the headline size, lists with the
        # default skin, forces alone.
        {"name": "forces-water-23550", "kind": "forces", "waters": 7850, "tiles": 1, "skin": 0.1, "order": 4,
         "deterministic": False},
        # One small solvated configuration evaluated once: the build, the
        # sums and the energies read back (a minimizer's or a sampler's call).
        {"name": "evaluate-water-900", "kind": "evaluate", "waters": 300, "tiles": 1, "tilt": 0, "skin": 0.1,
         "order": 4, "deterministic": False},
        # A triclinic cell (the tilts of a truncated octahedron) evaluated
        # once; its grid is no power of two.
        {"name": "evaluate-octahedron-23490", "kind": "evaluate", "waters": 290, "tiles": 3, "tilt": 2, "skin": 0.1,
         "order": 4, "deterministic": False},
        # The large box evaluated once.
        {"name": "evaluate-water-1070091", "kind": "evaluate", "waters": 13211, "tiles": 3, "tilt": 0, "skin": 0.1,
         "order": 4, "deterministic": False},
        # MD of the smallest system in use, no electrostatics: every step is
        # latency.
        {"name": "md-argon-864", "kind": "md", "argon": 6, "skin": 0.2, "pruned": 0.05, "switch": 2, "steps": 500,
         "verlet": True},
        # MD of a small water box on a grid that is no power of two, launch
        # shapes as they come.
        {"name": "md-water-8013", "kind": "md", "waters": 2671, "tiles": 1, "skin": 0.5, "pruned": 0.1, "order": 4,
         "deterministic": False, "steps": 100, "sms": 0},
        # The headline: the 23,550-atom TIP3P box at the reaches and the
        # launch shape that the tuner settles on for it.
        {"name": "md-water-23550", "kind": "md", "waters": 7850, "tiles": 1, "skin": 0.8, "pruned": 0.125, "order": 4,
         "deterministic": False, "steps": 100, "sms": 128},
        # The precision form: the large box in the deterministic mode.
        {"name": "md-water-1070091-fixed", "kind": "md", "waters": 13211, "tiles": 3, "skin": 0.7, "pruned": 0.125,
         "order": 4, "deterministic": True, "steps": 20, "sms": 0},
        # The differentiation form: one force-matching step over 64 frames of
        # the headline box (8 LJ types and every charge).
        {"name": "gradient-64x23550", "kind": "gradient", "waters": 7850, "frames": 64, "types": 8},
        # Energies of a few small frames with the gradients in the parameters
        # and the positions (a fit to energies).
        {"name": "energies-8x3000", "kind": "energies", "waters": 1000, "frames": 8, "types": 4},
        # The batching form: 256 uneven solvated systems of 1,000 to 8,000
        # atoms, each in a cell of its own, new positions built and evaluated.
        {"name": "batch-256", "kind": "batch", "frames": 256, "low": 1000, "high": 8000, "types": 8},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _box(rng, high):
    """Waters of a base box and its tiles a side, `high` waters at most."""
    total = _log(rng, 210, high)
    if total <= 9000:
        return total, 1
    tiles = 2 if total <= 72000 else 3
    return total // tiles ** 3, tiles


def draw(rng):
    kind = rng.choice(["forces", "forces", "evaluate", "evaluate", "md", "md", "md", "gradient", "energies", "batch"])
    mode = rng.random() < 0.3
    order = rng.choice([4, 4, 4, 4, 5, 6, 8])
    if kind in ("forces", "md") and rng.random() < 0.2:
        cells = rng.randint(5, 14)
        if kind == "forces":
            return {"kind": kind, "argon": cells, "skin": round(rng.uniform(0.08, 0.2), 3), "switch": rng.randint(0, 2)}
        return {"kind": kind, "argon": cells, "skin": round(rng.uniform(0.15, 0.3), 3), "pruned": 0.05,
                "switch": rng.randint(0, 2), "steps": rng.randint(150, 500), "verlet": rng.random() < 0.5}
    if kind == "forces":
        waters, tiles = _box(rng, 200000)
        return {"kind": kind, "waters": waters, "tiles": tiles, "skin": round(rng.uniform(0.08, 0.15), 3),
                "order": order, "deterministic": mode}
    if kind == "evaluate":
        waters, tiles = _box(rng, 200000)
        tilt = rng.choice([0, 0, 1, 2])
        if tilt:  # a triclinic cell is cut from a tiled cubic box
            waters, tiles = rng.randint(210, 1200), tilt + 1
        return {"kind": kind, "waters": waters, "tiles": tiles, "tilt": tilt, "skin": round(rng.uniform(0.08, 0.15), 3),
                "order": order, "deterministic": mode}
    if kind == "md":
        waters, tiles = _box(rng, 100000)
        waters = max(waters, 400)
        edge = tiles * (waters / DENSITY) ** (1 / 3)
        skin = min(round(rng.uniform(0.4, 0.8), 3), round(0.95 * edge - CUTOFF, 3))
        steps = max(10, min(125, int(4.0e6 / (waters * tiles ** 3))))
        return {"kind": kind, "waters": waters, "tiles": tiles, "skin": skin, "pruned": round(rng.uniform(0.08, 0.15), 3),
                "order": order, "deterministic": mode, "steps": steps, "sms": rng.choice([0, 0, 128])}
    if kind == "gradient":
        waters = _log(rng, 400, 9000)
        return {"kind": kind, "waters": waters, "frames": rng.randint(2, 40), "types": rng.randint(2, 12)}
    if kind == "energies":
        waters = _log(rng, 300, 9000)
        return {"kind": kind, "waters": waters, "frames": rng.randint(1, 10), "types": rng.randint(2, 12)}
    low = _log(rng, 900, 3000)
    return {"kind": kind, "frames": _log(rng, 3, 100), "low": low, "high": low + rng.randint(300, 5000),
            "types": rng.randint(2, 12)}


# ---------------------------------------------------------------- the inputs

def _ewald_beta(rc=CUTOFF, tol=1e-5):
    low, high = 0.0, 1.0
    while math.erfc(high * rc) > tol:
        high *= 2.0
    for _ in range(100):
        mid = 0.5 * (low + high)
        low, high = (mid, high) if math.erfc(mid * rc) > tol else (low, mid)
    return 0.5 * (low + high)


def _grid(box, order):
    """The smallest even 2,3,5,7-smooth size of at most 0.1 nm a point, per edge."""
    out = []
    for edge in box:
        size = max(int(math.ceil(edge / 0.1 - 1e-9)), 2 * order)
        while True:
            rest = size
            for f in (2, 3, 5, 7):
                while rest % f == 0:
                    rest //= f
            if size % 2 == 0 and rest == 1:
                break
            size += 1
        out.append(size)
    return out


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _rigid(p):
    """Sites (n, 3, 3) near a water's shape onto it, in f64."""
    p = p.double()
    m = torch.tensor([M_O, M_H, M_H], dtype=torch.float64, device=p.device)
    com = (p * m[:, None]).sum(1) / m.sum()
    bis = _unit(0.5 * (p[:, 1] + p[:, 2]) - p[:, 0])
    across = p[:, 1] - p[:, 2]
    across = _unit(across - (across * bis).sum(-1, keepdim=True) * bis)
    h = ROH * math.cos(THETA / 2)
    d = 2 * M_H * h / (M_O + 2 * M_H)
    o = com - d * bis
    mid = o + h * bis
    return torch.stack([o, mid + 0.5 * RHH * across, mid - 0.5 * RHH * across], 1)


@functools.lru_cache(maxsize=2)
def _liquid(waters, seed):
    """Sites (waters, 3, 3) f64 of a periodic water box near equilibrium and
    its edge.  Flexible waters of heavy hydrogens with a shifted-force
    Coulomb sum run for some hundred short steps at 300 K; only gathers and
    row sums, so that the same seed gives the same box."""
    g = torch.Generator().manual_seed(seed)
    edge = (waters / DENSITY) ** (1 / 3)
    m = math.ceil(waters ** (1 / 3) - 1e-9)
    pick = torch.randperm(m ** 3, generator=g)[:waters].sort().values
    site = torch.stack([pick // (m * m), (pick // m) % m, pick % m], 1).double()
    centre = (site + 0.5) * (edge / m) + 0.02 * (2 * torch.rand(waters, 3, generator=g).double() - 1)
    e1 = _unit(torch.randn(waters, 3, generator=g).double())
    e2 = torch.randn(waters, 3, generator=g).double()
    e2 = _unit(e2 - (e2 * e1).sum(-1, keepdim=True) * e1)
    h = ROH * math.cos(THETA / 2)
    p = torch.stack([centre, centre + h * e1 + 0.5 * RHH * e2, centre + h * e1 - 0.5 * RHH * e2], 1)
    p = p.float().to(DEV)
    mass = torch.tensor([16.0, 4.0, 4.0], device=DEV)[None, :, None]
    q = torch.tensor([Q_O, Q_H, Q_H], device=DEV)
    qq = F_COUL * q[:, None] * q[None, :]
    v = torch.randn(waters, 3, 3, generator=g).to(DEV) * torch.sqrt(KB * 300.0 / mass)
    rc, rlist, dt, steps, every = 0.6, 0.72, 0.001, 400, 20
    nb = live = None
    for k in range(steps):
        if k % every == 0:
            o = p[:, 0]
            near = []
            for a in range(0, waters, 2048):
                d = o[a:a + 2048, None] - o[None]
                d = d - edge * torch.round(d / edge)
                near.append((d * d).sum(-1) < rlist * rlist)
            near = torch.cat(near)
            near.fill_diagonal_(False)
            count = near.sum(1)
            width = max(int(count.max()), 1)
            row, col = near.nonzero(as_tuple=True)
            at = torch.arange(len(row), device=DEV) - (count.cumsum(0) - count)[row]
            nb = torch.zeros(waters, width, dtype=torch.int64, device=DEV)
            nb[row, at] = col
            live = torch.arange(width, device=DEV)[None] < count[:, None]
            del near, row, col, at
        pj = p[nb]  # (n, width, 3 sites, 3)
        doo = p[:, None, 0] - pj[:, :, 0]
        pj = pj + (edge * torch.round(doo / edge))[:, :, None]
        d = p[:, None, :, None] - pj[:, :, None, :]  # (n, width, site, partner's site, 3)
        r2 = (d * d).sum(-1).clamp_min(0.01)
        r = r2.sqrt()
        fr = torch.where(r < rc, qq * (1 / r2 - 1 / rc ** 2) / r, 0.0)
        s6 = (SIG_O ** 2 / r2[:, :, 0, 0]) ** 3
        fr[:, :, 0, 0] += torch.where(r[:, :, 0, 0] < rc, 24 * EPS_O * (2 * s6 * s6 - s6) / r2[:, :, 0, 0], 0.0)
        fr = fr * live[:, :, None, None]
        f = (fr[..., None] * d).sum((1, 3))
        for a, b, rest, stiff in ((0, 1, ROH, 2.0e5), (0, 2, ROH, 2.0e5), (1, 2, RHH, 1.0e5)):
            dab = p[:, a] - p[:, b]
            rab = dab.norm(dim=-1, keepdim=True)
            fab = -stiff * (rab - rest) / rab * dab
            f[:, a] += fab
            f[:, b] -= fab
        v = v + dt * f / mass
        t = (mass * v * v).sum() / (9 * waters * KB)
        v = v * torch.sqrt(300.0 / t).clamp(0.2, 1.1)
        v = v.clamp(-4.0, 4.0)
        p = p + dt * v
    return _rigid(p), edge


def _tiled(waters, tiles, seed):
    """Sites (tiles^3 waters, 3, 3) of the liquid tiled `tiles` times a side, and the edge."""
    p, edge = _liquid(waters, seed)
    if tiles == 1:
        return p.clone(), edge
    a = torch.arange(tiles, device=DEV, dtype=torch.float64) * edge
    shift = torch.stack(torch.meshgrid(a, a, a, indexing="ij"), -1).reshape(-1, 1, 1, 3)
    return (p[None] + shift).reshape(-1, 3, 3), edge * tiles


def _rigid_velocities(p, temperature, seed):
    """Maxwell velocities of rigid waters: the part of atomic ones that moves and turns each as a body."""
    g = torch.Generator().manual_seed(seed + 77)
    m = torch.tensor([M_O, M_H, M_H], dtype=torch.float64, device=p.device)[None, :, None]
    v = torch.randn(p.shape, generator=g, dtype=torch.float64).to(p.device) * torch.sqrt(KB * temperature / m)
    total = m.sum()
    com, vcom = (m * p).sum(1, keepdim=True) / total, (m * v).sum(1, keepdim=True) / total
    r = p - com
    ang = (m * torch.linalg.cross(r, v - vcom)).sum(1)
    eye = torch.eye(3, dtype=torch.float64, device=p.device)
    inertia = ((m * (r * r).sum(-1, keepdim=True)).sum(1)[:, :, None] * eye
               - torch.einsum("nia,nib,i->nab", r, r, m[0, :, 0]))
    w = torch.linalg.solve(inertia, ang)
    v = vcom + torch.linalg.cross(w[:, None].expand_as(r), r)
    return v - (m * v).sum((0, 1)) / (total * len(p))


def _mix(sig, eps):
    sig, eps = np.asarray(sig, dtype=np.float64), np.asarray(eps, dtype=np.float64)
    return 0.5 * (sig[:, None] + sig[None]), np.sqrt(eps[:, None] * eps[None])


def _water_system(sites, box, skin, order=4, cell=None):
    """The dict of mdir_b200.systems for TIP3P waters (cell: its tilts besides)."""
    n = len(sites)
    sigma, epsilon = _mix([SIG_O, 0.1], [EPS_O, 0.0])
    o = 3 * np.arange(n)
    excluded = np.concatenate([np.stack([o, o + 1], 1), np.stack([o, o + 2], 1), np.stack([o + 1, o + 2], 1)])
    return {"charges": np.tile([Q_O, Q_H, Q_H], n), "types": np.tile([0, 1, 1], n).astype(np.int32),
            "sigma": sigma, "epsilon": epsilon, "masses": np.tile([M_O, M_H, M_H], n), "box": np.asarray(box),
            "cutoff": CUTOFF, "reach": CUTOFF + skin, "pme": True, "beta": _ewald_beta(), "grid": _grid(box, order),
            "order": order, "excluded_pairs": excluded, "waters": np.stack([o, o + 1, o + 2], 1),
            "dispersion": False, "lj_switch": 0, "switch": 0.0}


def _argon_system(case, seed):
    """Argon at the density of the 864-atom box, near its lattice; positions."""
    cells = case["argon"]
    edge = 3.47 * cells / 6
    rng = np.random.default_rng(seed)
    base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    idx = np.stack(np.meshgrid(*[np.arange(cells)] * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    x = ((idx + base).reshape(-1, 3) + 0.25) * (edge / cells)
    x = x + rng.uniform(-0.02, 0.02, x.shape)
    sigma, epsilon = _mix([0.3405], [0.996])
    n = len(x)
    cutoff = 0.85
    return {"charges": np.zeros(n), "types": np.zeros(n, dtype=np.int32), "sigma": sigma, "epsilon": epsilon,
            "masses": np.full(n, 39.948), "box": np.full(3, edge), "cutoff": cutoff, "reach": cutoff + case["skin"],
            "pme": False, "beta": 0.0, "grid": None, "order": 4, "excluded_pairs": np.zeros((0, 2), dtype=np.int64),
            "waters": None, "dispersion": True, "lj_switch": case["switch"], "switch": 0.75}, x


def _cell(case, edge):
    """The cell (3 or 6 numbers) of an evaluate case whose cubic box has this edge."""
    tiles = case["tiles"]
    s = edge / tiles
    if case["tilt"] == 1:  # two cubes a side, the tilts at half an edge
        return np.array([edge, edge, edge, s, s, s])
    if case["tilt"] == 2:  # three cubes a side, the tilts of a truncated octahedron
        return np.array([edge, edge, edge, s, -s, s])
    return np.array([edge, edge, edge])


def _system(case, seed):
    """(system, positions (n, 3) f64 tensor, cell) of a forces, evaluate or md case."""
    if "argon" in case:
        s, x = _argon_system(case, seed)
        return s, torch.as_tensor(x, device=DEV), s["box"]
    sites, edge = _tiled(case["waters"], case["tiles"], seed)
    cell = _cell(case, edge) if case["kind"] == "evaluate" else np.full(3, edge)
    s = _water_system(sites, cell[:3], case["skin"], case["order"])
    return s, sites.reshape(-1, 3).contiguous(), cell


def _term(s, deterministic):
    t = NonbondedTerm(len(s["charges"]))
    t.set_particles(s["charges"], s["types"], s["sigma"], s["epsilon"])
    t.set_exclusions(pairs=s["excluded_pairs"])
    t.set_interaction(s["cutoff"], s["reach"], s["beta"], lj_switch=s["lj_switch"], switch_distance=s["switch"])
    if s["pme"]:
        t.set_pme(s["grid"], s["order"])
    t.set_deterministic(deterministic)
    return t


def _moved(x, scale, seed, frames=None):
    """x with every coordinate moved by N(0, scale) (frames of it)."""
    g = torch.Generator().manual_seed(seed + 31)
    shape = x.shape if frames is None else (frames, *x.shape)
    return x + scale * torch.randn(shape, generator=g, dtype=torch.float64).to(x.device)


def _frames_system(case, seed):
    """A water box whose oxygens take `types` LJ types of differing sigma and
    epsilon, and frames of it; (system, X (K, n, 3), sigma, epsilon, charges)."""
    types = case["types"]
    sites, edge = _liquid(case["waters"], seed)
    skin = min(0.1, 0.95 * edge - CUTOFF)
    s = _water_system(sites, np.full(3, edge), skin)
    n = len(sites)
    rng = np.random.default_rng(seed + 5)
    t = np.full(3 * n, types, dtype=np.int32)
    t[0::3] = np.arange(n) % types
    sig = np.append(SIG_O * (1 + 0.02 * rng.standard_normal(types)), 0.1)
    eps = np.append(EPS_O * (1 + 0.05 * rng.standard_normal(types)), 0.0)
    sigma, epsilon = _mix(sig, eps)
    s.update({"types": t, "sigma": sigma, "epsilon": epsilon})
    X = _moved(sites.reshape(-1, 3), 0.005, seed, case["frames"])
    return s, X, sig, eps, s["charges"]


def _solvated(case, seed):
    """The frames of a batch case: cubes cut whole molecules at a time from
    one liquid, with room at their faces, one molecule in twenty a solute (its
    centre of one of the solute types, its charges drawn)."""
    sizes = np.random.default_rng(case["frames"])  # the systems' sizes belong to the case, not to its inputs
    atoms = 3 * sizes.integers(case["low"] // 3, case["high"] // 3 + 1, size=case["frames"])
    rng = np.random.default_rng(seed + 9)
    waters = max(int(atoms.max()) // 3 + 200, 1500)
    sites, edge = _liquid(waters, seed)
    sites = sites.cpu().numpy()
    types = case["types"]
    sig = np.concatenate([[SIG_O], rng.uniform(0.25, 0.33, types - 1), [0.1]])
    eps = np.concatenate([[EPS_O], rng.uniform(0.2, 1.0, types - 1), [0.0]])
    sigma, epsilon = _mix(sig, eps)
    out = []
    for a in atoms:
        m = int(a) // 3
        d = sites - rng.uniform(0, edge, 3)
        d -= edge * np.round(d[:, :1] / edge)
        far = np.abs(d).max((1, 2))
        keep = np.sort(np.argpartition(far, m - 1)[:m])
        x = d[keep]
        box = 2 * far[keep].max() + 0.24
        s = _water_system(x, np.full(3, box), 0.1)
        q, t = s["charges"].reshape(m, 3).copy(), np.tile(np.array([0, types, types], dtype=np.int32), (m, 1))
        solute = rng.permutation(m)[:max(1, m // 20)]
        qs = rng.normal(0.0, 0.3, (len(solute), 3))
        q[solute] = qs - qs.mean(1, keepdims=True)
        t[solute, 0] = 1 + rng.integers(0, types - 1, len(solute))
        s.update({"charges": q.reshape(-1), "types": t.reshape(-1), "sigma": sigma, "epsilon": epsilon,
                  "positions": x.reshape(-1, 3) + 0.5 * box})
        out.append(s)
    return out


def _start_velocities(case, x, seed):
    if "argon" in case:
        g = torch.Generator().manual_seed(seed + 77)
        return torch.randn(x.shape, generator=g, dtype=torch.float64).to(DEV) * math.sqrt(KB * 94.4 / 39.948)
    return _rigid_velocities(x.reshape(-1, 3, 3), 300.0, seed).reshape(-1, 3).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("forces", "evaluate"):
        s, x, cell = _system(case, seed)
        t = _term(s, case.get("deterministic", False))
        if kind == "forces":
            t.build(x, cell)
            x = _moved(x, 0.003, seed)  # somewhat moved since the build, as between two builds
        return {"kind": kind, "term": t, "x": x, "cell": cell}
    if kind == "md":
        s, x, cell = _system(case, seed)
        v = _start_velocities(case, x, seed)
        system = System.from_dict(s)
        system.pruned_distance = s["cutoff"] + case["pruned"]
        it, ens, ex = Integrator(), Ensemble(), Execution()
        it.timestep = 0.002
        if case.get("verlet"):
            it.method = "VELOCITY_VERLET"
        ex.deterministic = case.get("deterministic", False)
        ex.pair_sms = case.get("sms", 0)
        state = InitialState(x.cpu().numpy(), v.cpu().numpy(), cell)
        sim = Simulation(compile(system, state, it, ens, ex, Schedule()))
        return {"kind": kind, "sim": sim, "x": x, "v": v, "steps": case["steps"]}
    if kind in ("gradient", "energies"):
        s, X, sig, eps, q = _frames_system(case, seed)
        ev = FrameEvaluator(s, sigma=sig, epsilon=eps, charges=q)
        theta = [torch.tensor(a, dtype=torch.float64, device=DEV, requires_grad=True) for a in (sig, eps, q)]
        st = {"kind": kind, "ev": ev, "theta": theta, "X": X}
        if kind == "gradient":
            st["target"] = _targets(X, seed)
        else:
            X.requires_grad_(True)
        # the fit is under way: its first step opened the evaluator's lanes
        run(st)
        torch.cuda.synchronize()
        return st
    frames = _solvated(case, seed)
    ev = BatchEvaluator(frames)
    return {"kind": kind, "ev": ev, "x": ev.x.clone()}


def _targets(X, seed):
    """Reference forces of the frames; the spread of forces in liquid water."""
    g = torch.Generator(device=DEV).manual_seed(seed + 13)
    return 600.0 * torch.randn(X.shape, generator=g, dtype=torch.float64, device=DEV)


# ---------------------------------------------------------------- the calls

TERMS = ("lj", "coulomb", "excluded", "reciprocal")


def run(state):
    kind = state["kind"]
    if kind == "forces":
        return state["term"].force(state["x"])
    if kind == "evaluate":
        t = state["term"]
        t.build(state["x"], state["cell"])
        forces = t.force(state["x"], energy=True)
        return forces, t.energies()
    if kind == "md":
        sim = state["sim"]
        sim.set_state(state["x"], state["v"])
        sim.run(state["steps"])
        return sim.x, sim.v
    if kind == "gradient":
        sigma, epsilon, charges = state["theta"]
        forces = mtorch.forces(state["ev"], sigma, epsilon, charges, state["X"])
        loss = ((forces - state["target"]) ** 2).sum() / len(state["X"])
        grads = torch.autograd.grad(loss, (sigma, epsilon, charges))
        return forces.detach(), loss.detach(), grads
    if kind == "energies":
        sigma, epsilon, charges = state["theta"]
        e = mtorch.evaluate(state["ev"], {"sigma": sigma, "epsilon": epsilon, "charges": charges}, state["X"])
        grads = torch.autograd.grad(e.sum(), (sigma, epsilon, charges, state["X"]))
        return e.detach(), grads
    ev = state["ev"]
    ev.set_positions(state["x"])
    ev.build()
    forces = ev.force(energy=True)
    e = ev.energies()
    return forces, {k: e[k] for k in TERMS + ("potential", "virial_pair", "virial_reciprocal")}


# ------------------------------------------------------- work and tolerance

def _atoms(case):
    if "argon" in case:
        return 4 * case["argon"] ** 3
    return 3 * case["waters"] * case.get("tiles", 1) ** 3


def _atoms_of(case):
    return case["high"] if case["kind"] == "batch" else _atoms(case)


def _force_flops(atoms, rho, cutoff, order, points):
    """50 a pair within the cutoff; spreading and gathering 2 and 6 a grid
    point of an atom; two real transforms and the multiplication."""
    pairs = 0.5 * atoms * rho * 4 / 3 * math.pi * cutoff ** 3
    pme = atoms * 8 * order ** 3 + points * (5 * math.log2(points) + 3) if points else 0
    return 50 * pairs + pme


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = case["frames"] * 0.5 * (case["low"] + case["high"])
        return {"bytes": n * (24 + 24 + 8), "flops": _force_flops(n, 80.0, CUTOFF, 4, 1.3 * n * 10)}
    n = _atoms(case)
    if "argon" in case:
        one = _force_flops(n, 864 / 3.47 ** 3, 0.85, 0, 0)
    else:
        edge = (n / (3 * DENSITY)) ** (1 / 3)
        order = case.get("order", 4)
        one = _force_flops(n, 3 * DENSITY, CUTOFF, order, float(np.prod(_grid([edge] * 3, order))))
    if kind == "md":
        return {"bytes": n * 96, "flops": case["steps"] * (one + 150 * n)}
    if kind in ("gradient", "energies"):
        return {"bytes": case["frames"] * n * (24 + 24 + 24), "flops": 2 * case["frames"] * one}
    return {"bytes": n * (24 + 24 + 8), "flops": one}


def tolerance(case):
    """About four times the error against 64 bits that was seen over the
    range (f32 pair terms and frames, f64 sums).  The f32 frames of a large
    cell round coarser; a liquid's trajectories part exponentially, twice as
    far about every ten steps."""
    if case["kind"] == "md":
        parted = 4e-4 * 2.0 ** ((case["steps"] - 100) / 10) if "waters" in case else 0.0
        return {"rel": max(4e-5, parted)}
    return {"rel": 4e-5 if _atoms_of(case) > 100000 else 1.5e-5}


# ------------------------------------------------------------- in 64 bits

def _image(d, cell):
    """The minimum image of displacements in the cell (along c, then b, then a)."""
    n = torch.round(d[..., 2] / cell[2])
    d0, d1, d2 = d[..., 0] - n * cell[4], d[..., 1] - n * cell[5], d[..., 2] - n * cell[2]
    n = torch.round(d1 / cell[1])
    d0, d1 = d0 - n * cell[3], d1 - n * cell[1]
    return torch.stack([d0 - torch.round(d0 / cell[0]) * cell[0], d1, d2], -1)


def _pairs(x, cell, reach):
    """Batches (i, j) of every pair i < j within the reach."""
    n = len(x)
    side = [int(cell[k] / reach) for k in range(3)]
    if n <= 40000 or min(side) < 3 or any(cell[3:]):
        step = max(1, int(4.0e8 / (24 * n)))
        for a in range(0, n, step):
            xa = x[a:a + step]
            d = _image(xa[:, None] - x[None, a:], cell)
            near = ((d * d).sum(-1) < reach * reach).triu(1)
            i, j = near.nonzero(as_tuple=True)
            yield i + a, j + a
        return
    edges = torch.tensor(cell[:3], device=x.device, dtype=torch.float64)
    dims = torch.tensor(side, device=x.device)
    c3 = torch.minimum(((x / edges - torch.floor(x / edges)) * dims).long(), dims - 1)
    key = (c3[:, 0] * side[1] + c3[:, 1]) * side[2] + c3[:, 2]
    order = key.argsort()
    count = torch.bincount(key, minlength=side[0] * side[1] * side[2])
    start = count.cumsum(0) - count
    most, wide = int(count.max()), 16
    for off in range(14):  # the cell itself and half of its neighbors
        o = off + 13
        shift = torch.tensor([o // 9 - 1, o // 3 % 3 - 1, o % 3 - 1], device=x.device)
        c = torch.remainder(c3 + shift, dims)
        other = (c[:, 0] * side[1] + c[:, 1]) * side[2] + c[:, 2]
        for k in range(0, most, wide):
            slot = torch.arange(k, k + wide, device=x.device)
            ok = slot[None] < count[other][:, None]
            j = order[(start[other][:, None] + slot[None]).clamp_max(n - 1)]
            if off == 0:
                ok &= j > torch.arange(n, device=x.device)[:, None]
            d = _image(x[:, None] - x[j], cell)
            ok &= (d * d).sum(-1) < reach * reach
            i, s = ok.nonzero(as_tuple=True)
            yield i, j[i, s]


def _pair_terms(d, qq, sig, eps, p):
    """(force on i / d, LJ energy, Coulomb energy) of pairs with displacements d."""
    r2 = (d * d).sum(-1)
    r = r2.sqrt()
    on = (r < p["cutoff"]).double()
    s6 = (sig * sig / r2) ** 3
    u = 4 * eps * (s6 * s6 - s6)
    du = 24 * eps * (s6 - 2 * s6 * s6) / r  # dU/dr
    if p["lj_switch"] == 1:
        a, c = p["switch"] ** 2, p["cutoff"] ** 2
        y = ((r2 - a) / (c - a)).clamp(0, 1)
        du = du * (1 - y) ** 2 * (1 + 2 * y) + u * (-6 * y * (1 - y)) / (c - a) * 2 * r
        u = u * (1 - y) ** 2 * (1 + 2 * y)
    elif p["lj_switch"] == 2:
        t = ((r - p["switch"]) / (p["cutoff"] - p["switch"])).clamp(0, 1)
        w = 1 - 10 * t ** 3 + 15 * t ** 4 - 6 * t ** 5
        du = du * w + u * (-30 * t ** 2 + 60 * t ** 3 - 30 * t ** 4) / (p["cutoff"] - p["switch"])
        u = u * w
    b = p["beta"]
    er = torch.erfc(b * r)
    fc = F_COUL * qq * (er / r + 2 * b / math.sqrt(math.pi) * torch.exp(-(b * r) ** 2)) / r2
    return on * (fc - du / r), on * u, on * F_COUL * qq * er / r


def _spline(t, order):
    """Weights M_p(t + j) and slopes, j = 0 .. p - 1; (n, p) each."""
    a = [t, 1 - t] + [torch.zeros_like(t)] * (order - 2)
    slope = None
    for m in range(3, order + 1):
        prev = a
        if m == order:
            slope = [(prev[j] if j < m - 1 else 0 * t) - (prev[j - 1] if j > 0 else 0 * t) for j in range(order)]
        a = [((t + j) * (prev[j] if j < m - 1 else 0 * t) + (m - t - j) * (prev[j - 1] if j > 0 else 0 * t)) / (m - 1)
             if j < m else 0 * t for j in range(order)]
    return torch.stack(a, 1), torch.stack(slope, 1)


def _moduli(size, order):
    m_int, _ = _spline(torch.zeros(1, dtype=torch.float64), order)
    k = torch.arange(size, dtype=torch.float64)
    arg = 2 * math.pi * k[:, None] * torch.arange(order - 1, dtype=torch.float64)[None] / size
    s = (m_int[0, 1:] * torch.cos(arg)).sum(1) ** 2 + (m_int[0, 1:] * torch.sin(arg)).sum(1) ** 2
    b = torch.where(s < 1e-7, torch.zeros_like(s), 1 / s)
    mean = 0.5 * (b.roll(1) + b.roll(-1))
    return torch.where(b == 0, mean, b)


def _reciprocal(x, q, cell, grid, order, beta):
    """Smooth PME: (energy, forces, virial, potential at the atoms); differentiable in q."""
    dev = x.device
    ax, by, cz, bx, cx, cy = cell
    H = torch.tensor([[ax, 0, 0], [bx, by, 0], [cx, cy, cz]], dtype=torch.float64, device=dev)
    inv = torch.linalg.inv(H)
    K = torch.tensor(grid, device=dev)
    u = x @ inv
    u = (u - torch.floor(u)) * K
    k0 = torch.floor(u)
    w, dw = zip(*[_spline(u[:, a] - k0[:, a], order) for a in range(3)])
    back = torch.arange(order, device=dev)
    at = [torch.remainder(k0[:, a].long()[:, None] - back[None], int(grid[a])) for a in range(3)]
    Q = torch.zeros(int(np.prod(grid)), dtype=torch.float64, device=dev)
    step = max(1, 30_000_000 // order ** 3)
    parts = []
    for s in range(0, len(x), step):
        e = slice(s, s + step)
        idx = ((at[0][e][:, :, None, None] * grid[1] + at[1][e][:, None, :, None]) * grid[2]
               + at[2][e][:, None, None, :])
        wt = w[0][e][:, :, None, None] * w[1][e][:, None, :, None] * w[2][e][:, None, None, :]
        Q = Q.index_add(0, idx.reshape(-1), (q[e][:, None, None, None] * wt).reshape(-1))
        parts.append(e)
    S = torch.fft.rfftn(Q.reshape(*grid))
    ks = [torch.fft.fftfreq(g, 1 / g, dtype=torch.float64, device=dev) for g in grid[:2]]
    ks.append(torch.arange(grid[2] // 2 + 1, dtype=torch.float64, device=dev))
    k3 = torch.meshgrid(*ks, indexing="ij")
    m = [sum(inv[a, b] * k3[b] for b in range(3)) for a in range(3)]
    m2 = m[0] ** 2 + m[1] ** 2 + m[2] ** 2
    m2[0, 0, 0] = 1.0
    mod = [_moduli(g, order).to(dev) for g in grid]
    V = ax * by * cz
    bc = (mod[0][:, None, None] * mod[1][None, :, None] * mod[2][None, None, :grid[2] // 2 + 1]
          * F_COUL / (math.pi * V) * torch.exp(-math.pi ** 2 * m2 / beta ** 2) / m2)
    bc[0, 0, 0] = 0.0
    phi = torch.fft.irfftn(S * bc, s=tuple(grid), norm="forward").reshape(-1)
    weight = torch.full((grid[2] // 2 + 1,), 2.0, dtype=torch.float64, device=dev)
    weight[0] = weight[-1] = 1.0
    em = 0.5 * weight * bc * (S.real ** 2 + S.imag ** 2)
    f = -2 * (1 / m2 + math.pi ** 2 / beta ** 2)
    vir = torch.stack([torch.stack([(em * ((a == b) + f * m[a] * m[b])).sum() for b in range(3)]) for a in range(3)])
    forces, pot = [], []
    for e in parts:
        idx = ((at[0][e][:, :, None, None] * grid[1] + at[1][e][:, None, :, None]) * grid[2]
               + at[2][e][:, None, None, :])
        ph = phi[idx]
        W = [w[a][e] for a in range(3)]
        D = [dw[a][e] for a in range(3)]
        g = torch.stack([torch.einsum("nabc,na,nb,nc->n", ph, *[D[b] if b == a else W[b] for b in range(3)]) * grid[a]
                         for a in range(3)], 1)
        forces.append(-q[e][:, None] * (g @ inv.T))
        pot.append(torch.einsum("nabc,na,nb,nc->n", ph, *W))
    return em.sum(), torch.cat(forces), vir, torch.cat(pot)


class _Exact:
    """A system's sums in f64."""

    def __init__(self, s, cell):
        self.p = s
        self.cell = list(np.asarray(cell, dtype=np.float64)) + [0.0] * (6 - len(cell))
        self.q = torch.as_tensor(s["charges"], dtype=torch.float64, device=DEV)
        self.t = torch.as_tensor(s["types"], dtype=torch.int64, device=DEV)
        self.sigma, self.epsilon = (torch.as_tensor(s[k], dtype=torch.float64, device=DEV) for k in ("sigma", "epsilon"))
        self.ex = torch.as_tensor(s["excluded_pairs"], dtype=torch.int64, device=DEV).reshape(-1, 2)
        n = len(self.q)
        lo, hi = self.ex.min(1).values, self.ex.max(1).values
        self.skip = (lo * n + hi).sort().values

    def pairs(self, x, reach):
        """Batches (i, j) of the pairs within the reach, none of them excluded."""
        n = len(self.q)
        for i, j in _pairs(x, self.cell, reach):
            if len(self.skip):
                key = torch.minimum(i, j) * n + torch.maximum(i, j)
                at = torch.searchsorted(self.skip, key).clamp_max(len(self.skip) - 1)
                keep = self.skip[at] != key
                i, j = i[keep], j[keep]
            yield i, j

    def excluded(self, x, q):
        d = _image(x[self.ex[:, 0]] - x[self.ex[:, 1]], self.cell)
        r2 = (d * d).sum(-1)
        r, b = r2.sqrt(), self.p["beta"]
        qq = F_COUL * q[self.ex[:, 0]] * q[self.ex[:, 1]]
        fs = qq * (2 * b / math.sqrt(math.pi) * torch.exp(-(b * r) ** 2) / r2 - torch.erf(b * r) / (r * r2))
        return -(qq * torch.erf(b * r) / r), fs[:, None] * d, d

    def evaluate(self, x, pairs=None):
        """(forces, energies and virials) at x; `pairs`: batches that hold every pair within the cutoff."""
        out = {k: torch.zeros((), dtype=torch.float64, device=DEV) for k in TERMS}
        W = torch.zeros(3, 3, dtype=torch.float64, device=DEV)
        F = torch.zeros_like(x)
        for i, j in (self.pairs(x, self.p["cutoff"]) if pairs is None else pairs):
            for s in range(0, len(i), 20_000_000):
                a, b = i[s:s + 20_000_000], j[s:s + 20_000_000]
                d = _image(x[a] - x[b], self.cell)
                tt = self.t[a], self.t[b]
                fs, lj, co = _pair_terms(d, self.q[a] * self.q[b], self.sigma[tt], self.epsilon[tt], self.p)
                f = fs[:, None] * d
                F.index_add_(0, a, f)
                F.index_add_(0, b, -f)
                out["lj"] += lj.sum()
                out["coulomb"] += co.sum()
                W += d.T @ f
        W_rec = torch.zeros_like(W)
        if self.p["pme"]:
            e, f, d = self.excluded(x, self.q)
            F.index_add_(0, self.ex[:, 0], f)
            F.index_add_(0, self.ex[:, 1], -f)
            out["excluded"] = e.sum()
            W += d.T @ f
            out["reciprocal"], f, W_rec, _ = _reciprocal(x, self.q, self.cell, self.p["grid"], self.p["order"],
                                                         self.p["beta"])
            F += f
        return F, {**out, "virial_pair": W, "virial_reciprocal": W_rec}

    def md(self, x, v, steps, dt, verlet):
        """Leap-frog (or velocity Verlet) with every water rigid."""
        m = torch.as_tensor(self.p["masses"], dtype=torch.float64, device=DEV)[:, None]
        near, at = None, None
        skin = 0.15

        def force(x):
            nonlocal near, at
            if near is None or 2.0 * (x - at).norm(dim=-1).max() > skin:
                near, at = list(self.pairs(x, self.p["cutoff"] + skin)), x.clone()
            return self.evaluate(x, near)[0]

        if verlet:
            v = v - 0.5 * dt * force(x) / m
        for _ in range(steps):
            v = v + dt * force(x) / m
            new = x + dt * v
            if self.p["waters"] is not None:
                new = _shake(x.reshape(-1, 3, 3), new.reshape(-1, 3, 3)).reshape(-1, 3)
                v = (new - x) / dt
            x = new
        if verlet:
            v = v + 0.5 * dt * force(x) / m
        return x, v


def _shake(old, new):
    """new with the waters' three distances restored by forces along the old ones (Newton's iteration)."""
    inv = torch.tensor([1 / M_O, 1 / M_H, 1 / M_H], dtype=torch.float64, device=old.device)
    ends = ((0, 1, ROH), (0, 2, ROH), (1, 2, RHH))
    dirs = torch.stack([old[:, a] - old[:, b] for a, b, _ in ends], 1)
    move = torch.zeros(3, 3, dtype=torch.float64, device=old.device)  # atom a's share of constraint k
    for k, (a, b, _) in enumerate(ends):
        move[a, k], move[b, k] = inv[a], -inv[b]
    want = torch.tensor([r * r for _, _, r in ends], dtype=torch.float64, device=old.device)
    for _ in range(8):
        d = torch.stack([new[:, a] - new[:, b] for a, b, _ in ends], 1)
        off = want - (d * d).sum(-1)
        rel = torch.stack([move[a] - move[b] for a, b, _ in ends], 0)  # d(d_c)/d(lambda_k) / dirs_k
        jac = 2 * torch.einsum("nca,nka,ck->nck", d, dirs, rel)
        lam = torch.linalg.solve(jac, off)
        new = new + torch.einsum("ak,nk,nkc->nac", move, lam, dirs)
    return new


def _exact_frames(case, seed):
    s, X, sig, eps, q = _frames_system(case, seed)
    target = _targets(X, seed) if case["kind"] == "gradient" else None
    ex = _Exact(s, s["box"])
    theta = [torch.tensor(a, dtype=torch.float64, device=DEV, requires_grad=True) for a in (sig, eps, q)]
    sums = [torch.zeros_like(t) for t in theta]
    forces, energies, loss = [], [], 0.0
    b = s["beta"]
    for k in range(len(X)):
        x = X[k]
        sg, ep, qt = theta
        i, j = (torch.cat(c) for c in zip(*ex.pairs(x, s["cutoff"])))
        ti, tj = ex.t[i], ex.t[j]
        # sqrt is not differentiable at an epsilon of 0; such a type has no LJ term
        live = (ep.detach()[ti] > 0) & (ep.detach()[tj] > 0)
        eij = torch.zeros(len(i), dtype=torch.float64, device=DEV)
        eij = eij.masked_scatter(live, torch.sqrt(ep[ti[live]] * ep[tj[live]]))
        d = _image(x[i] - x[j], ex.cell)
        fs, lj, co = _pair_terms(d, qt[i] * qt[j], 0.5 * (sg[ti] + sg[tj]), eij, s)
        e_ex, f_ex, _ = ex.excluded(x, qt)
        e_rec, f_rec, _, _ = _reciprocal(x, qt, ex.cell, s["grid"], s["order"], b)
        f = fs[:, None] * d
        F = (torch.zeros_like(x).index_add(0, i, f).index_add(0, j, -f)
             .index_add(0, ex.ex[:, 0], f_ex).index_add(0, ex.ex[:, 1], -f_ex) + f_rec)
        V = float(np.prod(s["box"]))
        e = (lj.sum() + co.sum() + e_ex.sum() + e_rec - F_COUL * b / math.sqrt(math.pi) * (qt * qt).sum()
             - F_COUL * math.pi * qt.sum() ** 2 / (2 * V * b * b))
        what = ((F - target[k]) ** 2).sum() / len(X) if target is not None else e
        for total, g in zip(sums, torch.autograd.grad(what, theta)):
            total += g
        forces.append(F.detach())
        energies.append(e.detach())
        loss = loss + what.detach()
    if target is not None:
        return torch.stack(forces), loss, tuple(sums)
    return torch.stack(energies), (*sums, -torch.stack(forces))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("forces", "evaluate"):
        s, x, cell = _system(case, seed)
        if kind == "forces":
            return _Exact(s, cell).evaluate(_moved(x, 0.003, seed))[0]
        forces, out = _Exact(s, cell).evaluate(x)
        return forces, out
    if kind == "md":
        s, x, cell = _system(case, seed)
        v = _start_velocities(case, x, seed)
        if len(x) * case["steps"] > 25_000_000:
            return None
        return _Exact(s, cell).md(x, v, case["steps"], 0.002, case.get("verlet", False))
    if kind in ("gradient", "energies"):
        if _atoms(case) * case["frames"] > 2_000_000:
            return None
        return _exact_frames(case, seed)
    forces, terms = [], []
    for s in _solvated(case, seed):
        ex = _Exact(s, s["box"])
        F, e = ex.evaluate(torch.as_tensor(s["positions"], device=DEV))
        self_e = -F_COUL * s["beta"] / math.sqrt(math.pi) * (ex.q * ex.q).sum()
        e["potential"] = sum(e[k] for k in TERMS) + self_e
        for k in ("virial_pair", "virial_reciprocal"):
            e[k] = torch.stack([e[k][a, b] for a, b in ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))])
        forces.append(F)
        terms.append(e)
    return torch.cat(forces), {k: torch.stack([t[k] for t in terms]) for k in terms[0]}
