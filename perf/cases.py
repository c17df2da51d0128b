"""The work a program has this framework do, as cases to be timed and checked.

A case is one call pattern on one synthetic system: flexible three-site waters
around a chain that carries every bonded term (the framework's own workloads
are the same kind of system).  Kinds:

  eval      energies and forces of consecutive frames that lie on the device
            (mdf_set_positions_device, mdf_compute_async, mdf_forces_device)
  forces    the same without energies: the inner loop of somebody's integrator
  host      mdf_set_positions + mdf_compute, one frame at a time, host arrays
  pipeline  mdf_submit / mdf_collect: frames from and to pinned host memory
  rebuild   a new pair list for every frame, then its energies and forces
  backward  gradients with respect to charges and LJ coefficients (mdf_backward)
  train     the same through the autograd function: forward, loss, backward
  batch     many small systems per call (mdf_batch_submit / mdf_batch_collect)
  md        velocity-Verlet dynamics of water, lists rebuilt every ten steps

What the mixed-precision path computes are single-precision numbers (2.5e-7
rms against FP64 at 100k atoms) that the C ABI hands over in doubles; a program
that chose that path keeps them in float32, and so do these cases.  The FP64
path's results stay float64.
"""
import math

import numpy as np
import torch

from md_b200 import abi, autograd, engine, synth, topology

KC = 18.2206899283247 ** 2      # Coulomb constant in the framework's charge unit
TOL = 1e-5                      # Ewald tolerance of the direct sum
WATER_SPACING = 3.105           # A between water oxygens (0.1 atoms per cubic A)
ACCEL = 418.4                   # (kcal/mol/A)/amu in A/ps^2
DT = 0.0005                     # ps per dynamics step


def _case(name, kind, edge, precision="mixed", **over):
    lx, ly, lz = (edge,) * 3 if isinstance(edge, float) else edge
    c = {"name": name, "kind": kind, "lx": lx, "ly": ly, "lz": lz, "precision": precision, "residues": 120,
         "cutoff": 10.0, "switched": True, "frames": 2, "layout": 0, "schedule": 0, "systems": 1, "steps": 0}
    c.update(over)
    return c


def listed():
    return [
        # a small molecule in water, stepped by an outside integrator: latency
        _case("forces_2k_mixed", "forces", 30.0, residues=8, frames=4),
        # a peptide in an oblong box, checked in double precision from host arrays
        _case("host_8k_fp64", "host", (41.0, 36.0, 52.0), "fp64", residues=28),
        # a small protein, frames streamed through pinned host memory
        _case("pipeline_28k_mixed", "pipeline", 66.0, frames=4),
        # the 100 A box the headline figure is quoted on, on the device
        _case("eval_100k_mixed", "eval", 100.0),
        # the same in FP64, with the launch shape the tuner takes there
        _case("eval_100k_fp64", "eval", 100.0, "fp64", layout=1, schedule=1),
        # frames too far apart to share a list (trajectory analysis, Monte Carlo moves)
        _case("rebuild_100k_mixed", "rebuild", 100.0),
        # one parameter-fitting step through torch
        _case("train_28k_mixed", "train", 66.0, frames=1),
        # gradients alone, in double precision
        _case("backward_28k_fp64", "backward", 66.0, "fp64", frames=1),
        # uneven small systems evaluated together (conformer scoring)
        _case("batch_128_mixed", "batch", 32.0, residues=20, cutoff=9.0, systems=128),
        # everyday dynamics of a small box (waters alone: the chain is not relaxed, which a time step of 0.5 fs needs)
        _case("md_28k_mixed", "md", 66.0, residues=0, frames=1, steps=20),
        # a million-atom box: single evaluations ...
        _case("eval_960k_mixed", "eval", 215.0, residues=0),
        # ... and dynamics
        _case("md_960k_mixed", "md", 215.0, residues=0, frames=1, steps=50, schedule=1),
    ]


def draw(rng):
    kind = rng.choice(["eval", "eval", "forces", "host", "pipeline", "rebuild", "backward", "train", "batch", "md"])
    precision = "fp64" if rng.random() < 0.35 else "mixed"
    atoms = math.exp(rng.uniform(math.log(2000.0), math.log(300000.0 if kind in ("eval", "forces", "md") else 120000.0)))
    cutoff = rng.choice([9.0, 10.0])
    if kind == "batch":
        return {"kind": kind, "lx": 32.0, "ly": 32.0, "lz": 32.0, "precision": precision,
                "residues": rng.randrange(8, 25), "cutoff": 9.0, "switched": rng.random() < 0.85, "frames": 2,
                "layout": 0, "schedule": 0, "systems": rng.randrange(8, 129), "steps": 0}
    edge = (atoms / 0.1) ** (1.0 / 3.0)
    aspect = [math.exp(rng.uniform(-0.25, 0.25)) for _ in range(2)]
    size = [max(25.0, round(edge * a, 2)) for a in (aspect[0], aspect[1], 1.0 / (aspect[0] * aspect[1]))]
    half = precision == "fp64" and kind in ("eval", "forces", "host", "md") and rng.random() < 0.5
    return {"kind": kind, "lx": size[0], "ly": size[1], "lz": size[2], "precision": precision,
            "residues": 0 if kind == "md" else min(120, rng.randrange(0, max(2, int(atoms * 0.004)))), "cutoff": cutoff,
            "switched": kind == "md" or rng.random() < 0.85, "frames": 1 if kind in ("backward", "train", "md") else 2,
            "layout": int(half), "schedule": rng.choice([0, 1]), "systems": 1,
            "steps": 20 if kind == "md" else 0}


# ------------------------------------------------------------------ systems
_SYSTEMS = {}
_STREAM = []


def _stream():
    """The program's one stream."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0]


def _system(lx, ly, lz, residues):
    """(topology, box, masses, oxygen positions' first index, coordinates) of a chain of `residues` residues in water.
    The topology is a property of the system, not of a frame: made once."""
    key = (lx, ly, lz, residues)
    if key in _SYSTEMS:
        return _SYSTEMS[key]
    chain = synth.make_system("chain", (lx, ly, lz), 0, residues, 7000 + residues, min_contact=2.0)
    flat = topology.flatten(chain, abi.MDF_SEM_PHYSICAL, engine.cmap_coefficients)
    box = np.array([lx, ly, lz])
    nc = chain.natoms
    n = np.maximum(1, np.round(box / WATER_SPACING).astype(int))
    o = (np.stack(np.meshgrid(*[np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3) + 0.5) * (box / n)
    o += np.random.default_rng(17).uniform(-0.15, 0.15, o.shape)
    if nc:
        dev = torch.device("cuda")
        c, b, w = (torch.tensor(v, device=dev) for v in (chain.coords, box, o))
        far = [((lambda d: d - b * torch.round(d / b))(w[k:k + 4096, None] - c[None]).square().sum(-1).amin(1) > 3.2 ** 2)
               for k in range(0, len(o), 4096)]
        o = o[torch.cat(far).cpu().numpy()]
    nw = len(o)
    first = nc + 3 * np.arange(nw, dtype=np.int32)
    to, th = flat.ntypes - 2, flat.ntypes - 1
    q = synth.charge_to_internal(np.array([-0.834, 0.417]) * synth.SQRT_KC)

    def more(a, b, dtype=np.float64):
        return np.ascontiguousarray(np.concatenate([np.asarray(a).reshape(-1), np.asarray(b).reshape(-1)]).astype(dtype))

    pair = lambda a, b: np.stack([first + a, first + b], 1)                                # noqa: E731
    excl = np.stack([pair(0, 1), pair(0, 2), pair(1, 2)], 1)
    d = dict(flat.__dict__)
    d.pop("_struct")
    d.update(
        charge=more(flat.charge, np.tile([q[0], q[1], q[1]], nw)),
        type=more(flat.type, np.tile([to, th, th], nw), np.int32),
        bond_atoms=more(flat.bond_atoms, np.stack([pair(0, 1), pair(0, 2)], 1), np.int32),
        bond_k=more(flat.bond_k, np.full(2 * nw, synth.WATER_K_BOND)),
        bond_r0=more(flat.bond_r0, np.full(2 * nw, synth.WATER_R_OH)),
        angle_atoms=more(flat.angle_atoms, np.stack([first + 1, first, first + 2], 1), np.int32),
        angle_k=more(flat.angle_k, np.full(nw, synth.WATER_K_ANGLE)),
        angle_theta0=more(flat.angle_theta0, np.full(nw, synth.WATER_THETA)),
        excl_pairs=more(flat.excl_pairs, excl, np.int32))
    mass = more(chain.mass, np.tile([15.999, 1.008, 1.008], nw))
    _SYSTEMS[key] = (topology.FlatTopology(**d), box, mass, chain.coords, o)
    return _SYSTEMS[key]


def _frames(case, seed, frames, size=None):
    """`frames` consecutive snapshots [N, 3]: molecules whole, waters tilted and stretched as at room temperature."""
    flat, box, _, chain, o = _system(*(size or (case["lx"], case["ly"], case["lz"])), case["residues"])
    rng = np.random.default_rng(seed)
    th = synth.WATER_THETA
    legs = np.array([[1.0, 0.0, 0.0], [math.cos(th), math.sin(th), 0.0]])
    v = legs + rng.normal(0.0, 0.15, (len(o), 2, 3))
    v *= synth.WATER_R_OH * (1.0 + rng.normal(0.0, 0.015, (len(o), 2, 1))) / np.linalg.norm(v, axis=2, keepdims=True)
    po = o + rng.normal(0.0, 0.08, o.shape)
    water = np.concatenate([po[:, None], po[:, None] + v], 1).reshape(-1, 3)
    x = np.concatenate([chain + rng.normal(0.0, 0.02, chain.shape), water])
    out = [x]
    for _ in range(frames - 1):
        x = x + rng.normal(0.0, 0.015, x.shape)
        out.append(x)
    return flat, box, out


def _grid(box):
    return tuple(synth.smooth_grid_size(v, 1.0) for v in box)


def _prec(case):
    return abi.MDF_PREC_FP64 if case["precision"] == "fp64" else abi.MDF_PREC_MIXED


def _sizes(case):
    """Boxes of a batch's distinct molecules: eight uneven systems, each in systems / 8 copies."""
    edges = [25.0, 27.5, 29.0, 31.0, 33.0, 35.5, 38.0, 40.0]
    return [(edges[k % 8],) * 3 for k in range(case["systems"])]


def prepare(case, seed):
    kind, dt = case["kind"], torch.float64 if case["precision"] == "fp64" else torch.float32
    common = dict(precision=_prec(case), cutoff=case["cutoff"], skin=2.0,
                  switch_radius=case["cutoff"] - 1.0 if case["switched"] else 0.0, ewald_tol=TOL,
                  pair_layout=case["layout"], pair_schedule=case["schedule"])
    if kind == "batch":
        made = [_frames(case, 1000 * seed + k, case["frames"], s) for k, s in enumerate(_sizes(case))]
        b = engine.Batch([m[0] for m in made], [m[1] for m in made], [_grid(m[1]) for m in made], **common)
        xs = [torch.from_numpy(np.concatenate([m[2][f] for m in made])).pin_memory() for f in range(case["frames"])]
        fs = [torch.empty_like(x).pin_memory() for x in xs]
        b.set_positions(xs[0].numpy())
        b.build_pairlists()
        return {"kind": kind, "batch": b, "x": xs, "f": fs, "dt": dt}
    flat, box, frames = _frames(case, seed, case["frames"])
    if kind == "md":     # lists that prune themselves on the device, as long runs use them
        common.update(prune_every=-1, prune_margin=0.2)
    eng = engine.Engine(flat, box, grid=_grid(box), **common)
    s = {"kind": kind, "eng": eng, "dt": dt, "steps": case["steps"], "x": frames}
    eng.set_positions(frames[0])
    eng.build_pairlist()
    if kind in ("eval", "forces", "rebuild"):
        eng.set_stream(_stream().cuda_stream)
        s["x"] = [torch.tensor(x, device="cuda") for x in frames]
        s["f"] = torch.empty((flat.natoms, 3), dtype=torch.float64, device="cuda")
    elif kind == "pipeline":
        s["x"] = [torch.from_numpy(x).pin_memory() for x in frames]
        s["f"] = [torch.empty_like(x).pin_memory() for x in s["x"]]
    elif kind == "backward":
        s["gF"], s["gE"] = _force_gradient(flat.natoms, seed), 1e-3
    elif kind == "train":
        s["target"] = torch.from_numpy(_target_forces(flat.natoms, seed))
        s["theta"] = [torch.from_numpy(a.copy()).requires_grad_(True) for a in (flat.charge, flat.lj_a, flat.lj_b)]
    elif kind == "md":
        eng.md_init(_system(case["lx"], case["ly"], case["lz"], case["residues"])[2], velocities=_velocities(case, seed))
    return s


def _force_gradient(n, seed):
    return np.random.default_rng(seed + 5).normal(0.0, 1.0 / n, (n, 3))


def _target_forces(n, seed):
    return np.random.default_rng(seed + 6).normal(0.0, 20.0, (n, 3))


def _velocities(case, seed):
    mass = _system(case["lx"], case["ly"], case["lz"], case["residues"])[2]
    v = np.random.default_rng(seed + 7).normal(0.0, 1.0, (len(mass), 3))
    return v * np.sqrt(0.0019872041 * 300.0 * ACCEL / mass)[:, None]


def _terms(e):
    return np.array([e[k] for k in abi.E_NAMES] + [e["total"]])


def run(s):
    kind, dt = s["kind"], s["dt"]
    if kind == "batch":
        b, out = s["batch"], []
        for x, f in zip(s["x"], s["f"]):
            b.submit(x.data_ptr(), f.data_ptr())
        for f in s["f"]:
            e = b.collect()
            out.append({"f": f.to(dt), "e": torch.from_numpy(np.stack([_terms(v) for v in e])).to(dt)})
        return out
    eng, out = s["eng"], []
    if kind in ("eval", "forces", "rebuild"):
        with torch.cuda.stream(_stream()):
            for x in s["x"]:
                eng.set_positions_device(x.data_ptr())
                if kind == "rebuild":
                    eng.build_pairlist()
                eng.compute_async(energy=kind != "forces")
                eng.forces_device(s["f"].data_ptr())
                o = {"f": s["f"].to(dt, copy=True)}
                if kind != "forces":
                    o["e"] = torch.from_numpy(_terms(eng.fetch(forces=False)[0])).to(dt)
                out.append(o)
    elif kind == "host":
        for x in s["x"]:
            eng.set_positions(x)
            e, f = eng.compute()
            out.append({"f": torch.from_numpy(f).to(dt), "e": torch.from_numpy(_terms(e)).to(dt)})
    elif kind == "pipeline":
        n = len(s["x"])
        for k in range(n + 1):
            if k < n:
                eng.submit(s["x"][k].data_ptr(), s["f"][k].data_ptr())
            if k:
                e = eng.collect()
                out.append({"f": s["f"][k - 1].to(dt), "e": torch.from_numpy(_terms(e)).to(dt)})
    elif kind == "backward":
        out = [torch.from_numpy(g).to(dt) for g in eng.backward(s["gF"], s["gE"])]
    elif kind == "train":
        for t in s["theta"]:
            t.grad = None
        f, e = autograd.MDForces.apply(*s["theta"], eng)
        loss = (f - s["target"]).square().sum() / f.shape[0] + 1e-3 * e
        loss.backward()
        out = [t.grad.to(dt) for t in s["theta"]] + [f.detach().to(dt), loss.detach().to(dt)]
    elif kind == "md":
        _, samples = eng.md_run(s["steps"], DT, chunk=10, rebuild_every=10)
        x, v = eng.md_state()
        out = [torch.from_numpy(x).to(dt), torch.from_numpy(v).to(dt), torch.from_numpy(samples[:, 1:].copy()).to(dt)]
    return out


def work(case):
    """Pairs inside the cutoff (60 operations each), spread and gather of 64 mesh points per atom, the mesh's two
    transforms; positions and charges in, forces out, once."""
    total = {"bytes": 0.0, "flops": 0.0}
    times = {"backward": 2.0, "train": 3.0}.get(case["kind"], float(max(case["frames"], case["steps"])))
    for size in _sizes(case) if case["kind"] == "batch" else [(case["lx"], case["ly"], case["lz"])]:
        n = 0.1 * size[0] * size[1] * size[2]
        mesh = float(np.prod(_grid(size)))
        pairs = 0.5 * n * 0.1 * 4.0 / 3.0 * math.pi * case["cutoff"] ** 3
        total["flops"] += times * (60.0 * pairs + 64.0 * 12.0 * n + 5.0 * mesh * math.log2(mesh))
        total["bytes"] += times * n * (24 + 8 + 4 + 24 + (48 if case["kind"] == "md" else 0))
    return total


# ------------------------------------------------------- the same in 64 bits
def _pairs(x, box, rc, excluded):
    """Pairs i < j within rc (minimum image) that are not excluded, in pieces: atoms sorted along x, windows of columns."""
    n = len(x)
    w = x - box * torch.floor(x / box)
    w, order = w[w[:, 0].argsort()], w[:, 0].argsort()
    three, origin = torch.cat([w[:, 0] - box[0], w[:, 0], w[:, 0] + box[0]]), torch.arange(3 * n, device=x.device) % n
    got_i, got_j, size, step = [], [], 0, 1024
    for k in range(0, n, step):
        a = w[k:k + step]
        lo = int(torch.searchsorted(three, a[0, 0] - rc))
        hi = min(int(torch.searchsorted(three, a[-1, 0] + rc)), lo + n)
        at = origin[lo:hi]
        r2 = torch.zeros((len(a), len(at)), dtype=torch.float64, device=x.device)
        for d in range(3):
            t = a[:, d, None] - w[at, d][None]
            r2 += (t - box[d] * torch.round(t / box[d])) ** 2
        i, j = torch.nonzero(r2 <= rc * rc, as_tuple=True)
        i, j = order[k + i], order[at[j]]
        keep = i < j
        i, j = i[keep], j[keep]
        if len(excluded):
            key = i * n + j
            at = torch.searchsorted(excluded, key).clamp(max=len(excluded) - 1)
            keep = excluded[at] != key
            i, j = i[keep], j[keep]
        got_i.append(i)
        got_j.append(j)
        size += len(i)
        if size > 6_000_000 or k + step >= n:
            yield torch.cat(got_i), torch.cat(got_j)
            got_i, got_j, size = [], [], 0


class _Exact:
    """Energies of the PHYSICAL semantics in FP64 torch; forces and gradients by automatic differentiation."""

    def __init__(self, flat, box, case):
        dev = torch.device("cuda")
        t = lambda a: torch.as_tensor(np.asarray(a), device=dev)                             # noqa: E731
        idx = lambda a, k: t(a).long().reshape(-1, k)                                        # noqa: E731
        self.flat, self.n, self.t = flat, flat.natoms, t
        self.box, self.rc, self.switched = t(box), case["cutoff"], case["switched"]
        self.alpha = math.sqrt(-math.log(2 * TOL)) / self.rc
        self.type, self.nb = t(flat.type).long(), t(flat.nb_index).long().reshape(flat.ntypes, -1) - 1
        self.bonds = [(idx(flat.bond_atoms, 2), t(flat.bond_k), t(flat.bond_r0)), (idx(flat.ub_atoms, 2), t(flat.ub_k), t(flat.ub_r0))]
        self.angles = (idx(flat.angle_atoms, 3), t(flat.angle_k), t(flat.angle_theta0))
        self.dih = (idx(flat.dihedral_atoms, 4), t(flat.dihedral_k), t(flat.dihedral_n), t(flat.dihedral_phase))
        self.imp = (idx(flat.improper_atoms, 4), t(flat.improper_k), t(flat.improper_phase))
        self.cmap = (idx(flat.cmap_atoms, 5), t(flat.cmap_set).long())
        self.table = t(flat.cmap_coeff).reshape(flat.cmap_nsets, flat.cmap_res, flat.cmap_res, 4, 4)
        self.excl, self.p14 = idx(flat.excl_pairs, 2), idx(flat.pairs14, 2)
        self.scee, self.scnb, self.a14, self.b14 = t(flat.scee14), t(flat.scnb14), t(flat.lj14_a), t(flat.lj14_b)
        lo, hi = self.excl.min(1).values, self.excl.max(1).values
        self.excl_key = torch.sort(lo * self.n + hi).values
        # reciprocal space: influence function of smooth PME, order 4
        K = _grid(box)
        self.K = K
        L = [float(v) for v in box]
        self.V = L[0] * L[1] * L[2]
        m = [np.fft.fftfreq(K[d], 1.0 / K[d]) / L[d] for d in range(2)] + [np.arange(K[2] // 2 + 1) / L[2]]
        m2 = t(m[0])[:, None, None] ** 2 + t(m[1])[None, :, None] ** 2 + t(m[2])[None, None] ** 2
        m2[0, 0, 0] = 1.0
        c = KC / (math.pi * self.V) * torch.exp(-(math.pi / self.alpha) ** 2 * m2) / m2
        for d in range(3):
            a = 2 * np.pi * np.arange(K[d]) / K[d]
            b = np.abs((1 + 4 * np.exp(1j * a) + np.exp(2j * a)) / 6) ** 2       # |sum_k M4(k+1) e^{2 pi i m k/K}|^2, never 0
            b = t(1.0 / b)[: c.shape[d]]
            c = c * b.reshape([-1 if e == d else 1 for e in range(3)])
        c[0, 0, 0] = 0.0
        wgt = torch.full((K[2] // 2 + 1,), 2.0, dtype=torch.float64, device=dev)
        wgt[0] = 1.0
        if K[2] % 2 == 0:
            wgt[-1] = 1.0
        self.infl = c * wgt

    def _mic(self, d):
        return d - self.box * torch.round(d / self.box)

    def pair_terms(self, q, A, B, x, i, j):
        r2 = self._mic(x[i] - x[j]).square().sum(-1)
        r = r2.sqrt()
        k = self.nb[self.type[i], self.type[j]]
        a, b = (torch.where(k >= 0, v[k.clamp(min=0)], 0.0) for v in (A, B))
        i6 = 1.0 / (r2 * r2 * r2)
        u = (a * i6 - b) * i6
        if self.switched:
            s = ((r - (self.rc - 1.0)) / 1.0).clamp(0.0, 1.0)
            u = u * (1 + s ** 3 * (-10 + s * (15 - 6 * s)))
        else:       # force-shifted
            c6 = self.rc ** -6
            u = u - (a * c6 - b) * c6 + (r - self.rc) * (12 * a * c6 - 6 * b) * c6 / self.rc
        return u.sum(), (KC * q[i] * q[j] * torch.special.erfc(self.alpha * r) / r).sum()

    def other_terms(self, q, x):
        e, al = {}, self.alpha
        for name, (at, k, r0) in zip(("bond", "ub"), self.bonds):
            e[name] = (k * ((x[at[:, 0]] - x[at[:, 1]]).norm(dim=-1) - r0) ** 2).sum()
        at, k, t0 = self.angles
        u, v = x[at[:, 0]] - x[at[:, 1]], x[at[:, 2]] - x[at[:, 1]]
        th = torch.atan2(torch.linalg.cross(u, v).norm(dim=-1), (u * v).sum(-1))
        e["angle"] = (k * (th - t0) ** 2).sum()
        at, k, n, ph = self.dih
        e["dihedral"] = (k * (1 + torch.cos(n * self._torsion(x, at) - ph))).sum()
        at, k, ph = self.imp
        w = self._torsion(x, at) - ph
        e["improper"] = (k * (w - 2 * math.pi * torch.round(w / (2 * math.pi)).detach()) ** 2).sum()
        at, which = self.cmap
        res = self.flat.cmap_res
        g = [(self._torsion(x, at[:, k:k + 4]) + math.pi) * (res / (2 * math.pi)) for k in (0, 1)]
        cell = [torch.floor(v.detach()) for v in g]
        co = self.table[which, cell[0].long() % res, cell[1].long() % res]
        pu, pv = (torch.stack([(v - c) ** p for p in range(4)], -1) for v, c in zip(g, cell))
        e["cmap"] = torch.einsum("nij,ni,nj->", co, pu, pv)
        i, j = self.excl[:, 0], self.excl[:, 1]
        r = self._mic(x[i] - x[j]).norm(dim=-1)
        e["ee_excl"] = -(KC * q[i] * q[j] * torch.special.erf(al * r) / r).sum()
        i, j = self.p14[:, 0], self.p14[:, 1]
        r = self._mic(x[i] - x[j]).norm(dim=-1)
        e["ee14"] = (KC * q[i] * q[j] / (self.scee * r)).sum()
        k = self.nb[self.type[i], self.type[j]]
        e["vdw14"] = torch.where(k >= 0, (self.a14[k] / r ** 12 - self.b14[k] / r ** 6) / self.scnb, 0.0).sum()
        e["ee_self"] = -KC * al / math.sqrt(math.pi) * (q * q).sum()
        e["ee_recip"] = self._recip(q, x) - KC * math.pi * q.sum() ** 2 / (2 * self.V * al * al)
        return e

    @staticmethod
    def _torsion(x, at):
        b1, b2, b3 = (x[at[:, k + 1]] - x[at[:, k]] for k in range(3))
        n1, n2 = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
        return torch.atan2((b1 * n2).sum(-1) * b2.norm(dim=-1), (n1 * n2).sum(-1))

    def _recip(self, q, x):
        K = self.t(np.array(self.K, dtype=np.float64))
        u = (x - self.box * torch.floor((x / self.box).detach())) * (K / self.box)
        base = torch.floor(u.detach())
        w, base = u - base, base.long()
        th = torch.stack([(1 - w) ** 3, 3 * w ** 3 - 6 * w ** 2 + 4, -3 * w ** 3 + 3 * w ** 2 + 3 * w + 1, w ** 3], -1) / 6
        off = torch.arange(4, device=x.device) - 1
        at = [(base[:, d, None] + off) % self.K[d] for d in range(3)]
        idx = (at[0][:, :, None, None] * self.K[1] + at[1][:, None, :, None]) * self.K[2] + at[2][:, None, None]
        val = q[:, None, None, None] * th[:, 0, :, None, None] * th[:, 1, None, :, None] * th[:, 2, None, None]
        g = torch.zeros(self.K[0] * self.K[1] * self.K[2], dtype=torch.float64, device=x.device)
        S = torch.fft.rfftn(g.index_add(0, idx.reshape(-1), val.reshape(-1)).reshape(self.K))
        return 0.5 * (self.infl * (S.real ** 2 + S.imag ** 2)).sum()

    def evaluate(self, x, q=None, A=None, B=None):
        """Energy terms [17] and forces [N, 3] at positions x."""
        q, A, B = (self.t(f) if v is None else v for v, f in ((q, self.flat.charge), (A, self.flat.lj_a), (B, self.flat.lj_b)))
        x = torch.as_tensor(x, device=self.box.device).detach().requires_grad_(True)
        e = self.other_terms(q, x)
        f = -torch.autograd.grad(sum(e.values()), x)[0]
        e = {k: float(v.detach()) for k, v in e.items()}
        e["vdw"] = e["ee_direct"] = 0.0
        for i, j in _pairs(x.detach(), self.box, self.rc, self.excl_key):
            u, c = self.pair_terms(q, A, B, x, i, j)
            f = f - torch.autograd.grad(u + c, x)[0]
            e["vdw"] += float(u.detach())
            e["ee_direct"] += float(c.detach())
        e = [e.get(k, 0.0) for k in abi.E_NAMES]
        return np.array(e + [math.fsum(e)]), f.detach()

    def gradients(self, x, v, gE):
        """d/d(q, A, B) of gE E + v . F, F = -dE/dx: the derivative along v of the energy's gradient."""
        th = [self.t(a).clone().requires_grad_(True) for a in (self.flat.charge, self.flat.lj_a, self.flat.lj_b)]
        x, v = (torch.as_tensor(a, device=self.box.device) for a in (x, v))
        total = [torch.zeros_like(t) for t in th]

        def add(energy):
            s = torch.zeros((), dtype=torch.float64, device=x.device, requires_grad=True)
            e = energy(x + s * v)
            along, = torch.autograd.grad(e, s, create_graph=True)
            got = torch.autograd.grad(gE * e - along, th, allow_unused=True)
            for t, g in zip(total, got):
                if g is not None:
                    t += g
        add(lambda y: sum(self.other_terms(th[0], y)[k] for k in ("ee_excl", "ee14", "ee_self", "ee_recip")))
        for i, j in _pairs(x, self.box, self.rc, self.excl_key):
            for a in range(0, len(i), 2_000_000):
                add(lambda y: sum(self.pair_terms(*th, y, i[a:a + 2_000_000], j[a:a + 2_000_000])))
        return total


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        made = [_frames(case, 1000 * seed + k, case["frames"], s) for k, s in enumerate(_sizes(case))]
        sys = {}
        out = []
        for f in range(case["frames"]):
            got = [(sys.get(id(m[0])) or sys.setdefault(id(m[0]), _Exact(m[0], m[1], case))).evaluate(m[2][f]) for m in made]
            out.append({"f": torch.cat([g[1] for g in got]), "e": np.stack([g[0] for g in got])})
        return out
    flat, box, frames = _frames(case, seed, case["frames"])
    E = _Exact(flat, box, case)
    if kind == "md":
        if flat.natoms * case["steps"] > 2_500_000:
            return None
        im = ACCEL / E.t(_system(case["lx"], case["ly"], case["lz"], case["residues"])[2])[:, None]
        x, v = E.t(frames[0]), E.t(_velocities(case, seed))
        _, f = E.evaluate(x)
        samples = []
        for k in range(case["steps"]):
            v = v + 0.5 * DT * im * f
            x = x + DT * v
            e, f = E.evaluate(x)
            v = v + 0.5 * DT * im * f
            if (k + 1) % 10 == 0:
                samples.append([e[-1], float((0.5 / im * v * v).sum())])
        return [x, v, np.array(samples)]
    if kind == "backward":
        return E.gradients(frames[0], _force_gradient(flat.natoms, seed), 1e-3)
    if kind == "train":
        e, f = E.evaluate(frames[0])
        d = f - E.t(_target_forces(flat.natoms, seed))
        return E.gradients(frames[0], 2 * d / len(f), 1e-3) + [f, float(d.square().sum() / len(f) + 1e-3 * e[-1])]
    out = []
    for x in frames:
        e, f = E.evaluate(x)
        out.append({"f": f} if kind == "forces" else {"f": f, "e": e})
    return out
