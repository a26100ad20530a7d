"""Performance cases of the engine's public entry points, for timing it and comparing its outputs.

What a user of the engine runs, over the sizes it is run at:

* ``poses``: energies of explicit trial poses (``Engine.energy_poses``) on a context that the
  program keeps: one fragment's few candidates up to a whole screening batch;
* ``grad``: the differentiable pose energy (``grad.RigidFragment`` / ``grad.pose_energy``), forward
  and backward: poses and site charges alone, or the per-type LJ parameters through the pair
  table too;
* ``chain``: one GCMC chain through the drop-in ``runGCMC`` on page-locked host arrays, with the
  reference's proposals, symmetric ones, force-biased ones, plain cutoff or Ewald electrostatics;
* ``batch``: many replicas in one ``runGCMC_batch`` call: a chemical-potential scan over systems of
  uneven size, force-biased replicas of one system, replicas of a large slab under Ewald.

A pass starts from the prepared state every time: the chains' calls update the caller's arrays in
place, so ``run`` first puts the occupied fragment slots back.
"""
import functools
import math

import numpy as np
import torch

from pygcmc_b200 import poses as PZ
from pygcmc_b200 import system as S
from pygcmc_b200._native import default_options
from pygcmc_b200.engine import Engine
from pygcmc_b200.gpu import runGCMC, runGCMC_batch
from pygcmc_b200.grad import RigidFragment, lj_table, pose_energy

CUTOFF = 12.0
COULOMB = 1388.431112
FLOPS_PER_PAIR = 19  # LJ + Coulomb of one atom-site pair, geometry included
PROTEIN_DENSITY = 6000 / 64.0 ** 3


def listed():
    return [
        # a handful of candidate poses on a small protein: the smallest call, latency alone
        {"name": "poses_few", "kind": "poses", "system": "protein", "atoms": 2000, "poses": 16, "ftype": 1},
        # a screening batch of poses on the ordinary protein
        {"name": "poses_many", "kind": "poses", "system": "protein", "atoms": 6000, "poses": 8192, "ftype": 4},
        # gradients of some tens of waters with respect to position, orientation and charges
        {"name": "grad_few", "kind": "grad", "system": "water", "atoms": 400, "poses": 61, "ftype": 0,
         "table": False},
        # the differentiation workload: 4096 poses, per-type eps and rmin/2 through the pair table too
        {"name": "grad_table", "kind": "grad", "system": "protein", "atoms": 6000, "poses": 4096, "ftype": 0,
         "table": True},
        # a short call on a small system, as a driver that interleaves GCMC with other work makes it
        {"name": "chain_short", "kind": "chain", "system": "protein", "atoms": 2000, "conf_bias": 256, "steps": 24,
         "proposal": 0, "mesh": 0},
        # the protein with eight fragments, reference proposals: the ordinary chain
        {"name": "chain_protein", "kind": "chain", "system": "protein", "atoms": 6000, "conf_bias": 1000,
         "steps": 512, "proposal": 0, "mesh": 0},
        # water box, symmetric proposals: nearly every molecule interacts with every other
        {"name": "chain_water", "kind": "chain", "system": "water", "atoms": 800, "conf_bias": 1000, "steps": 256,
         "proposal": 1, "mesh": 0},
        # a smaller water box under Ewald electrostatics
        {"name": "chain_water_ewald", "kind": "chain", "system": "water", "atoms": 400, "conf_bias": 128,
         "steps": 128, "proposal": 1, "mesh": 64},
        # one force-biased chain of the protein
        {"name": "chain_forcebias", "kind": "chain", "system": "protein", "atoms": 6000, "conf_bias": 1000,
         "steps": 256, "proposal": 2, "mesh": 0},
        # 64 replicas of uneven size, chemical potentials and seeds of their own
        {"name": "batch_scan", "kind": "batch", "system": "protein", "atoms": 0, "unique": 8, "replicas": 64,
         "conf_bias": 1000, "steps": 96, "proposal": 0, "mesh": 0, "tuned": True},
        # 64 force-biased replicas of one protein
        {"name": "batch_forcebias", "kind": "batch", "system": "protein", "atoms": 6000, "unique": 1,
         "replicas": 64, "conf_bias": 1000, "steps": 48, "proposal": 2, "mesh": 0, "tuned": False},
        # the largest: 16 replicas of the 200 000-atom slab, Ewald on a 128 x 128 x 96 mesh, force-biased
        {"name": "batch_slab_ewald", "kind": "batch", "system": "slab", "atoms": 200000, "unique": 1,
         "replicas": 16, "conf_bias": 1000, "steps": 32, "proposal": 2, "mesh": 128, "tuned": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["poses", "grad", "chain", "chain", "batch"])
    water = rng.random() < 0.35
    if kind in ("poses", "grad"):
        c = {"kind": kind, "system": "water" if water else "protein",
             "atoms": rng.randint(150, 500) if water else _log(rng, 1500, 9000),
             "poses": _log(rng, 9, 8192 if kind == "poses" else 4096), "ftype": 0 if water else rng.randint(0, 7)}
        if kind == "grad":
            c["table"] = (not water) and rng.random() < 0.6
        return c
    if kind == "chain":
        proposal = rng.choice([0, 1, 2])
        return {"kind": kind, "system": "water" if water else "protein",
                "atoms": rng.randint(150, 500) if water else _log(rng, 1500, 9000),
                "conf_bias": _log(rng, 40, 1000), "steps": _log(rng, 12, 400), "proposal": proposal,
                "mesh": rng.choice([0, 0, 0, 64])}
    proposal = rng.choice([0, 0, 1, 2])
    unique = rng.choice([1, 2, 5])
    return {"kind": kind, "system": "protein", "atoms": 0 if unique > 1 else _log(rng, 1500, 9000), "unique": unique,
            "replicas": unique * (2 * rng.randint(0, 30 // unique - 1) + 1), "conf_bias": _log(rng, 100, 1000),
            "steps": _log(rng, 12, 96), "proposal": proposal, "mesh": rng.choice([0, 0, 0, 48]),
            "tuned": rng.random() < 0.5}


# ---- systems ----
def _water_edge(n):
    """Box edge of n waters at the density of 800 in 30 A (at least 26 A: over two cutoffs)."""
    return max(26.0, 30.0 * (n / 800.0) ** (1.0 / 3.0))


def _protein(n, seed, steps, conf_bias):
    box = (n / PROTEIN_DENSITY) ** (1.0 / 3.0)
    return S.protein_system(seed=seed, n_atoms=n, box=max(40.0, box), radius=24.0 * (n / 6000.0) ** (1.0 / 3.0),
                            mcsteps=steps, conf_bias=conf_bias)


@functools.lru_cache(maxsize=2)
def _molecules(system, atoms, unique, steps, conf_bias):
    """The systems of a case before anything is drawn for it: molecules, force field, box, schedule."""
    if system == "water":
        return [S.water_box(n_water=atoms, box=_water_edge(atoms), seed=1, mcsteps=steps, conf_bias=conf_bias)]
    if system == "slab":
        return [S.slab_system(seed=1, n_atoms=atoms, mcsteps=steps, conf_bias=conf_bias)]
    if unique == 1:
        return [_protein(atoms, 1, steps, conf_bias)]
    return [_protein(_size_of(u, unique), 1 + u, steps, conf_bias) for u in range(unique)]


def _size_of(u, unique):
    """Fixed atoms of system u of a batch of uneven size: 2000 to 40000, spread over the logarithm."""
    return int(2000 * 20 ** ((u + 0.5) / unique))


def _drawn(base, g):
    """A configuration of its own: every fixed atom displaced a little, every fragment copy shifted
    as a whole, the move schedule in another order."""
    s = base.copy()
    first = int(s.fragmentInfo[0]["startRes"])
    nfix = s.n_fixed_atoms()
    s.atomInfo["position"][:nfix] += g.uniform(-0.05, 0.05, (nfix, 3)).astype(np.float32)
    shift = g.uniform(-0.1, 0.1, (len(s.residueInfo) - first, 3)).astype(np.float32)
    s.residueInfo["position"][first:] += shift
    s.atomInfo["position"][nfix:] += np.repeat(shift, s.residueInfo["atomNum"][first:], axis=0)
    s.moveArray = g.permutation(s.moveArray)
    return s


def _system(case, seed):
    """The system that explicit poses are evaluated in."""
    return _drawn(_molecules(case["system"], case["atoms"], 1, 8, 1000)[0], np.random.default_rng([seed, 3]))


def _systems(case, seed):
    """The replicas of a chain or batch case: `unique` systems, each `replicas / unique` times with a
    chemical-potential shift and a seed of its own."""
    unique, nrep = case.get("unique", 1), case.get("replicas", 1)
    base = _molecules(case["system"], case["atoms"], unique, case["steps"], case["conf_bias"])
    base = [_drawn(b, np.random.default_rng([seed, u])) for u, b in enumerate(base)]
    out = []
    for r in range(nrep):
        s = base[r % unique].copy()
        s.SimInfo[0]["seed"] = (seed * 7 + 131 * r) & 0xFFFFFFFF
        if unique > 1:
            s.fragmentInfo["muex"] += np.float32(-0.5 * (r // unique))
        out.append(s)
    return out


def _options(case):
    o = default_options(proposal=case["proposal"], muex_kcal=1 if case["system"] == "water" else 0)
    if case["mesh"]:
        o.pme, o.pme_alpha = 1, 0.32
        mesh = (128, 128, 96) if case["system"] == "slab" else (case["mesh"],) * 3
        for a in range(3):
            o.pme_grid[a] = mesh[a]
    if case["kind"] == "batch":
        o.grid_bits = 1
        o.branches = min(4, case["replicas"])
        if case["tuned"]:  # the shape that the autotuner settles on for such batches
            o.cells_per_cutoff, o.split_items, o.energy_variant = 1, 512, 1
    return o


def _page_locked(arrays):
    """The arrays one after another in one page-locked buffer: the whole and a view of each."""
    n = sum(len(a) for a in arrays)
    dt = arrays[0].dtype
    buf = torch.empty(max(1, n * dt.itemsize), dtype=torch.uint8, pin_memory=True)
    whole = buf.numpy()[:n * dt.itemsize].view(dt)
    views, at = [], 0
    for a in arrays:
        v = whole[at:at + len(a)]
        v[...] = a
        views.append(v)
        at += len(a)
    return buf, whole, views


# ---- explicit poses ----
def _pose_inputs(case, system, seed):
    """Trial poses as a translate / rotate step makes them: occupied copies of the fragment type,
    each displaced by up to 0.4 A per axis and turned by up to about 20 degrees, its own copy
    skipped.  com [n, 3], quat [n, 4] (float32) and the skipped residues."""
    g = np.random.default_rng([seed, 77])
    f = system.fragmentInfo[case["ftype"]]
    n0, r0 = int(f["totalNum"]), int(f["startRes"])
    slot = g.integers(0, n0, case["poses"])
    com = system.residueInfo["position"][r0 + slot] + g.uniform(-0.4, 0.4, (case["poses"], 3))
    quat = np.concatenate([np.ones((case["poses"], 1)), g.uniform(-0.1, 0.1, (case["poses"], 3))], axis=1)
    quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    # the copy's own orientation: the rotation that takes the template to its sites
    tpl, _, _ = PZ.template(system, case["ftype"])
    ns = len(tpl)
    first = system.residueInfo["atomStart"][r0 + slot]
    sites = system.atomInfo["position"][first[:, None] + np.arange(ns)[None, :]].astype(np.float64)
    sites -= sites.mean(axis=1, keepdims=True)
    own = _orientation(tpl, sites)
    return com.astype(np.float32), _quat_mul(quat, own).astype(np.float32), (r0 + slot).astype(np.int32)


def _orientation(tpl, sites):
    """Unit quaternions of the rotations that fit tpl [ns, 3] to each of sites [n, ns, 3] (the
    largest eigenvector of the 4 x 4 key matrix of the correlation)."""
    C = np.einsum("si,nsj->nij", tpl, sites)
    xx, xy, xz, yx, yy, yz, zx, zy, zz = C.reshape(-1, 9).T
    K = np.stack([xx + yy + zz, yz - zy, zx - xz, xy - yx,
                  yz - zy, xx - yy - zz, xy + yx, zx + xz,
                  zx - xz, xy + yx, yy - xx - zz, yz + zy,
                  xy - yx, zx + xz, yz + zy, zz - xx - yy], -1).reshape(-1, 4, 4)
    return np.linalg.eigh(K)[1][:, :, 3]


def _quat_mul(a, b):
    w1, x1, y1, z1 = a.T
    w2, x2, y2, z2 = b.T
    return np.stack([w1 * w2 - x1 * x2 - y1 * y2 - z1 * z2, w1 * x2 + x1 * w2 + y1 * z2 - z1 * y2,
                     w1 * y2 - x1 * z2 + y1 * w2 + z1 * x2, w1 * z2 + x1 * y2 - y1 * x2 + z1 * w2], -1)


def _lj_types(system):
    lt = system.meta["lj_types"]
    return lt["eps_kcal"].astype(np.float32), lt["rmin_half"].astype(np.float32)


# ---- the five functions ----
def prepare(case, seed):
    if case["kind"] in ("chain", "batch"):
        systems = _systems(case, seed)
        st = {"case": case, "options": _options(case), "keep": []}
        cols = {}
        for name in ("SimInfo", "fragmentInfo", "residueInfo", "atomInfo", "moveArray"):
            buf, whole, cols[name] = _page_locked([getattr(s, name) for s in systems])
            st["keep"].append(buf)
            st[name] = whole
        arrays, undo = [], []
        shared = {}  # inputs that replicas of one system have in common and no call writes
        for r, s in enumerate(systems):
            key = r % case.get("unique", 1)
            if key not in shared:
                grid = s.grid_bits if st["options"].grid_bits else s.grid
                held = [_page_locked([a]) for a in (grid, s.ff)]
                st["keep"] += [h[0] for h in held]
                shared[key] = [h[2][0] for h in held]
            frag, res, atoms = cols["fragmentInfo"][r], cols["residueInfo"][r], cols["atomInfo"][r]
            arrays.append((cols["SimInfo"][r], frag, res, atoms, *shared[key], cols["moveArray"][r]))
            undo.append((frag["totalNum"], s.fragmentInfo["totalNum"].copy()))
            for f in s.fragmentInfo:
                r0, n = int(f["startRes"]), int(f["totalNum"])
                if n:
                    a0 = int(s.residueInfo["atomStart"][r0])
                    a1 = a0 + n * int(f["num_atoms"])
                    undo.append((res[r0:r0 + n], s.residueInfo[r0:r0 + n].copy()))
                    undo.append((atoms[a0:a1], s.atomInfo[a0:a1].copy()))
        st["arrays"], st["undo"] = arrays, undo
        return st
    s = _system(case, seed)
    com, quat, self_res = _pose_inputs(case, s, seed)
    tpl, q, t = PZ.template(s, case["ftype"])
    st = {"case": case, "system": s, "engine": Engine(s, default_options())}
    if case["kind"] == "poses":
        xyz = PZ.rigid_sites(tpl, com, quat).astype(np.float32)
        st.update(xyz=xyz, q=q, types=t, com=com, self_res=self_res)
        return st
    dev = torch.device("cuda")
    st["frag"] = RigidFragment(st["engine"], 0, case["ftype"], dtype=torch.float32)
    leaves = {"com": com, "quat": quat, "charges": q}
    if case["table"]:
        leaves["eps"], leaves["rmin"] = _lj_types(s)
    else:
        st["ff"] = torch.tensor(s.ff, device=dev)
    st["leaves"] = {k: torch.tensor(v, device=dev, requires_grad=True) for k, v in leaves.items()}
    st["self_res"] = torch.tensor(self_res, device=dev)
    st["weight"] = torch.tensor(np.random.default_rng([seed, 5]).normal(size=case["poses"]), device=dev)
    st["ffx"] = int(s.SimInfo[0]["ffXNum"])
    return st


def run(state):
    case = state["case"]
    if case["kind"] == "poses":
        e, groups = state["engine"].energy_poses(state["xyz"], state["q"], state["types"], state["com"],
                                                 self_res=state["self_res"])
        return {"energy": e, "groups": groups}
    if case["kind"] == "grad":
        x, frag = state["leaves"], state["frag"]
        for v in x.values():
            v.grad = None
        ff = lj_table(x["eps"], x["rmin"], state["ffx"]) if case["table"] else state["ff"]
        e = pose_energy(state["engine"], 0, frag.sites(x["com"], x["quat"]), x["charges"], ff, frag.site_type,
                        centres=x["com"], self_res=state["self_res"])
        (e * state["weight"]).sum().backward()
        return {"energy": e, **{"d_" + k: v.grad for k, v in x.items()}}
    for there, kept in state["undo"]:
        there[...] = kept
    if case["kind"] == "chain":
        runGCMC(*state["arrays"][0], options=state["options"])
    else:
        runGCMC_batch(state["arrays"], state["options"])
    return {"count": state["fragmentInfo"]["totalNum"], "centre": state["residueInfo"]["position"],
            "position": state["atomInfo"]["position"], "charge": state["atomInfo"]["charge"],
            "type": state["atomInfo"]["type"]}


def _neighbours(atoms, edge):
    """Atoms within the cutoff of a pose, on average, of `atoms` in a box."""
    return min(atoms, atoms * 4.0 / 3.0 * math.pi * CUTOFF ** 3 / edge ** 3)


def _shape(system, atoms):
    """(atoms, box edge, sites per fragment, copies per fragment type, fragment types)"""
    if system == "water":
        return 3 * atoms, _water_edge(atoms), 3, atoms, 1
    if system == "slab":
        return atoms + 51000, 139.0, 6, 1800, 9
    edge = max(40.0, (atoms / PROTEIN_DENSITY) ** (1.0 / 3.0))
    copies = round(0.25 * edge ** 3 * 0.0006023)
    return atoms + 8 * 7 * copies, edge, 7, copies, 8


def work(case):
    if case["kind"] in ("poses", "grad"):
        atoms, edge, sites, _, _ = _shape(case["system"], case["atoms"])
        n = case["poses"]
        pairs = n * sites * _neighbours(atoms, edge)
        if case["kind"] == "poses":  # sites, centre, skipped residue in; energy and group count out
            return {"bytes": n * (12 * sites + 12 + 4 + 8 + 4) + 20 * atoms, "flops": FLOPS_PER_PAIR * pairs}
        # poses, weight and skipped residue in; energy and gradients out.  The backward's pairs cost about twice
        # the forward's operations
        return {"bytes": n * (28 + 8 + 4 + 8 + 28) + 20 * atoms, "flops": 3 * FLOPS_PER_PAIR * pairs}
    byts = flops = 0.0
    unique = case.get("unique", 1)
    for u in range(unique):
        size = case["atoms"] if unique == 1 else _size_of(u, unique)
        copies_of = case.get("replicas", 1) / unique
        atoms, edge, sites, copies, types = _shape(case["system"], size)
        p = (0.25, 0.25, 0.5) if case["system"] == "water" else (0.3, 0.3, 0.4)
        poses = p[0] * case["conf_bias"] + p[1] + p[2] * 2 * min(case["conf_bias"], copies)
        flops += copies_of * case["steps"] * poses * sites * _neighbours(atoms, edge) * FLOPS_PER_PAIR
        # the state in (atoms, residues, one bit or three floats per cavity voxel), the fragments' part out
        voxels = edge ** 3 / 8 if case["kind"] == "batch" else 12 * edge ** 3
        byts += copies_of * (24 * atoms + voxels + 20 * types * copies * (sites + 1))
        if case["mesh"]:  # a forward and an inverse real transform for each step that moves a charge
            mesh = 128 * 128 * 96 if case["system"] == "slab" else case["mesh"] ** 3
            flops += copies_of * case["steps"] * 0.5 * 5 * mesh * math.log2(mesh)
    return {"bytes": byts, "flops": flops}


def exact(case, seed):
    """Energies and gradients of explicit poses in 64 bits (plain torch).  Which groups count is the
    engine's own 32-bit rule; a chain's outcome is a sequence of decisions and has no such value."""
    if case["kind"] not in ("poses", "grad"):
        return None
    s = _system(case, seed)
    com, quat, self_res = _pose_inputs(case, s, seed)
    tpl, q, t = PZ.template(s, case["ftype"])
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    info = s.SimInfo[0]
    L32 = torch.tensor(np.asarray(info["cryst"], np.float32), device=dev)
    L = L32.double()
    # the groups and atoms that are there: fixed ones and occupied slots
    first = int(s.fragmentInfo[0]["startRes"])
    ids = np.concatenate([np.arange(first)] + [np.arange(int(f["startRes"]), int(f["startRes"]) + int(f["totalNum"]))
                                               for f in s.fragmentInfo])
    res = s.residueInfo[ids]
    atom = np.concatenate([np.arange(r["atomStart"], r["atomStart"] + r["atomNum"]) for r in res])
    group_of = torch.tensor(np.repeat(np.arange(len(res)), res["atomNum"]), device=dev)
    centre = torch.tensor(res["position"].copy(), device=dev)
    A = torch.tensor(s.atomInfo["position"][atom].astype(np.float64), device=dev)
    qa = torch.tensor(s.atomInfo["charge"][atom].astype(np.float64), device=dev)
    ta = torch.tensor(s.atomInfo["type"][atom].astype(np.int64), device=dev)
    ids_t = torch.tensor(ids, device=dev)
    ffx, ffy = int(info["ffXNum"]), int(info["ffYNum"])
    grads = case["kind"] == "grad"

    def leaf(a):
        return torch.tensor(np.asarray(a, np.float64), device=dev, requires_grad=grads)

    c32 = torch.tensor(com, device=dev)
    x = {"com": leaf(com), "quat": leaf(quat), "charges": leaf(q)}
    if grads and case["table"]:
        x["eps"], x["rmin"] = (leaf(v) for v in _lj_types(s))
    if grads:
        w = torch.tensor(np.random.default_rng([seed, 5]).normal(size=case["poses"]), device=dev)
    sites32 = None if grads else torch.tensor(PZ.rigid_sites(tpl, com, quat).astype(np.float32), device=dev).double()
    st = torch.tensor(t.astype(np.int64), device=dev)
    tpl64 = torch.tensor(tpl, device=dev)
    skip = torch.tensor(self_res, device=dev)
    energy, groups = [], []
    step = max(1, int(2.0e7 // max(1, len(tpl) * len(atom))))
    for p0 in range(0, case["poses"], step):
        p = slice(p0, min(case["poses"], p0 + step))
        d = c32[p][:, None, :] - centre[None, :, :]
        k = torch.trunc(d / L32 + torch.copysign(torch.full_like(d, 0.5), d))
        d = (d.double() - k.double() * L).float()
        r = (d[..., 0] * d[..., 0])
        r = (d[..., 1].double() ** 2 + r.double()).float()
        r = (d[..., 2].double() ** 2 + r.double()).float()
        inc = (torch.sqrt(r) <= float(info["cutoff"])) & (ids_t[None, :] != skip[p][:, None])
        groups.append(inc.sum(1).to(torch.int32))
        if grads and case["table"]:
            sig = 2.0 * x["rmin"] / 2.0 ** (1.0 / 6.0) / 10.0
            sigma = (sig[:ffx, None] + sig[None, :]) / 2
            e4 = 4.184 * x["eps"]
            eps = torch.sqrt(e4[:ffx, None] * e4[None, :])
        else:
            table = torch.tensor(s.ff.astype(np.float64), device=dev).reshape(ffx, ffy, 2)
            sigma, eps = table[..., 0], table[..., 1]
        if grads:
            qn = x["quat"][p] / x["quat"][p].norm(dim=-1, keepdim=True)
            qw, qx, qy, qz = qn.unbind(-1)
            R = torch.stack([1 - 2 * (qy * qy + qz * qz), 2 * (qx * qy - qw * qz), 2 * (qx * qz + qw * qy),
                             2 * (qx * qy + qw * qz), 1 - 2 * (qx * qx + qz * qz), 2 * (qy * qz - qw * qx),
                             2 * (qx * qz - qw * qy), 2 * (qy * qz + qw * qx), 1 - 2 * (qx * qx + qy * qy)],
                            -1).reshape(-1, 3, 3)
            X = x["com"][p][:, None, :] + torch.einsum("pij,sj->psi", R, tpl64)
        else:
            X = sites32[p]
        pose, a = torch.nonzero(inc[:, group_of], as_tuple=True)
        D = A[a][:, None, :] - X[pose]
        D = D - L * torch.round(D.detach() / L)
        r2 = (D * D).sum(-1)
        sg, ep = sigma[st][:, ta[a]].T, eps[st][:, ta[a]].T
        s6 = (100.0 * sg * sg / r2) ** 3
        pair = 4.0 * ep * (s6 * s6 - s6) + COULOMB * x["charges"][None, :] * qa[a][:, None] / torch.sqrt(r2)
        e = torch.zeros(p.stop - p.start, dtype=torch.float64, device=dev).index_add(0, pose, pair.sum(1))
        if grads:
            (e * w[p]).sum().backward()
        energy.append(e.detach())
    e = torch.cat(energy)
    if not grads:
        return {"energy": e, "groups": torch.cat(groups)}
    return {"energy": e, **{"d_" + k: v.grad for k, v in x.items()}}
