"""The work this framework is used for, as cases that can be timed and checked.

A case is a dict of plain values; its ``kind`` names the public entry point:

* ``eval``     energies and pose gradients of one batch (``energrad``), Euler or 4x4 poses;
* ``autograd`` energies, then the adjoint to the poses and to the grid values (``docking_energy``);
* ``minimise`` a batch of ligands through the fused ADAM minimiser (``minimise`` / ``MinimisePlan``);
* ``schema``   the quaternion / adabelief protocol of the reference (``minimise_schema``);
* ``rescore``  explicit all-pairs energies and gradients (``AllPairs.energy``);
* ``build``    a receptor's potential grids, neighbour lists and records (``Grid.build``);
* ``serve``    docking requests on host data through the continuous-batching ``DockingServer``.

The receptors, ligands and poses are those of ``attract_b200.synth`` (uniform
coarse-grained receptors, random-walk ligands, poses uniform in a ball or at
the receptor's surface).  Everything follows from the seed.
"""
import math

import numpy as np
import torch

import attract_b200 as A
from attract_b200 import synth
from attract_b200.allpairs import AllPairs
from attract_b200.autograd import docking_energy
from attract_b200.poses import pose_to_mat, random_in_ball, random_rotations
from attract_b200.reference_api import GRAVITY, SCHEMA
from attract_b200.serve import DockingServer, Request, lanes_by_size

CUTOFF = 10.0   # Angstrom: reach of a receptor bead's potential
PLATEAU = 5.0   # Angstrom: the neighbour lists' reach
SPACING = 0.9   # Angstrom: the inner grid (the outer grid has twice that)


def listed():
    return [
        # a few poses of a small fragment looked at by hand or by a driving script: all latency
        dict(name="eval_few", kind="eval", rec=1200, types=32, beads=7, poses=16, pose="euler", place="ball",
             mode="reference", gravity=False),
        # one step of an outer optimiser over a batch of trinucleotide poses
        dict(name="eval_batch", kind="eval", rec=2500, types=32, beads=24, poses=65536, pose="euler", place="ball",
             mode="reference", gravity=False),
        # a large ligand at the receptor's surface, matrices in and dE/dmat out, as the reference's callers pass them
        dict(name="eval_large_ligand", kind="eval", rec=5000, types=8, beads=301, poses=3000, pose="matrix",
             place="surface", mode="reference", gravity=True),
        # differentiation with respect to the poses and to the grid values (fitting the potential)
        dict(name="autograd", kind="autograd", rec=2500, types=32, beads=24, poses=65536, mode="analytic"),
        # a plain small minimisation: one 7-bead fragment
        dict(name="minimise_small", kind="minimise", rec=1200, types=32, fragments=1, lo=7, hi=7, poses=4096, steps=100,
             place="ball25", graph=False),
        # the batched minimisation of six uneven fragments in one graph-captured launch
        dict(name="minimise_batch", kind="minimise", rec=2500, types=32, fragments=6, lo=18, hi=30, poses=20000,
             steps=200, place="ball", graph=True),
        # a 40-bead ligand refined at the surface of a dense receptor: long neighbour lists
        dict(name="minimise_surface", kind="minimise", rec=5000, types=32, fragments=1, lo=40, hi=40, poses=100000,
             steps=50, place="surface", graph=False),
        # the reference's own protocol: 375 adabelief epochs on quaternions, with gravity in the first stages
        dict(name="schema", kind="schema", rec=2500, types=32, beads=24, poses=20000, epochs=375),
        # rescoring a handful of final poses against every receptor bead
        dict(name="rescore_few", kind="rescore", rec=2500, types=32, beads=24, poses=10, pose="euler", rcut=0.0),
        # rescoring a whole pose library, with gradients
        dict(name="rescore_library", kind="rescore", rec=2500, types=32, beads=24, poses=16384, pose="euler", rcut=0.0),
        # loading a receptor: potentials of every bead type, neighbour lists, records
        dict(name="build_receptor", kind="build", rec=2500, types=32),
        # a burst of docking requests of uneven ligands on two resident receptors, from host poses to host results
        dict(name="serve_burst", kind="serve", rec=1500, rec2=3000, types=32, requests=24, lo=5, hi=60, poses=4000,
             steps=200, round_steps=50),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any of the kinds, sizes over the whole range."""
    kind = rng.choice(["eval", "eval", "eval", "autograd", "minimise", "minimise", "minimise", "schema", "rescore",
                       "rescore", "build", "build", "serve"])
    types = rng.choice([4, 8, 13, 32])
    rec = _log(rng, 150, 5000)
    if kind == "eval":
        beads = _log(rng, 3, 320)
        return dict(kind=kind, rec=rec, types=types, beads=beads, poses=_log(rng, 1, min(65536, 1_500_000 // beads)),
                    pose=rng.choice(["euler", "euler", "matrix"]), place=rng.choice(["ball", "surface"]),
                    mode=rng.choice(["reference", "analytic"]), gravity=rng.random() < 0.3)
    if kind == "autograd":
        beads = _log(rng, 4, 100)
        return dict(kind=kind, rec=min(rec, 2500), types=types, beads=beads,
                    poses=_log(rng, 64, min(65536, 1_500_000 // beads)), mode=rng.choice(["reference", "analytic"]))
    if kind == "minimise":
        lo = _log(rng, 3, 48)
        hi = min(60, lo + rng.choice([0, 3, 12]))
        steps = rng.choice([25, 50, 100, 200])
        fragments = rng.choice([1, 1, 2, 6])
        most = 500_000_000 // (steps * (lo + hi) // 2 * fragments)
        return dict(kind=kind, rec=rec, types=types, fragments=fragments, lo=lo, hi=hi,
                    poses=_log(rng, 100, max(200, min(100_000, most))), steps=steps,
                    place=rng.choice(["ball", "surface"]), graph=rng.random() < 0.5)
    if kind == "schema":
        beads = _log(rng, 5, 60)
        return dict(kind=kind, rec=min(rec, 2500), types=types, beads=beads,
                    poses=_log(rng, 100, 400_000 // beads), epochs=rng.choice([75, 375]))
    if kind == "rescore":
        beads = _log(rng, 3, 320)
        return dict(kind=kind, rec=rec, types=types, beads=beads,
                    poses=_log(rng, 1, max(2, min(65536, 980_000_000 // (beads * rec)))),
                    pose=rng.choice(["euler", "matrix"]), rcut=rng.choice([0.0, 0.0, 12.0, 50.0]))
    if kind == "build":
        return dict(kind=kind, rec=_log(rng, 60, 2500), types=types)
    lo = _log(rng, 4, 30)
    return dict(kind=kind, rec=_log(rng, 150, 1500), rec2=_log(rng, 150, 3000), types=types,
                requests=rng.choice([1, 3, 8, 24]), lo=lo, hi=min(60, 2 * lo), poses=_log(rng, 1000, 4000), steps=200,
                round_steps=rng.choice([25, 50]))


# ----------------------------------------------------------------------- inputs
def _f32(a):
    return np.asarray(a, np.float32).astype(np.float64)


def _tables(types, seed):
    """Symmetric per-type-pair sigma and epsilon, as ForceField.synthetic draws them."""
    rng = np.random.default_rng(seed)
    s, e = rng.uniform(3.0, 5.0, (types, types)), rng.uniform(0.1, 2.0, (types, types))
    return np.triu(s) + np.triu(s, 1).T, np.triu(e) + np.triu(e, 1).T


def _receptor(n, types, seed):
    """Uniform beads 3.5 A apart at 0.01 beads / A^3, up to 2500 of them in a sphere of 40 A."""
    radius = 40.0 if 1000 <= n <= 2500 else (n / (0.01 * 4.0 / 3.0 * np.pi)) ** (1.0 / 3.0)
    xyz, t, r = synth.receptor_beads(n, radius=radius, n_types=types, seed=seed)
    return _f32(xyz), t, r


def _ligand(n, types, rng):
    t = rng.integers(0, types, n)
    # a large ligand is compact: its walk's steps shrink so that it stays within about 20 A
    return _f32(synth.random_walk(n, rng, 3.8 if n <= 60 else 3.8 * math.sqrt(60 / n))), t


def _poses(case, xyz, radius, n, rng):
    place = case.get("place", "ball")
    if place == "surface":
        t = synth.surface_points(xyz, n, rng)
    else:
        t = random_in_ball(n, min(25.0 if place == "ball25" else 30.0, radius), rng)
    return np.concatenate([random_rotations(n, rng), t], 1).astype(np.float32)


def _inputs(case, seed):
    """Host inputs of the kinds with one receptor and one ligand."""
    rng = np.random.default_rng(seed)
    xyz, rt, radius = _receptor(case["rec"], case["types"], seed)
    lig, lt = _ligand(case["beads"], case["types"], rng)
    poses = _poses(case, xyz, radius, case["poses"], rng)
    if case.get("pose") == "matrix":
        m = pose_to_mat(poses)
        m[:, :3, 3] = 0.0
        poses = m.astype(np.float32)
    return xyz, rt, radius, lig, lt, poses


def _force_field(case, seed):
    sigma, eps = _tables(case["types"], seed)
    return A.ForceField.from_eps_sigma(eps, sigma)


def _geom(radius, types):
    return A.GridGeom.around((0.0, 0.0, 0.0), radius, spacing=SPACING, plateau=PLATEAU, n_types=types)


def _grid(case, seed, xyz, rt, radius, **kw):
    return A.Grid.build(xyz, rt, _force_field(case, seed), _geom(radius, case["types"]), cutoff=CUTOFF, device="cuda",
                        **kw)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "build":
        xyz, rt, radius = _receptor(case["rec"], case["types"], seed)
        return dict(case=case, args=(xyz, rt, _force_field(case, seed), _geom(radius, case["types"])))
    if kind == "serve":
        rng = np.random.default_rng(seed)
        grids = [_grid(case, seed, *_receptor(n, case["types"], seed + i))
                 for i, n in enumerate((case["rec"], case["rec2"]))]
        reqs = []
        # lognormal pose counts, the same ones in another order for another seed
        counts = case["poses"] * np.exp(np.random.default_rng(case["requests"]).normal(size=case["requests"]))
        for n in rng.permutation(np.clip(counts, 1000, 5 * case["poses"]).astype(int)):
            lig, lt = _ligand(int(rng.integers(case["lo"], case["hi"] + 1)), case["types"], rng)
            poses = np.concatenate([random_rotations(n, rng), random_in_ball(n, 30.0, rng)], 1).astype(np.float32)
            reqs.append((int(rng.integers(0, 2)), (lig, lt, lt), poses))
        server = DockingServer(grids, steps=case["steps"], round_steps=case["round_steps"], max_inflight_poses=500_000)
        return dict(case=case, server=server, requests=reqs)
    if kind == "minimise":
        rng = np.random.default_rng(seed)
        xyz, rt, radius = _receptor(case["rec"], case["types"], seed)
        sizes = sorted({int(round(v)) for v in np.linspace(case["lo"], case["hi"], case["fragments"])}, reverse=True)
        ligs = [_ligand(n, case["types"], rng) for n in sizes]
        poses = torch.from_numpy(_poses(case, xyz, radius, case["poses"] * len(sizes), rng)).cuda()
        lanes = lanes_by_size(sizes[0])
        wl = A.Workload([_grid(case, seed, xyz, rt, radius)], A.LigandSet([(x, t, t) for x, t in ligs], device="cuda"),
                        [A.Segment(0, i, case["poses"]) for i in range(len(sizes))], lanes_per_pose=lanes)
        launch = A.LaunchShape(lanes)
        plan = A.MinimisePlan(wl, case["steps"], launch=launch) if case["graph"] else None
        return dict(case=case, wl=wl, poses=poses, launch=launch, plan=plan)

    xyz, rt, radius, lig, lt, poses = _inputs(case, seed)
    if kind == "rescore":
        ap = AllPairs(xyz, rt, lig, lt, _force_field(case, seed), device="cuda")
        return dict(case=case, ap=ap, poses=torch.from_numpy(poses).cuda(), rcut=case["rcut"] or None)
    grid = _grid(case, seed, xyz, rt, radius, keep_dense=kind == "autograd")
    lanes = lanes_by_size(case["beads"])
    wl = A.Workload([grid], A.LigandSet([(lig, lt, lt)], device="cuda"), [A.Segment(0, 0, case["poses"])],
                    lanes_per_pose=lanes)
    if kind == "schema":
        q = np.random.default_rng(seed + 1).normal(size=(case["poses"], 4))
        q /= np.linalg.norm(q, axis=1, keepdims=True)
        qt = np.concatenate([q, poses[:, 3:], np.zeros((len(q), 1))], 1).astype(np.float32)
        schema = SCHEMA if case["epochs"] == sum(s[0] for s in SCHEMA) else SCHEMA[:4]
        return dict(case=case, wl=wl, poses=torch.from_numpy(qt).cuda(), schema=schema)
    opts = A.EvalOptions(grad_mode=case["mode"], gravity=GRAVITY if case.get("gravity") else 0.0)
    state = dict(case=case, wl=wl, poses=torch.from_numpy(poses).cuda(), opts=opts, launch=A.LaunchShape(lanes))
    if kind == "autograd":
        state["poses"].requires_grad_(True)
        grid.inner.requires_grad_(True)
        grid.outer.requires_grad_(True)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "eval":
        energy, grad, status = A.energrad(state["wl"], state["poses"], state["opts"], launch=state["launch"])
        return {"energy": energy, "grad": grad, "status": status}
    if kind == "autograd":
        grid, poses = state["wl"].grids[0], state["poses"]
        poses.grad = grid.inner.grad = grid.outer.grad = None
        energy = docking_energy(state["wl"], poses, state["opts"], reduce="none")
        energy.sum().backward()
        return {"energy": energy.detach(), "poses": poses.grad, "inner": grid.inner.grad, "outer": grid.outer.grad}
    if kind == "minimise":
        if state["plan"] is not None:
            state["plan"].pose_in.copy_(state["poses"])
            poses, energy, status = state["plan"].replay()
        else:
            poses, energy, status, _ = A.minimise(state["wl"], state["poses"], case["steps"], launch=state["launch"])
        return {"poses": poses, "energy": energy, "status": status}
    if kind == "schema":
        poses, energy, status = A.minimise_schema(state["wl"], state["poses"], state["schema"], gravity_weight=GRAVITY)
        return {"poses": poses[:, :7], "energy": energy, "status": status}
    if kind == "rescore":
        energy, grad = state["ap"].energy(state["poses"], rcut=state["rcut"], grad=True)
        return {"energy": energy, "grad": grad}
    if kind == "build":
        grid = A.Grid.build(*state["args"], cutoff=CUTOFF, device="cuda")
        # the lists at one length for every receptor of this size (a bead is in about 51 600 of them)
        lists = torch.nn.functional.pad(grid.nb_list, (0, 52_500 * case["rec"] - grid.nb_list.numel()))
        return {"bricks": grid.bricks, "headers": grid.nb_hdr, "lists": lists, "records": grid.nb_rec}
    server = state["server"]
    sent = [server.submit(Request(rec, lig, poses)) for rec, lig, poses in state["requests"]]
    server.run_until_idle()
    server.done.clear()
    return {"poses": np.concatenate([r.result_poses for r in sent]),
            "energy": np.concatenate([r.result_energies for r in sent]),
            "status": np.concatenate([r.result_status for r in sent])}


# ------------------------------------------------------------------------- work
def _points(radius):
    """(inner, outer) grid points and cells of a receptor of this radius."""
    n = int(math.ceil(2 * (radius + 10.0) / SPACING)) + 1
    n2 = int(math.ceil((n - 1 + 64) / 2.0)) + 1
    return n ** 3, n2 ** 3, (n - 1) ** 3, (n2 - 1) ** 3, (4 * (n - 1) + 1) ** 3


def _radius(rec):
    return 40.0 if 1000 <= rec <= 2500 else (rec / (0.01 * 4.0 / 3.0 * math.pi)) ** (1.0 / 3.0)


# a bead's evaluation: its 8 corners (128 B), its list's header and the entries within the plateau (about 5)
BEAD_BYTES, PAIRS, PAIR_FLOPS, BEAD_FLOPS = 128 + 8 + 10, 5, 45, 110


def work(case):
    kind = case["kind"]
    if kind == "build":
        pi, po, ci, co, pl = _points(_radius(case["rec"]))
        near = 4.0 / 3.0 * math.pi * CUTOFF ** 3 * 0.0095  # receptor beads that reach a point inside
        return {"bytes": 128 * case["types"] * (ci + co) + (8 + 32) * pl,
                "flops": 40.0 * case["types"] * case["rec"] * (4189 / SPACING ** 3) * 1.125 + near * 10 * pi}
    if kind == "rescore":
        pairs = case["poses"] * case["beads"] * case["rec"]
        return {"bytes": case["poses"] * (52 if case["pose"] == "euler" else 132) + 16 * (case["rec"] + case["beads"]),
                "flops": 30.0 * pairs}
    if kind == "serve":
        n, evals, beads = case["requests"] * case["poses"] * 1.5, case["steps"] + 1, (case["lo"] + case["hi"]) / 2
        io = 24 + 32
    elif kind == "minimise":
        sizes = {int(round(v)) for v in np.linspace(case["lo"], case["hi"], case["fragments"])}
        n, evals, beads, io = case["poses"] * len(sizes), case["steps"] + 1, sum(sizes) / len(sizes), 24 + 32
    elif kind == "schema":
        n, evals, beads, io = case["poses"], case["epochs"], case["beads"], 32 + 40
    else:
        matrix = case.get("pose") == "matrix"
        n, evals, beads, io = case["poses"], 2 if kind == "autograd" else 1, case["beads"], 136 if matrix else 56
    # grids far larger than the caches, beads that stay in their cells from step to step: the bricks of a
    # minimisation are read once per pose and bead, those of an evaluation once per bead
    reads = n * beads * BEAD_BYTES * (evals if kind == "autograd" else 1)
    extra = 16.0 * case["types"] * sum(_points(_radius(case["rec"]))[:2]) if kind == "autograd" else 0.0
    return {"bytes": reads + n * io + extra, "flops": float(n) * evals * beads * (BEAD_FLOPS + PAIRS * PAIR_FLOPS)}


# ------------------------------------------------------------------------ exact
# The energies and gradients in 64 bits, written with plain tensor operations.
def _pair64(d2, rc, ac, cap):
    """Energy and derivative by d^2 of rc r^-8 - ac r^-6, constant below the cap."""
    rr = 1.0 / torch.maximum(d2, cap)
    return (rc * rr - ac) * rr ** 3, torch.where(d2 < cap, 0.0, rr ** 4 * (3.0 * ac - 4.0 * rc * rr))


def _tables64(case, seed, ltypes):
    """rc, ac, cap, plateau energy and derivative [receptor type, ligand type]."""
    sigma, eps = (torch.tensor(t[:, ltypes], dtype=torch.float64, device="cuda") for t in _tables(case["types"], seed))
    rc, ac, cap = eps * sigma ** 8, eps * sigma ** 6, (0.6 * sigma) ** 2
    ep, gp = _pair64(torch.full_like(rc, PLATEAU ** 2), rc, ac, cap)
    return rc, ac, cap, ep, gp


def _frame(radius):
    """Origin, inner and outer points per axis, and the spacing as the grid holds it."""
    n = int(math.ceil(2 * (radius + 10.0) / SPACING)) + 1
    n2 = int(math.ceil((n - 1 + 64) / 2.0)) + 1
    return float(np.float32(-(n - 1) * SPACING / 2.0)), n, n2, float(np.float32(SPACING))


def _potentials64(tabs, xyz, rt, start, step, n):
    """[T, n, n, n, 4]: energy and force of the receptor on a cubic grid, per ligand type."""
    rc, ac, cap, ep, gp = tabs
    T = rc.shape[1]
    out = torch.zeros((4, T, n ** 3), dtype=torch.float64, device="cuda")
    w = int(2 * CUTOFF / step) + 2
    rec = torch.tensor(xyz, dtype=torch.float64, device="cuda")
    typ = torch.tensor(rt, device="cuda")
    for c0 in range(0, len(rec), 64):
        r, t = rec[c0:c0 + 64], typ[c0:c0 + 64]
        i = torch.ceil((r - CUTOFF - start) / step).long()[:, :, None] + torch.arange(w, device="cuda")  # [c, 3, w]
        d = start + i * step - r[:, :, None]
        ok = (i >= 0) & (i < n)
        d2 = d[:, 0, :, None, None] ** 2 + d[:, 1, None, :, None] ** 2 + d[:, 2, None, None, :] ** 2
        hit = (d2 < CUTOFF ** 2) & ok[:, 0, :, None, None] & ok[:, 1, None, :, None] & ok[:, 2, None, None, :]
        c, a, b, e = hit.nonzero(as_tuple=True)
        at = (i[c, 0, a] * n + i[c, 1, b]) * n + i[c, 2, e]
        q, ty = d2[c, a, b, e], t[c]
        v, dv = _pair64(q, *(x[ty].T for x in (rc, ac, cap)))
        near = q < PLATEAU ** 2
        v = torch.where(near, ep[ty].T, v)
        dv = -2.0 * torch.where(near, gp[ty].T * PLATEAU / q.clamp_min(1e-300).sqrt(), dv)
        out[0].index_add_(1, at, v)
        for k, dk in enumerate((d[c, 0, a], d[c, 1, b], d[c, 2, e])):
            out[k + 1].index_add_(1, at, dv * dk)
    return out.permute(1, 2, 0).reshape(T, n, n, n, 4)


def _cells64(dense):
    """[T, cells, 8, 4] of a dense grid: the 8 corners of every cell."""
    T, n = dense.shape[:2]
    return torch.stack([dense[:, a:n - 1 + a, b:n - 1 + b, c:n - 1 + c].reshape(T, -1, 4)
                        for a in (0, 1) for b in (0, 1) for c in (0, 1)], 2)


def _rotation64(p):
    """Column-form rotation, and the axes of the three Euler angles."""
    c, s = torch.cos(p[:, :3]), torch.sin(p[:, :3])
    (cp, cs, ct), (sp, ss, st) = c.unbind(1), s.unbind(1)
    q = torch.stack([cp * cs * ct + sp * st, cp * cs * st - sp * ct, cp * ss,
                     sp * cs * ct - cp * st, sp * cs * st + cp * ct, sp * ss, -ss * ct, -ss * st, cs], 1)
    zero, one = torch.zeros_like(cp), torch.ones_like(cp)
    axes = torch.stack([torch.stack([zero, zero, one], 1), torch.stack([-sp, cp, zero], 1),
                        -torch.stack([cp * ss, sp * ss, cs], 1)], 1)
    return q.reshape(-1, 3, 3), axes


def _placed64(case, poses, lig):
    """Bead positions, translations, and what turns bead gradients into pose gradients."""
    p = torch.tensor(poses, dtype=torch.float64, device="cuda")
    x = torch.tensor(lig, dtype=torch.float64, device="cuda")
    if case.get("pose") == "matrix":
        m, t = p[:, :3, :3], p[:, 3, :3]

        def back(g, dt):
            out = torch.zeros((len(g), 4, 4), dtype=torch.float64, device="cuda")
            out[:, :3, :3] = torch.einsum("nr,bnc->brc", x, g)
            out[:, 3, :3] = g.sum(1) + dt
            return out

        return torch.einsum("nr,brc->bnc", x, m) + t[:, None], t, back
    q, axes = _rotation64(p)
    t = p[:, 3:]
    X = torch.einsum("brc,nc->bnr", q, x) + t[:, None]

    def back(g, dt):
        torque = torch.linalg.cross(X - t[:, None], g).sum(1)
        return torch.cat([torch.einsum("bkc,bc->bk", axes, torque), g.sum(1) + dt], 1)

    return X, t, back


def _scored64(case, seed):
    """exact() of the eval and autograd kinds."""
    xyz, rt, radius, lig, lt, poses = _inputs(case, seed)
    used, slot = np.unique(lt, return_inverse=True)
    tabs = _tables64(case, seed, used)
    rc, ac, cap, ep, gp = tabs
    o, n, n2, h = _frame(radius)
    inner = _potentials64(tabs, xyz, rt, o, h, n)
    outer = _potentials64(tabs, xyz, rt, o - 32 * h, 2 * h, n2)
    rec, typ = torch.tensor(xyz, device="cuda"), torch.tensor(rt, device="cuda")
    slot = torch.tensor(slot, device="cuda")
    analytic = case["mode"] == "analytic"
    gravity = GRAVITY if case.get("gravity") else 0.0
    auto = case["kind"] == "autograd"
    dgrid = [torch.zeros(case["types"], g.shape[1] ** 3, dtype=torch.float64, device="cuda") if auto else None
             for g in (inner, outer)]
    energies, grads = [], []
    step = max(1, 60_000_000 // (case["beads"] * len(xyz)))
    for b0 in range(0, len(poses), step):
        X, t, back = _placed64(case, poses[b0:b0 + step], lig)
        B, N = X.shape[:2]
        X = X.reshape(-1, 3)
        sl = slot.repeat(B)
        v = (X - o) / h
        inn = ((v >= 0) & (v < n - 1)).all(1)
        u = (v + 32) / 2
        out = ~inn & ((u >= 0) & (u < n2 - 1)).all(1)
        E, G = torch.zeros(len(X), dtype=torch.float64, device="cuda"), torch.zeros_like(X)
        for which, grid, c, sc, dg in ((inn, inner, v, 1 / h, dgrid[0]), (out, outer, u, 0.5 / h, dgrid[1])):
            k = which.nonzero()[:, 0]
            i = torch.floor(c[k]).long()
            f = c[k] - i
            m = grid.shape[1]
            for a in range(8):
                bit = torch.tensor([a >> 2, (a >> 1) & 1, a & 1], device="cuda")
                w1 = torch.where(bit == 1, f, 1 - f)
                w = w1.prod(1)
                j = i + bit
                val = grid[sl[k], j[:, 0], j[:, 1], j[:, 2]]
                E[k] += w * val[:, 0]
                if analytic:
                    s = (2 * bit - 1).double() * sc
                    G[k] += val[:, :1] * s * torch.stack([w1[:, 1] * w1[:, 2], w1[:, 0] * w1[:, 2],
                                                          w1[:, 0] * w1[:, 1]], 1)
                else:
                    G[k] -= w[:, None] * val[:, 1:]
                if auto:
                    dg.view(-1).index_add_(0, torch.tensor(used, device="cuda")[sl[k]] * m ** 3 +
                                           (j[:, 0] * m + j[:, 1]) * m + j[:, 2], w)
        d2 = sum((X[:, None, k] - rec[None, :, k]) ** 2 for k in range(3))
        a, b = ((d2 < PLATEAU ** 2) & inn[:, None]).nonzero(as_tuple=True)
        q, ty, s = d2[a, b], typ[b], sl[a]
        e, de = _pair64(q, rc[ty, s], ac[ty, s], cap[ty, s])
        E.index_add_(0, a, e - ep[ty, s])
        de = 2 * de if analytic else 2 * de - 2 * gp[ty, s] * PLATEAU / q.sqrt()
        G.index_add_(0, a, de[:, None] * (X[a] - rec[b]))
        energies.append(E.reshape(B, N).sum(1) + gravity * (t * t).sum(1))
        grads.append(back(G.reshape(B, N, 3), 2 * gravity * t))
    energy, grad = torch.cat(energies), torch.cat(grads)
    if not auto:
        return {"energy": energy, "grad": grad, "status": None}
    full = [torch.zeros(case["types"], *g.shape[1:4], 4, dtype=torch.float64, device="cuda") for g in (inner, outer)]
    for f, d in zip(full, dgrid):
        f[..., 0] = d.view(f.shape[:-1])
    return {"energy": energy, "poses": grad, "inner": full[0], "outer": full[1]}


def _rescored64(case, seed):
    xyz, rt, _, lig, lt, poses = _inputs(case, seed)
    rc, ac, cap, _, _ = _tables64(case, seed, lt)
    rec = torch.tensor(xyz, device="cuda")
    ty = torch.tensor(rt, device="cuda")
    energies, grads = [], []
    step = max(1, 30_000_000 // (len(lig) * len(xyz)))
    for b0 in range(0, len(poses), step):
        X, t, back = _placed64(case, poses[b0:b0 + step], lig)
        d = X[:, :, None] - rec
        d2 = (d * d).sum(-1)
        e, de = _pair64(d2, *(x[ty].T for x in (rc, ac, cap)))
        if case["rcut"]:
            e, de = (torch.where(d2 < case["rcut"] ** 2, x, 0.0) for x in (e, de))
        energies.append(e.sum((1, 2)))
        grads.append(back(2 * (de[..., None] * d).sum(2), torch.zeros_like(t)))
    return {"energy": torch.cat(energies), "grad": torch.cat(grads)}


def exact(case, seed):
    if case["kind"] in ("eval", "autograd"):
        return _scored64(case, seed)
    if case["kind"] == "rescore":
        return _rescored64(case, seed)
    if case["kind"] == "build":
        xyz, rt, radius = _receptor(case["rec"], case["types"], seed)
        tabs = _tables64(case, seed, np.arange(case["types"]))
        o, n, n2, h = _frame(radius)
        cells = [_cells64(_potentials64(tabs, xyz, rt, *a)) for a in ((o, h, n), (o - 32 * h, 2 * h, n2))]
        return {"bricks": torch.cat(cells, 1), "headers": None, "lists": None, "records": None}
    return None  # a minimisation follows its rounding from step to step: no value to compare with
