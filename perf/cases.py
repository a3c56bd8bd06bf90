"""Performance cases of the docking library: what a user's program has it do, through its public entry points.

Every case is a dict of plain values; ``prepare`` makes what a program has in hand before the call (receptor, ligand
batch, maps, packed problem, network), ``run`` is one pass, ``work`` the bytes and operations that pass cannot do
without and ``exact`` its result in 64 bits where it has one. The kinds:

maps      Vina / Vinardo maps of one receptor (``grid.prepare_grid``): once per receptor of a screen
fitted    maps of the fitted function (``grid.prepare_grid_fit``): once per receptor of a rescoring screen
energy    energies and gradients of a batch of poses (``B200KernelProblem.energy_grad``): rescoring, checks, external
          optimisers; grid maps in any storage type, or exact over the receptor's atoms
mc        start optimisation + Monte-Carlo steps (``run_mc``), the search's main phase, with the launch variant that
          the search's autotuner picks
polish    receptor neighbour lists and exact BFGS of each ligand's best chains (``receptor_neighbours``, ``run_mc``)
stage_a   start poses of a batch (``search.stage_a_starts``)
finalize  float64 re-score, clustering and output coordinates (``rescore64``, ``cluster``, ``pose_atoms``)
proposal  one segment's learned targets: features, network, sampling (``prop_features``, ``ProposalNet.forward``,
          ``prop_sample``)
train     loss and gradients of a minibatch of the proposal network (``ProposalNet.loss_grad``)
dock      the whole search of a batch (``search.dock_problem_kernel``)

Receptors, ligands and box sizes are the synthetic workloads of ``adock_b200.synth``. The maps that the search reads
are inputs here (made in plain torch), so that a case measures and compares only its own path. Monte Carlo, BFGS and
start selection branch on the last bit of an energy, so these kinds have no 64-bit value.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from adock_b200 import params, synth
from adock_b200.grid import GridSet, grid_dims, prepare_grid, prepare_grid_fit
from adock_b200.kernel import B200KernelProblem
from adock_b200.ligand import LigandBatch
from adock_b200.problem import PairPotential, Problem, pad_receptors
from adock_b200.proposal import IN, ProposalNet
from adock_b200.search import dock_problem_kernel, stage_a_starts

DEV = "cuda"
SPACING, PENALTY = params.GRID_SPACING, params.OUT_OF_BOX_PENALTY


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a protein pocket at full size: 8,000 receptor atoms, 30 A box (81^3 points), the 8 usual atom types
        {"name": "maps_vina", "kind": "maps", "atoms": 8000, "extent": 60.0, "box": 30.0, "types": 8, "sf": "vina"},
        # the same pocket with the fitted function's maps (108 receptor types, buried atoms)
        {"name": "maps_fitted", "kind": "fitted", "atoms": 8000, "extent": 60.0, "box": 30.0, "types": 8},
        # rescoring a library's poses on half-precision maps
        {"name": "energy_f16", "kind": "energy", "ligands": 64, "poses": 256, "large": False, "grid": "f16",
         "sf": "vina", "exact": False},
        # a handful of poses: launch and call overhead
        {"name": "energy_few", "kind": "energy", "ligands": 1, "poses": 32, "large": False, "grid": "f32",
         "sf": "vina", "exact": False},
        # one ligand docked alone (redocking): 32 chains, the latency of a chain
        {"name": "mc_single", "kind": "mc", "ligands": 1, "chains": 32, "steps": 32, "large": False, "grid": "f32"},
        # a screening batch: 256 ligands of 10-60 heavy atoms and 0-15 torsions, 32 chains each
        {"name": "mc_batch", "kind": "mc", "ligands": 256, "chains": 32, "steps": 8, "large": False, "grid": "f32"},
        # the best poses of a batch on exact receptor energies
        {"name": "polish", "kind": "polish", "ligands": 64, "poses": 32, "atoms": 1500, "iters": 100},
        # start poses of a batch with the default Stage-A settings
        {"name": "stage_a", "kind": "stage_a", "ligands": 64, "chains": 32, "box": 22.5},
        # final scores, clusters and coordinates of a screening batch
        {"name": "finalize", "kind": "finalize", "ligands": 256, "poses": 32, "atoms": 1500},
        # learned targets of a screening batch's chains for one 32-step segment with 4 tries per step
        {"name": "proposal", "kind": "proposal", "ligands": 256, "chains": 32, "targets": 128},
        # one training minibatch of the proposal network
        {"name": "train", "kind": "train", "batch": 4096},
        # a small screen from packed problem to ranked poses
        {"name": "dock", "kind": "dock", "ligands": 16, "chains": 32, "steps": 64},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["maps", "fitted", "energy", "mc", "polish", "stage_a", "finalize", "proposal", "train", "dock"])
    if kind in ("maps", "fitted"):
        atoms = _log_int(rng, 1200, 8000)
        extent = max(30.0, round(60.0 * (atoms / 8000) ** (1 / 3), 1))
        case = {"kind": kind, "atoms": atoms, "extent": extent, "box": round(rng.uniform(10.0, min(30.0, extent)), 2),
                "types": rng.randint(2, 8)}
        return dict(case, sf=rng.choice(["vina", "vinardo"])) if kind == "maps" else case
    if kind == "energy":
        exact = rng.random() < 0.25
        ligands, poses = _log_int(rng, 1, 64), _log_int(rng, 16, 256)
        return {"kind": kind, "ligands": ligands, "poses": poses if not exact else max(1, poses // 8),
                "large": rng.random() < 0.25, "grid": rng.choice(["f32", "f16", "bf16"]),
                "sf": rng.choice(["vina", "vinardo"]), "exact": exact}
    if kind == "mc":
        large = rng.random() < 0.2
        return {"kind": kind, "ligands": _log_int(rng, 1, 24 if large else 200), "chains": rng.randint(16, 32),
                "steps": rng.randint(4, 8), "large": large, "grid": rng.choice(["f32", "f16", "bf16"])}
    if kind == "polish":
        return {"kind": kind, "ligands": _log_int(rng, 1, 56), "poses": rng.randint(8, 32),
                "atoms": _log_int(rng, 1200, 1500), "iters": rng.randint(40, 100)}
    if kind == "stage_a":
        return {"kind": kind, "ligands": _log_int(rng, 1, 56), "chains": rng.randint(16, 256),
                "box": round(rng.uniform(14.0, 22.5), 2)}
    if kind == "finalize":
        return {"kind": kind, "ligands": _log_int(rng, 1, 240), "poses": rng.randint(8, 32),
                "atoms": _log_int(rng, 1200, 1500)}
    if kind == "proposal":
        return {"kind": kind, "ligands": _log_int(rng, 4, 256), "chains": rng.randint(16, 32),
                "targets": rng.choice([32, 64, 128])}
    if kind == "train":
        return {"kind": kind, "batch": _log_int(rng, 256, 4096)}
    return {"kind": "dock", "ligands": _log_int(rng, 1, 14), "chains": rng.randint(16, 32),
            "steps": rng.randint(16, 64)}


# ------------------------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=8)
def _receptor_points(atoms, extent):
    return synth.receptor(atoms, extent, seed=0)[0]


def _receptor(atoms, extent, box, seed):
    """Receptor of the seed: the base point set under a random symmetry of its cube, types drawn from the XS mix."""
    rng = np.random.default_rng([seed, 1])
    xyz = _receptor_points(atoms, extent)[:, rng.permutation(3)]
    flip = rng.integers(0, 2, 3).astype(bool)
    xyz = np.where(flip, np.float32(extent) - xyz, xyz).astype(np.float32)
    types = synth.MIX_TYPES[rng.choice(len(synth.MIX_TYPES), size=atoms, p=synth.MIX_P)]
    return synth.receptor_dict(xyz, types, np.full(3, extent / 2), np.full(3, box))


@functools.lru_cache(maxsize=2)
def _ligand_pool(large):
    return (synth.ligand_set(24, (65, 80), (10, 20), seed0=5000) if large
            else synth.ligand_set(320, (10, 60), (0, 15)))


def _ligands(n, large, seed):
    """n ligands: which ones is the case's (its padded sizes are then those of every seed), their order the seed's."""
    if n == 1 and not large:   # a drug-sized ligand for a ligand docked alone
        return [synth.ligand(24, 5, 0)]
    pool = _ligand_pool(large)
    pick = np.random.default_rng([n, 2]).choice(len(pool), size=n, replace=n > len(pool))
    return [pool[i] for i in np.random.default_rng([seed, 2]).permutation(pick)]


def _terms(r, rsum, p):
    """The five distance terms [5, ...] of pairs at distance r with radius sum rsum (ungated, zero past the cutoff)."""
    d = r - rsum
    near = (r < p["cutoff"]).to(r.dtype)
    ramp = lambda good, bad: ((bad - d) / (bad - good)).clamp(0.0, 1.0)
    return torch.stack([torch.exp(-((d - p["g1_off"]) / p["g1_w"]) ** 2), torch.exp(-((d - p["g2_off"]) / p["g2_w"]) ** 2),
                        (d - p["rep_off"]).clamp(max=0.0) ** 2, ramp(p["hyd_good"], p["hyd_bad"]),
                        ramp(p["hb_good"], p["hb_bad"])]) * near


def _points(origin, dims, dtype):
    axes = [torch.arange(n, device=DEV, dtype=dtype) * SPACING + float(o) for n, o in zip(dims, origin)]
    return torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)


def _near_box(rec, cutoff):
    lo, hi = rec["center"] - rec["size"] / 2 - cutoff - 1e-3, rec["center"] + rec["size"] / 2 + cutoff + SPACING
    return ((rec["rec_xyz"] >= lo) & (rec["rec_xyz"] <= hi)).all(1)


def _plain_maps(rec, lig_types, sfp, dtype):
    """Maps [T, nx, ny, nz] of a receptor in plain torch."""
    keep = _near_box(rec, sfp["cutoff"])
    xyz = torch.as_tensor(rec["rec_xyz"][keep], device=DEV, dtype=dtype)
    t = rec["rec_types"][keep]
    dims = grid_dims(rec["size"], SPACING)
    pts = _points(rec["center"] - rec["size"] / 2, dims, dtype)
    on = lambda k: torch.as_tensor(np.asarray(sfp[k])[t] != 0, device=DEV).to(dtype)
    rad, hyd, don, acc = torch.as_tensor(sfp["radius"][t], device=DEV, dtype=dtype), on("hydrophobic"), on("donor"), on("acceptor")
    w = [sfp[k] for k in ("w_g1", "w_g2", "w_rep", "w_hyd", "w_hb")]
    out = torch.empty(len(lig_types), len(pts), device=DEV, dtype=dtype)
    step = max(1, (1 << 25) // max(1, len(xyz)))
    for a in range(0, len(pts), step):
        r = torch.cdist(pts[a:a + step], xyz, compute_mode="donot_use_mm_for_euclid_dist")
        for radius in np.unique(sfp["radius"][lig_types]):
            g1, g2, rep, ramp_hyd, ramp_hb = _terms(r, rad + float(radius), sfp)
            common = w[0] * g1.sum(1) + w[1] * g2.sum(1) + w[2] * rep.sum(1)
            for q in np.flatnonzero(sfp["radius"][lig_types] == radius):
                lt = lig_types[q]
                gate = (don if sfp["acceptor"][lt] else 0.0) + (acc if sfp["donor"][lt] else 0.0)
                e = common + (w[3] * (ramp_hyd @ hyd) if sfp["hydrophobic"][lt] else 0.0)
                if torch.is_tensor(gate):
                    e = e + w[4] * (ramp_hb @ gate.clamp(max=1.0))
                out[q, a:a + step] = e
    return out.view(len(lig_types), *dims)


def _problem(case, seed, atoms=1500, extent=40.0, box=22.5, sf="vina"):
    """A packed docking problem: one receptor, the case's ligands, FP32 maps of the ligands' types."""
    rec = _receptor(atoms, extent, box, seed)
    ligs = _ligands(case["ligands"], case.get("large", False), seed)
    sfp = params.sf_params(sf)
    lt = np.unique(np.concatenate([[0]] + [p.types for p in ligs]))
    maps = _plain_maps(rec, lt, sfp, torch.float32)
    slot = -np.ones((1, params.N_XS), np.int64)
    slot[0, lt] = np.arange(len(lt))
    f32 = lambda a: torch.tensor(np.asarray(a, np.float32)[None], device=DEV)
    lo, hi = rec["center"] - rec["size"] / 2, rec["center"] + rec["size"] / 2
    gs = GridSet([maps], f32(lo), f32(lo), f32(hi), SPACING, PENALTY, slot=torch.tensor(slot, device=DEV),
                 n_types=params.N_XS)
    prob = Problem(gs, LigandBatch(ligs, DEV), torch.zeros(len(ligs), dtype=torch.long, device=DEV),
                   PairPotential(sfp, DEV), rec=pad_receptors([rec], DEV))
    return prob, rec, sfp


def _poses(prob, kp, per_ligand, seed, spread=2.0, basins=None):
    """Random poses around the box centre, per_ligand for each ligand (ligand-major): chain ligands and states.
    basins: that many centres per ligand, with small displacements around them."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    L, n = prob.lb.L, per_ligand
    m = basins or n
    t = torch.randn(L, m, 3, device=DEV, generator=g) * spread + (prob.gs.lo[0] + prob.gs.hi[0]) / 2
    q = torch.randn(L, m, 4, device=DEV, generator=g)
    th = (torch.rand(L, m, prob.lb.K, device=DEV, generator=g) * 2 - 1) * math.pi * prob.lb.tvalid[:, None]
    if basins:
        pick = torch.randint(0, m, (L, n), device=DEV, generator=g)
        take = lambda x: x.gather(1, pick[..., None].expand(L, n, x.shape[2]))
        t, q, th = take(t), take(q), take(th)
        t = t + 0.3 * torch.randn(L, n, 3, device=DEV, generator=g)
    q = q / q.norm(dim=-1, keepdim=True)
    lig = torch.arange(L, device=DEV, dtype=torch.int32).repeat_interleave(n)
    return lig, kp.pack(t.reshape(-1, 3), q.reshape(-1, 4), th.reshape(L * n, -1))


def _mc_args(cfg):
    return cfg["mc_temperature"], cfg["mc_amp_pos"], cfg["mc_amp_rot"]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("maps", "fitted"):
        rec = _receptor(case["atoms"], case["extent"], case["box"], seed)
        origin, dims = rec["center"] - rec["size"] / 2, grid_dims(rec["size"], SPACING)
        lt = np.sort(synth.MIX_TYPES)[:case["types"]].astype(np.int32)
        if kind == "maps":
            sfp = params.sf_params(case["sf"])
            launch, size, shape = prepare_grid(rec["rec_xyz"], rec["rec_types"], sfp, origin, SPACING, dims, lt, device=DEV)
            more = {"sfp": sfp}
        else:
            spec = params.fitted_spec()
            pot = params.FittedPotential(spec, params.fitted_weights(), lt)
            ext = params.receptor_ext_types(rec["rec_xyz"], rec["rec_types"], spec)
            launch, size, shape = prepare_grid_fit(rec["rec_xyz"], ext, pot, origin, SPACING, dims, device=DEV)
            more = {"pot": pot, "ext": ext}
        return {"kind": kind, "rec": rec, "types": lt, "launch": launch, "shape": shape,
                "out": torch.empty(size, dtype=torch.float32, device=DEV), **more}
    if kind == "train":
        g = torch.Generator(device=DEV).manual_seed(seed)
        B = case["batch"]
        x = torch.randn(B, IN, device=DEV, generator=g)
        x[:, 275:] = 0   # the hint columns of a network without the hint
        y = torch.zeros(B, 32, device=DEV)
        y[:, :3] = 2.0 * torch.randn(B, 3, device=DEV, generator=g)
        y[:, 3:6] = 0.5 * torch.randn(B, 3, device=DEV, generator=g)
        nt = torch.randint(0, 16, (B, 1), device=DEV, generator=g)
        th = (torch.rand(B, 20, device=DEV, generator=g) * 2 - 1) * math.pi
        y[:, 6:26] = torch.where(torch.arange(20, device=DEV)[None] < nt, th, torch.zeros_like(th))
        y[:, 26] = nt[:, 0]
        return {"kind": kind, "net": ProposalNet(DEV, seed=seed, n_comp=3), "x": x.to(torch.bfloat16), "y": y}
    prob, rec, sfp = _problem(case, seed, atoms=case.get("atoms", 1500), box=case.get("box", 22.5),
                              sf=case.get("sf", "vina"))
    if kind == "dock":
        L = prob.lb.L
        c = torch.tensor(rec["center"], dtype=torch.float32, device=DEV)[None].expand(L, 3)
        return {"kind": kind, "prob": prob, "centers": c, "sizes": [rec["size"]] * L, "seed": seed,
                "cfg": params.workload_preset(case["chains"], case["steps"], polish_top=8)}
    kp = B200KernelProblem(prob, grid_dtype=case.get("grid", "f32"))
    state = {"kind": kind, "prob": prob, "kp": kp, "rec": rec, "sfp": sfp, "seed": seed}
    if kind == "energy":
        state["lig"], state["state"] = _poses(prob, kp, case["poses"], seed)
        state["exact"] = case["exact"]
    elif kind == "mc":
        cfg = params.workload_preset(case["chains"], case["steps"])
        state["lig"], state["state"] = _poses(prob, kp, case["chains"], seed)
        state["ids"] = torch.arange(len(state["lig"]), device=DEV, dtype=torch.int32)
        state["cfg"] = cfg
        kp.tune(state["lig"], state["state"])
    elif kind == "polish":
        cfg = params.workload_preset(case["poses"], 0, polish_iters=case["iters"])
        lig, start = _poses(prob, kp, case["poses"], seed)
        ids = torch.arange(len(lig), device=DEV, dtype=torch.int32)
        best = start.clone()
        # poses as the search hands them over: minima of the grid energy
        kp.run_mc(lig, ids, start, torch.zeros(len(lig), device=DEV), best,
                  torch.full((len(lig),), float("inf"), device=DEV), True, 0, 0, *_mc_args(cfg), seed, 0)
        state.update(lig=lig, ids=ids, state=best, cfg=cfg)
    elif kind == "stage_a":
        state["cfg"] = params.workload_preset(case["chains"], 0)
        L = prob.lb.L
        state["centers"], state["sizes"] = np.tile(rec["center"], (L, 1)), [rec["size"]] * L
    elif kind == "finalize":
        state["lig"], state["state"] = _poses(prob, kp, case["poses"], seed, basins=6)
        state["poses"], state["cfg"] = case["poses"], params.workload_preset(case["poses"], 0)
    elif kind == "proposal":
        state["lig"], state["state"] = _poses(prob, kp, case["chains"], seed)
        state["ids"] = torch.arange(len(state["lig"]), device=DEV, dtype=torch.int32)
        state["net"], state["targets"] = ProposalNet(DEV, seed=seed, n_comp=3), case["targets"]
    return state


# ------------------------------------------------------------------------------------------------ one pass
def _padded(results, n_out):
    """The result dicts of a search as arrays of one shape (a ligand may have fewer poses, a batch fewer atoms)."""
    out = {k: np.zeros((len(results), n_out)) for k in ("affinity", "inter", "intra", "total")}
    out["coords"] = np.zeros((len(results), n_out, 64, 3), np.float32)
    for l, r in enumerate(results):
        n, atoms = r["coords"].shape[:2]
        out["coords"][l, :n, :atoms] = r["coords"]
        for k in ("affinity", "inter", "intra", "total"):
            out[k][l, :n] = r[k]
    return out


def run(s):
    kind = s["kind"]
    if kind in ("maps", "fitted"):
        return s["launch"](s["out"]).view(s["shape"])
    if kind == "train":
        loss, grads = s["net"].loss_grad(s["x"], s["y"])
        return {"loss": loss, "grads": grads}
    if kind == "dock":
        return _padded(dock_problem_kernel(s["prob"], s["centers"], s["sizes"], s["cfg"], seed=s["seed"]), s["cfg"]["n_out"])
    kp = s["kp"]
    if kind == "energy":
        e, g = kp.energy_grad(s["lig"], s["state"], exact=s["exact"])
        return {"e": e, "g": g}
    if kind == "mc":
        cfg, n = s["cfg"], len(s["lig"])
        cur, best = s["state"].clone(), s["state"].clone()
        cur_e, best_e = torch.zeros(n, device=DEV), torch.full((n,), float("inf"), device=DEV)
        kp.run_mc(s["lig"], s["ids"], cur, cur_e, best, best_e, True, cfg["mc_steps"], cfg["bfgs_iters"], *_mc_args(cfg),
                  s["seed"], 0)
        return {"cur": cur, "cur_e": cur_e, "best": best, "best_e": best_e}
    if kind == "polish":
        cfg, n = s["cfg"], len(s["lig"])
        cur, best = s["state"].clone(), s["state"].clone()
        best_e = torch.full((n,), float("inf"), device=DEV)
        nbr, nbr_n = kp.receptor_neighbours(s["prob"], s["lig"], cur, s["prob"].lb.K, cfg["polish_nbr_margin"])
        kp.run_mc(s["lig"], s["ids"], cur, torch.zeros(n, device=DEV), best, best_e, True, 0, cfg["polish_iters"],
                  *_mc_args(cfg), s["seed"], 0, exact=True, nbr=nbr, nbr_n=nbr_n)
        return {"best": best, "best_e": best_e, "nbr_n": nbr_n}
    if kind == "stage_a":
        state, e = stage_a_starts(s["prob"], kp, s["centers"], s["sizes"], s["cfg"], s["seed"])
        return {"state": state, "e": e}
    if kind == "finalize":
        L, P, n_out = s["prob"].lb.L, s["poses"], s["cfg"]["n_out"]
        total, intra, X = kp.rescore64(s["lig"], s["state"], exact=True)
        reps, n_reps = kp.cluster(total, X, L, P, s["cfg"]["cluster_rmsd"], n_out)
        pick = (torch.arange(L, device=DEV)[:, None] * P + reps.clamp(min=0).long()).reshape(-1)
        return {"total": total, "intra": intra, "heavy": X, "reps": reps, "n_reps": n_reps,
                "coords": kp.pose_atoms(s["prob"].lb, s["lig"][pick], s["state"][pick])}
    feat = kp.prop_features(s["lig"], s["state"])
    out = s["net"].forward(feat)
    return {"features": feat, "out": out,
            "targets": kp.prop_sample(s["lig"], s["ids"], out, s["state"], s["targets"], s["seed"], 0, s["net"].n_comp)}


# ------------------------------------------------------------------------------------------------ work
PAIR_FLOPS = 40      # distance, two Gaussians, repulsion, ramps and the derivative of one atom pair
ATOM_FLOPS = 150     # kinematics, map interpolation with its gradient and the box penalty of one atom
HEAVY, PAIRS, TORS = 35, 500, 7        # means of the 10-60 atom ligands
HEAVY_L, PAIRS_L, TORS_L = 72, 2200, 14


def _eval_flops(large, near=0):
    na, pairs = (HEAVY_L, PAIRS_L) if large else (HEAVY, PAIRS)
    return na * (ATOM_FLOPS + near * PAIR_FLOPS) + pairs * PAIR_FLOPS


def work(case):
    kind = case["kind"]
    ball = 4 / 3 * math.pi * 8.0 ** 3
    if kind in ("maps", "fitted"):
        pts = (math.ceil(case["box"] / SPACING) + 1) ** 3
        near = case["atoms"] / case["extent"] ** 3 * ball
        radii = min(4, case["types"])
        return {"bytes": 16 * case["atoms"] + 4 * case["types"] * pts, "flops": pts * near * (10 + 25 * radii + 6 * case["types"])}
    if kind == "train":
        weights = IN * 256 + 256 * 256 + 256 * 64
        return {"bytes": case["batch"] * (2 * IN + 128) + 6 * weights, "flops": 6 * case["batch"] * weights}
    L, large = case["ligands"], case.get("large", False)
    na, nt = (HEAVY_L, TORS_L) if large else (HEAVY, TORS)
    n = L * case.get("chains", case.get("poses", 1))
    box = (math.ceil(case.get("box", 22.5) / SPACING) + 1) ** 3
    map_bytes = box * 8 * (2 if case.get("grid", "f32") != "f32" else 4)
    state_bytes = 4 * n * (14 + 2 * nt)
    near = case.get("atoms", 1500) / 40.0 ** 3 * ball
    if kind == "energy":
        return {"bytes": map_bytes + state_bytes, "flops": n * _eval_flops(large, near if case["exact"] else 0)}
    if kind == "mc":
        return {"bytes": map_bytes + 2 * state_bytes, "flops": n * (case["steps"] + 1) * (25 + na) / 3 * _eval_flops(large)}
    if kind == "polish":
        return {"bytes": 2 * state_bytes, "flops": n * case["iters"] * _eval_flops(False, near)}
    stage_a = L * 8 * 384 * (max(1.0, case.get("box", 22.5) / 1.5 - 1) ** 3 / 4) * na * 12
    if kind == "stage_a":
        return {"bytes": map_bytes + state_bytes, "flops": stage_a}
    if kind == "finalize":
        return {"bytes": state_bytes + 12 * n * na, "flops": n * (na * near + PAIRS) * PAIR_FLOPS}
    if kind == "proposal":
        weights = IN * 256 + 256 * 256 + 256 * 64
        return {"bytes": n * (2 * IN + 256 + 128 * case["targets"]), "flops": 2 * n * weights + 400 * n * case["targets"]}
    steps = n * ((case["steps"] + 1) * (25 + na) / 3 + 100)
    return {"bytes": map_bytes + 2 * state_bytes, "flops": stage_a + steps * _eval_flops(False) + 8 * L * 100 * _eval_flops(False, near)}


# ------------------------------------------------------------------------------------------------ 64-bit results
def _rotation(q):
    w, x, y, z = (q / q.norm(dim=-1, keepdim=True)).unbind(-1)
    return torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                        2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                        2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1).view(*q.shape[:-1], 3, 3)


def _f64(a):
    return torch.as_tensor(np.asarray(a), device=DEV).double()


def _coords(p, st):
    """World coordinates [n, atoms, 3] of ligand p in states st [n, >= 7 + torsions] (float64)."""
    ref = _f64(p.ref)
    X = ref.expand(len(st), -1, -1)
    for k in range(p.n_tors):
        a, b = p.tors_axis[k]
        u = ref[b] - ref[a]
        u = u / u.norm()
        v = X - ref[a]
        c, s = torch.cos(st[:, 7 + k])[:, None, None], torch.sin(st[:, 7 + k])[:, None, None]
        turned = ref[a] + v * c + torch.linalg.cross(u.expand_as(v), v) * s + u * (v @ u)[..., None] * (1 - c)
        X = torch.where(torch.as_tensor(p.tors_mask[k], device=DEV)[None, :, None], turned, X)
    return X @ _rotation(st[:, 3:7]).transpose(1, 2) + st[:, None, :3]


def _pair_sum(r, ti, tj, sfp):
    rad = _f64(sfp["radius"])
    on = lambda k, t: torch.as_tensor(np.asarray(sfp[k]) != 0, device=DEV)[t]
    g1, g2, rep, hyd, hb = _terms(r, rad[ti] + rad[tj], sfp)
    bond = (on("donor", ti) & on("acceptor", tj)) | (on("acceptor", ti) & on("donor", tj))
    return (sfp["w_g1"] * g1 + sfp["w_g2"] * g2 + sfp["w_rep"] * rep + sfp["w_hyd"] * hyd *
            (on("hydrophobic", ti) & on("hydrophobic", tj)) + sfp["w_hb"] * hb * bond).flatten(1).sum(1)


def _intra(p, X, sfp):
    i, j = (torch.as_tensor(p.pairs[:, k], device=DEV) for k in (0, 1))
    t = torch.as_tensor(p.types, device=DEV)
    return _pair_sum((X[:, i] - X[:, j]).norm(dim=-1), t[i], t[j], sfp)


def _inter_exact(p, X, rec, sfp):
    lo, hi = X.detach().amin((0, 1)).cpu().numpy() - 8.01, X.detach().amax((0, 1)).cpu().numpy() + 8.01
    keep = ((rec["rec_xyz"] >= lo) & (rec["rec_xyz"] <= hi)).all(1)
    rx, rt = _f64(rec["rec_xyz"][keep]), torch.as_tensor(rec["rec_types"][keep], device=DEV)
    t = torch.as_tensor(p.types, device=DEV)
    step = max(1, (1 << 22) // max(1, p.n * len(rt)))
    return torch.cat([_pair_sum((x[:, :, None] - rx).norm(dim=-1), t[:, None], rt[None], sfp) for x in X.split(step)])


def _inter_grid(p, X, gs, maps):
    dims = torch.tensor(maps.shape[1:], device=DEV)
    f = (X - gs.origin[0].double()) / gs.spacing
    fc = torch.minimum(f.clamp(min=0.0), (dims - 1).double() - 1e-4)
    i = fc.detach().floor().long()
    w = fc - i
    slot = gs.slot[0][torch.as_tensor(p.types, device=DEV)]
    e = 0.0
    for c in range(8):
        d = [(c >> k) & 1 for k in (2, 1, 0)]
        ww = math.prod(w[..., k] if d[k] else 1 - w[..., k] for k in range(3))
        e = e + ww * maps[slot, i[..., 0] + d[0], i[..., 1] + d[1], i[..., 2] + d[2]]
    return e.sum(1)


def _penalty(X, gs):
    over = (gs.lo[0].double() - X).clamp(min=0) ** 2 + (X - gs.hi[0].double()).clamp(min=0) ** 2
    return gs.penalty * over.sum((1, 2))


def _exact_maps(s):
    return _plain_maps(s["rec"], s["types"], s["sfp"], torch.float64)


def _exact_fitted(s):
    rec, pot = s["rec"], s["pot"]
    spec = pot.spec
    keep = _near_box(rec, spec.cutoff)
    xyz, ext = _f64(rec["rec_xyz"][keep]), s["ext"][keep]
    rad, W = _f64(spec.rec_radius[ext]), _f64(pot.W[ext])
    pts = _points(rec["center"] - rec["size"] / 2, s["shape"][1:], torch.float64)
    out = torch.empty(len(pot.radius), len(pts), device=DEV, dtype=torch.float64)
    p = dict(spec.prm, cutoff=spec.cutoff)
    step = max(1, (1 << 24) // max(1, len(xyz)))
    for a in range(0, len(pts), step):
        r = torch.cdist(pts[a:a + step], xyz, compute_mode="donot_use_mm_for_euclid_dist")
        ion = (1 / r.clamp(min=spec.ion_rmin) ** 2 - 1 / spec.cutoff ** 2) * (r < spec.cutoff)
        for radius in np.unique(pot.radius):
            t = _terms(r, rad + float(radius), p)
            if spec.rep_cap is not None:
                t[2].clamp_(max=spec.rep_cap)
            for q in np.flatnonzero(pot.radius == radius):
                out[q, a:a + step] = sum(t[b] @ W[:, q, b] for b in range(5)) + ion @ W[:, q, 5]
    return out.view(s["shape"])


def _exact_energy(s, grid):
    prob, sfp, gs = s["prob"], s["sfp"], s["prob"].gs
    maps = gs.flat.view(-1, *gs.dims[0].tolist())
    if grid == "f16":
        maps = maps.clamp(-65504.0, 65504.0).half()
    maps = (maps.bfloat16() if grid == "bf16" else maps).double()
    e = torch.empty(len(s["lig"]), device=DEV, dtype=torch.float64)
    g = torch.zeros(len(s["lig"]), s["kp"].DM, device=DEV, dtype=torch.float64)
    for l, p in enumerate(prob.lb.preps):
        rows = torch.nonzero(s["lig"] == l)[:, 0]
        st = s["state"][rows].double()
        X = _coords(p, st).requires_grad_(True)
        inter = _inter_exact(p, X, s["rec"], sfp) if s["exact"] else _inter_grid(p, X, gs, maps)
        el = inter + _penalty(X, gs) + (_intra(p, X, sfp) if len(p.pairs) else 0.0)
        F, = torch.autograd.grad(el.sum(), X)
        X = X.detach()
        e[rows] = el.detach()
        g[rows, :3] = F.sum(1)
        g[rows, 3:6] = torch.linalg.cross(X - st[:, None, :3], F).sum(1)
        for k in range(p.n_tors):
            a, b = p.tors_axis[k]
            u = X[:, b] - X[:, a]
            u = u / u.norm(dim=-1, keepdim=True)
            m = torch.as_tensor(p.tors_mask[k], device=DEV)
            g[rows, 6 + k] = (torch.linalg.cross(X[:, m] - X[:, a:a + 1], F[:, m]).sum(1) * u).sum(1)
    return {"e": e, "g": g}


def _exact_finalize(s):
    prob, sfp, kp = s["prob"], s["sfp"], s["kp"]
    n = len(s["lig"])
    total, intra = torch.empty(n, device=DEV, dtype=torch.float64), torch.empty(n, device=DEV, dtype=torch.float64)
    heavy = torch.zeros(n, kp.AM, 3, device=DEV, dtype=torch.float64)
    for l, p in enumerate(prob.lb.preps):
        rows = slice(l * s["poses"], (l + 1) * s["poses"])
        X = _coords(p, s["state"][rows].double())
        heavy[rows, :p.n] = X
        intra[rows] = _intra(p, X, sfp) if len(p.pairs) else 0.0
        total[rows] = intra[rows] + _inter_exact(p, X, s["rec"], sfp) + _penalty(X, prob.gs)
    return {"total": total, "intra": intra, "heavy": heavy, "reps": None, "n_reps": None, "coords": None}


def _silu(a):
    return a * torch.sigmoid(a)


def _net64(net, x, W=None, b=None):
    W = [w.double() for w in net.Wb] if W is None else W
    b = [v.double() for v in net.b] if b is None else b
    return _silu(_silu(x @ W[0] + b[0]) @ W[1] + b[1]) @ W[2] + b[2]


def _exact_proposal(s):
    prob, kp, gs = s["prob"], s["kp"], s["prob"].gs
    slog = lambda v: torch.sign(v) * torch.log1p(v.abs())
    st, lig = s["state"].double(), s["lig"].long()
    n, lb = len(st), prob.lb
    f = torch.zeros(n, IN, device=DEV, dtype=torch.float64)
    maps = gs.flat.view(-1, *gs.dims[0].tolist()).double()
    off = torch.tensor([[i % 3 - 1, (i // 3) % 3 - 1, i // 9 - 1] for i in range(27)], device=DEV) * 2.0
    # the nearest grid point is found in 32 bits, as a half-way position has no right answer
    at = ((s["state"][:, None, :3] + off.float() - gs.origin[0]) * (1.0 / SPACING)).round().long()
    at = torch.minimum(at.clamp(min=0), gs.dims[0] - 1)
    for q in range(min(8, len(maps))):
        f[:, q:216:8] = slog(maps[q, at[..., 0], at[..., 1], at[..., 2]])
    f[:, 216:219] = (st[:, :3] - (gs.lo[0] + gs.hi[0]).double() / 2) * 0.1
    f[:, 219:223] = st[:, 3:7] / st[:, 3:7].norm(dim=1, keepdim=True) * torch.where(st[:, 3:4] < 0, -1.0, 1.0)
    k = min(20, prob.lb.K, st.shape[1] - 7)
    live = lb.tvalid[lig][:, :k]
    f[:, 223:223 + 2 * k:2] = torch.sin(st[:, 7:7 + k]) * live
    f[:, 224:224 + 2 * k:2] = torch.cos(st[:, 7:7 + k]) * live
    desc = [[p.n / 64, p.n_tors / 20, p.rg / 10, len(p.pairs) / 2000] for p in lb.preps]
    f[:, 263:267] = _f64(desc)[lig]
    slot = gs.slot[0].cpu().numpy()
    f[:, 267:275] = _f64([np.bincount(slot[p.types], minlength=params.N_XS)[:8] / p.n for p in lb.preps])[lig]
    return {"features": f, "out": _net64(s["net"], f), "targets": None}


def _exact_train(s):
    net, y = s["net"], s["y"].double()
    W = [w.double().requires_grad_(True) for w in net.Wb]
    b = [v.double().requires_grad_(True) for v in net.b]
    o = _net64(net, s["x"].double(), W, b)
    ls = o[:, 32:58].clamp(-4.0, 2.0)
    live = (torch.arange(26, device=DEV)[None] < 6) | (torch.arange(26, device=DEV)[None] - 6 < y[:, 26:27])
    live[:, :3] = False   # the translation is a mixture of three components
    nll = (torch.where(live, 0.5 * ((y[:, :26] - o[:, :26]) * torch.exp(-ls)) ** 2 + ls, 0.0)).sum(1)
    mean = torch.stack([o[:, c:c + 3] for c in (0, 27, 58)], 1)
    logit = o[:, [26, 30, 61]]
    z = (y[:, None, :3] - mean) * torch.exp(-ls[:, None, :3])
    nll = nll + torch.logsumexp(logit, 1) - torch.logsumexp(logit - 0.5 * (z ** 2).sum(2), 1) + ls[:, :3].sum(1)
    loss = nll.mean()
    return {"loss": loss.detach()[None], "grads": list(torch.autograd.grad(loss, W + b))}


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("maps", "fitted", "energy", "finalize", "proposal", "train"):
        return None
    s = prepare(case, seed)
    if kind == "energy":
        return _exact_energy(s, case["grid"])
    return {"maps": _exact_maps, "fitted": _exact_fitted, "finalize": _exact_finalize, "proposal": _exact_proposal,
            "train": _exact_train}[kind](s)
