"""The intra-pair loop of the search kernels: how the slots of a round are linked (adock_prepare), and energies and
gradients of ligands whose rounds repeat atoms the most (few atoms, one rotatable bond) or fill every atom bucket,
against the oracle's C restatement at the parity bar of test_gpu_parity.py (1e-4)."""
import numpy as np
import pytest
import torch

from helpers import lig_types, make_problem, random_states, receptor, rel_close, vec_rel, SPACING

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
SIZES = [(4, 1), (6, 1), (8, 2), (12, 1), (31, 6), (32, 1), (33, 9), (64, 12), (65, 10), (96, 8), (100, 16)]


def _problems(n_heavy, n_rot):
    from adock_b200 import params, synth
    from adock_b200.grid import build_grid, grid_dims
    sfp = params.sf_params("vina")
    rec = receptor("small")
    ligs = [synth.ligand(n_heavy, n_rot, 40 + n_heavy)]
    lt = lig_types(ligs)
    o = rec["center"] - rec["size"] / 2
    G = build_grid(rec["rec_xyz"], rec["rec_types"], sfp, o, SPACING, grid_dims(rec["size"], SPACING), lt,
                   device=DEV).cpu().numpy()
    return make_problem(rec, ligs, sfp, G, lt, DEV), make_problem(rec, ligs, sfp, G, lt, "cpu")


@pytest.mark.parametrize("n_heavy,n_rot", SIZES)
def test_rounds_are_linked_in_lane_order(n_heavy, n_rot):
    from adock_b200.kernel import B200KernelProblem
    pg, _ = _problems(n_heavy, n_rot)
    kp = B200KernelProblem(pg)
    rec = kp.t_work[3].view(-1, 32, 2).cpu().numpy()
    for x, y in zip(rec[:, :, 0], rec[:, :, 1]):
        lanes = np.flatnonzero(x >= 0)
        for side in (0, 1):
            atom = (x >> (8 * side)) & 0xff
            most = 0
            for a in np.unique(atom[lanes]):
                chain = [k for k in lanes if atom[k] == a]
                want = dict(zip(chain, chain[1:] + chain[-1:]))
                assert all((x[k] >> (18 + 5 * side)) & 31 == want[k] for k in chain)
                assert [(x[k] >> (28 + side)) & 1 for k in chain] == [1] + [0] * (len(chain) - 1)
                most = max(most, len(chain) - 1)
            if len(lanes):
                assert ((y >> (5 * side)) & 31 == most).all()


@pytest.mark.parametrize("n_heavy,n_rot", SIZES)
def test_energy_and_gradient_over_atom_buckets(n_heavy, n_rot):
    from adock_b200.kernel import B200KernelProblem
    from oracle.port import PortProblem
    pg, pc = _problems(n_heavy, n_rot)
    kp = B200KernelProblem(pg)
    cl, st = random_states(pc, 16, seed=n_heavy)
    for exact in (False, True):
        e, g = kp.energy_grad(torch.as_tensor(cl, device=DEV), torch.as_tensor(st, device=DEV), exact=exact)
        ec, gc = PortProblem.from_problem(pc).energy_grad(cl, st, exact=exact)
        D = 6 + pc.lb.preps[0].n_tors
        assert rel_close(e.cpu().numpy(), ec) < 1e-4
        assert vec_rel(g.cpu().numpy()[:, :D], gc[:, :D]) < 1e-4


@pytest.mark.parametrize("n_rec", [1, 31, 33, 63, 64, 65, 129])
def test_exact_energy_over_receptor_tiles(n_rec):
    """The exact inter energy stages receptor atoms in tiles of 64: sizes around the tile, each with ligands that use
    one, two and three atoms per lane, and the same sums through a neighbour list that holds every atom."""
    from adock_b200 import params, synth
    from adock_b200.grid import build_grid, grid_dims
    from adock_b200.kernel import B200KernelProblem
    from oracle.port import PortProblem
    sfp = params.sf_params("vina")
    xyz, types = synth.receptor(129, 14.0, min_sep=2.0, seed=3)
    rec = synth.receptor_dict(xyz[:n_rec], types[:n_rec], np.full(3, 7.0), np.full(3, 9.0))
    for n_heavy in (24, 40, 70):
        ligs = [synth.ligand(n_heavy, 3, 7)]
        lt = lig_types(ligs)
        n = grid_dims(rec["size"], SPACING)
        G = build_grid(rec["rec_xyz"], rec["rec_types"], sfp, rec["center"] - rec["size"] / 2, SPACING, n, lt,
                       device=DEV).cpu().numpy()
        pg, pc = make_problem(rec, ligs, sfp, G, lt, DEV), make_problem(rec, ligs, sfp, G, lt, "cpu")
        kp = B200KernelProblem(pg)
        cl, st = random_states(pc, 8, seed=n_rec)
        clg, stg = torch.as_tensor(cl, device=DEV), torch.as_tensor(st, device=DEV)
        e, g = kp.energy_grad(clg, stg, exact=True)
        ec, gc = PortProblem.from_problem(pc).energy_grad(cl, st, exact=True)
        D = 6 + pc.lb.preps[0].n_tors
        assert rel_close(e.cpu().numpy(), ec) < 1e-4
        assert vec_rel(g.cpu().numpy()[:, :D], gc[:, :D]) < 1e-4
        best_e = []
        for nbr in (None, torch.arange(n_rec, device=DEV, dtype=torch.int32).expand(len(cl), n_rec)):
            cur, best = stg.clone(), stg.clone()
            be = torch.full((len(cl),), float("inf"), device=DEV)
            kp.run_mc(clg, torch.arange(len(cl), device=DEV), cur, torch.zeros(len(cl), device=DEV), best, be, True, 0, 5,
                      1.2, 2.0, 2.0, 0, 0, exact=True, nbr=nbr,
                      nbr_n=None if nbr is None else torch.full((len(cl),), n_rec, device=DEV))
            best_e.append(be)
        assert torch.equal(*best_e)


@pytest.mark.parametrize("n_heavy,n_rot", [(12, 0), (24, 5), (60, 15), (110, 27), (120, 32)])
def test_one_bfgs_iteration_matches_the_restatement(n_heavy, n_rot):
    """One BFGS iteration (first direction, line search with its gradient-free trials, first update) and its energies
    on >= 99 % of the chains within 1e-3 (the bar of test_gpu_parity.py), for BFGS vectors of up to 38 components."""
    from adock_b200.kernel import B200KernelProblem
    from oracle.port import PortProblem
    pg, pc = _problems(n_heavy, n_rot)
    kp = B200KernelProblem(pg)
    cl, st = random_states(pc, 128, seed=2, sigma=1.0)
    st[:, 7:] = 0.0
    M = len(cl)
    ci = np.arange(M, dtype=np.int32)
    cur, best, be = st.copy(), st.copy(), np.full(M, np.inf, np.float32)
    PortProblem.from_problem(pc).run_mc(cl, ci, cur, np.zeros(M, np.float32), best, be, True, 0, 1, 1.2, 2.0, 2.0, 0, 0)
    cg, bg = torch.as_tensor(st, device=DEV).clone(), torch.as_tensor(st, device=DEV).clone()
    beg = torch.full((M,), float("inf"), device=DEV)
    kp.run_mc(torch.as_tensor(cl, device=DEV), torch.as_tensor(ci, device=DEV), cg, torch.zeros(M, device=DEV), bg, beg,
              True, 0, 1, 1.2, 2.0, 2.0, 0, 0)
    ok = np.abs(be - beg.cpu().numpy()) <= 1e-3 * np.maximum(np.abs(be), 1)
    assert ok.mean() >= 0.99, ok.mean()
