"""The float64 re-score pose by pose against the float64 oracle, with the receptor's part apart from the penalty, so that a
receptor pair left out or counted twice shows.

Both sides work in float64 from the same float32 inputs: a term is off by a few 1e-15 times its slope (below 1e-13 of the
largest terms) and sums of up to 3e5 terms in another order by 3e5 x 1.1e-16, together below 1e-10 of the sum of the absolute
terms; subtracting the penalty leaves its rounding."""
import copy

import numpy as np
import pytest
import torch

from helpers import lig_types, make_problem, random_states, SPACING

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("n_rec,n_heavy", [(1, 1), (1, 24), (31, 5), (127, 40), (128, 65), (129, 12), (895, 24), (1025, 33),
                                           (1100, 24), (3000, 100)])
def test_receptor_pairs_of_each_pose(n_rec, n_heavy):
    from adock_b200 import params, synth
    from adock_b200.grid import grid_dims
    from adock_b200.kernel import B200KernelProblem
    from adock_b200.problem import pack_host
    from oracle.fp64 import Packed
    sfp = params.sf_params("vina")
    rng = np.random.default_rng(n_rec)
    xyz = rng.uniform(0, 16, (n_rec, 3)).astype(np.float32)
    types = synth.MIX_TYPES[rng.integers(0, len(synth.MIX_TYPES), n_rec)]
    rec = synth.receptor_dict(xyz, types, np.full(3, 8.0), np.full(3, 9.0))
    ligs = [synth.ligand(n_heavy, min(4, n_heavy // 5), 9)]
    lt = lig_types(ligs)
    G = np.zeros((len(lt),) + tuple(grid_dims(rec["size"], SPACING)), np.float32)
    pg, pc = make_problem(rec, ligs, sfp, G, lt, DEV), make_problem(rec, ligs, sfp, G, lt, "cpu")
    kp = B200KernelProblem(pg)
    cl, st = random_states(pc, 12, seed=n_rec)
    st[-1, :3] += 300.0               # no receptor atom in reach
    st[-2, 0] += 8.0 + 4.0 * 1.7      # the receptor's edge
    et, ei, _ = kp.rescore64(torch.as_tensor(cl, device=DEV), torch.as_tensor(st, device=DEV), exact=True)
    et, ei = et.cpu().numpy(), ei.cpu().numpy()
    model = Packed(*pack_host(pc)[2:])
    size = copy.copy(model)           # the sum of the absolute terms
    size.w = np.abs(model.w)
    X = model.pose_heavy(0, st)
    inter, intra = model.exact_inter(0, X, xyz, types), model.intra(0, X)
    pen = model.penalty(X, pc.gs.lo[0].numpy(), pc.gs.hi[0].numpy(), pc.gs.penalty)
    assert inter[-1] == 0.0
    bar = 1e-10 * (1.0 + size.exact_inter(0, X, xyz, types) + size.intra(0, X)) + 1e-13 * pen
    assert (np.abs(ei - intra) <= bar).all()
    assert (np.abs(et - ei - pen - inter) <= bar).all()
