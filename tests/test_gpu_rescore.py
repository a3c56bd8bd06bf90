"""The float64 re-score (one CTA per pose, culled and queued receptor pairs) against the float64 oracle: receptor sizes
around the staging batches and the list's capacity, ligands in every atom bucket, poses far from the receptor and the
clusters of many poses against a host restatement. Energies 1e-9 (float64 sums in another order), coordinates 1e-5."""
import numpy as np
import pytest
import torch

from helpers import lig_types, make_problem, random_states, SPACING

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("n_rec,n_heavy", [(1, 24), (127, 40), (128, 65), (129, 12), (1100, 24), (3000, 100)])
def test_rescore_over_receptor_sizes(n_rec, n_heavy):
    from adock_b200 import params, synth
    from adock_b200.grid import build_grid, grid_dims
    from adock_b200.kernel import B200KernelProblem
    from adock_b200.problem import pack_host
    from oracle.fp64 import Packed
    sfp = params.sf_params("vina")
    rng = np.random.default_rng(n_rec)
    xyz = rng.uniform(0, 16, (n_rec, 3)).astype(np.float32)   # dense: more atoms in reach than one list holds
    types = synth.MIX_TYPES[rng.integers(0, len(synth.MIX_TYPES), n_rec)]
    rec = synth.receptor_dict(xyz, types, np.full(3, 8.0), np.full(3, 9.0))
    ligs = [synth.ligand(n_heavy, 4, 9)]
    lt = lig_types(ligs)
    G = build_grid(xyz, types, sfp, rec["center"] - rec["size"] / 2, SPACING, grid_dims(rec["size"], SPACING), lt,
                   device=DEV).cpu().numpy()
    pg, pc = make_problem(rec, ligs, sfp, G, lt, DEV), make_problem(rec, ligs, sfp, G, lt, "cpu")
    kp = B200KernelProblem(pg)
    cl, st = random_states(pc, 12, seed=n_rec)
    st[-1, :3] += 300.0    # no receptor atom in reach
    et, ei, X = kp.rescore64(torch.as_tensor(cl, device=DEV), torch.as_tensor(st, device=DEV), exact=True)
    model = Packed(*pack_host(pc)[2:])
    Xw = model.pose_heavy(0, st)
    np.testing.assert_allclose(X[:, :n_heavy].cpu().numpy(), Xw, rtol=0, atol=5e-5)
    intra = model.intra(0, Xw)
    want = model.exact_inter(0, Xw, xyz, types) + intra + model.penalty(Xw, pc.gs.lo[0].numpy(), pc.gs.hi[0].numpy(),
                                                                         pc.gs.penalty)
    scale = np.abs(want) + 1.0
    # the kernel's scoring constants are float32
    assert np.abs(et.cpu().numpy() - want).max() / scale.max() < 1e-6
    assert np.abs(ei.cpu().numpy() - intra).max() / (np.abs(intra).max() + 1.0) < 1e-6


@pytest.mark.parametrize("P,n_out", [(1, 9), (32, 9), (100, 3), (257, 32)])
def test_clusters_match_the_serial_greedy(P, n_out):
    from adock_b200.kernel import B200KernelProblem
    from adock_b200 import params, synth
    sfp = params.sf_params("vina")
    rec = synth.receptor_dict(np.zeros((1, 3), np.float32), np.zeros(1, np.int64), np.zeros(3), np.full(3, 3.0))
    ligs = [synth.ligand(20, 3, 1), synth.ligand(45, 5, 2)]
    lt = lig_types(ligs)
    kp = B200KernelProblem(make_problem(rec, ligs, sfp, np.zeros((len(lt), 9, 9, 9), np.float32), lt, DEV))
    g = torch.Generator().manual_seed(P)
    L = 2
    X = (torch.randn(L, 12, 1, 3, generator=g)[:, torch.randint(0, 12, (P,), generator=g)] * 2
         + torch.randn(L, P, kp.AM, 3, generator=g) * 0.4)
    e = torch.randn(L * P, generator=g, dtype=torch.float64).round(decimals=1)   # with ties
    reps, cnt = kp.cluster(e.to(DEV), X.reshape(L * P, kp.AM, 3).to(DEV), L, P, 2.0, n_out)
    for l in range(L):
        na = ligs[l].n
        want = []
        for i in np.argsort(e[l * P:(l + 1) * P].numpy(), kind="stable"):
            d = [float(((X[l, i, :na] - X[l, j, :na]) ** 2).sum().div(na).sqrt()) for j in want]
            assert all(abs(v - 2.0) > 1e-5 for v in d)
            if all(v >= 2.0 for v in d):
                want.append(int(i))
            if len(want) == n_out:
                break
        assert reps[l, :cnt[l]].tolist() == want and (reps[l, cnt[l]:] == -1).all()
