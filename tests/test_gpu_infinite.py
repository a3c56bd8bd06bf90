"""Poses and starts of infinite energy keep their place behind the finite ones: a sort over a power of two of entries pads."""
import numpy as np
import pytest
import torch

from helpers import lig_types, make_problem

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
INF = float("inf")


def _problem():
    from adock_b200 import params, synth
    from adock_b200.kernel import B200KernelProblem
    rec = synth.receptor_dict(np.zeros((1, 3), np.float32), np.zeros(1, np.int64), np.zeros(3), np.full(3, 3.0))
    ligs = [synth.ligand(20, 3, 1), synth.ligand(25, 2, 2)]
    lt = lig_types(ligs)
    return B200KernelProblem(make_problem(rec, ligs, params.sf_params("vina"), np.zeros((len(lt), 9, 9, 9), np.float32), lt, DEV))


@pytest.mark.parametrize("P", [3, 5, 33, 100])
def test_clusters_with_infinite_energies(P):
    kp = _problem()
    e = torch.full((2, P), INF, dtype=torch.float64)
    e[:, P // 2] = 1.0
    e[0, 0] = float("nan")   # behind the finite energies, before the infinite ones
    X = (torch.arange(2 * P, dtype=torch.float32) * 10)[:, None, None].expand(2 * P, kp.AM, 3).contiguous()   # all apart
    reps, n = kp.cluster(e.reshape(-1).to(DEV), X.to(DEV), 2, P, 2.0, min(P, 32))
    for l in range(2):
        key = np.where(np.isnan(e[l].numpy()), 1.7e308, e[l].numpy())
        assert reps[l].tolist() == np.argsort(key, kind="stable")[:min(P, 32)].tolist() and int(n[l]) == min(P, 32)


@pytest.mark.parametrize("C,Q", [(1, 3), (3, 7), (12, 256)])
def test_starts_with_infinite_totals(C, Q):
    kp = _problem()
    L, M = 2, C * Q
    g = torch.Generator().manual_seed(Q)
    best_e = torch.full((L, C * Q), 3.4e38)
    best_e[:, ::3] = torch.randn(L, len(range(0, C * Q, 3)), generator=g)
    e_conf = torch.full((L, C), 3.4e38)   # conformers without a finite energy: 3.4e38 twice is infinite
    e_conf[:, 0] = 0.5
    quats = torch.randn(Q, 4, generator=g)
    theta, trans = torch.randn(L, C, kp.KM, generator=g), torch.randn(1, 2, 3, generator=g)
    best_i = torch.randint(0, 2, (L, C * Q), generator=g, dtype=torch.int32)
    d = [t.contiguous().to(DEV) for t in (best_e, best_i, e_conf, quats, theta, trans, torch.zeros(L, dtype=torch.int32))]
    state, e = kp.select_starts(*d, M)
    total = (best_e.view(L, C, Q) + e_conf[:, :, None]).reshape(L, C * Q)
    for l in range(L):
        order = np.argsort(total[l].numpy(), kind="stable")
        assert np.array_equal(e.view(L, M)[l].cpu().numpy(), total[l].numpy()[order])
        s = state.view(L, M, -1)[l].cpu().numpy()
        assert np.array_equal(s[:, :3], trans[0].numpy()[best_i[l].numpy()[order]])
        assert np.array_equal(s[:, 3:7], quats.numpy()[order % Q])
        assert np.array_equal(s[:, 7:], theta[l].numpy()[order // Q])
