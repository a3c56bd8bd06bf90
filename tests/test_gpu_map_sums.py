"""Fitted maps against float64 at each point's own scale (the sum of the absolute terms that cancel there), and the map and
pair-energy exponentials against exp() where they fade out."""
import numpy as np
import pytest
import torch

from test_gpu_maps import _boundary, _receptor

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _points(n, spacing):
    return np.stack(np.meshgrid(*[spacing * np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3)


@pytest.mark.parametrize("n", [(3, 3, 3), (23, 31, 17)])
@pytest.mark.parametrize("n_rec,extent,n_types", [(900, 25.0, 3), (2500, 22.0, 17)])
def test_fitted_map_points(n, n_rec, extent, n_types):
    """A term's distance carries 1 ulp of at most 8 A (4.8e-7 A) and the steepest term, a repulsion capped at 2.5, changes by 3.2
    per A: 1.5e-6 per unit of weight for each pair within reach, and 2^-24 of the sum for each of the additions."""
    from adock_b200 import params
    from adock_b200.grid import build_grid_fit
    X = params.N_XS
    spec = params.FittedSpec("vina", buried_threshold=1, rep_cap=2.5)
    rng = np.random.default_rng(n_rec)
    pot = params.FittedPotential(spec, rng.normal(size=len(params.TERM_NAMES)).astype(np.float32),
                                 np.sort(rng.choice(3 * X, n_types, replace=False)))
    xyz, ty = _receptor(n_rec, extent, n_types, on_points=True)
    ext = ty + X * rng.integers(0, 6, n_rec)
    G = build_grid_fit(xyz, ext, pot, np.zeros(3), 0.5, n, device=DEV).cpu().numpy().reshape(n_types, -1)
    keep = ~_boundary(xyz, n, 0.5)
    p, W = spec.prm, pot.W.astype(np.float64)
    gauss = lambda d, g: np.exp(-((d - p[g + "_off"]) / p[g + "_w"]) ** 2)
    ramp = lambda d, h: np.clip((p[h + "_bad"] - d) / (p[h + "_bad"] - p[h + "_good"]), 0, 1)
    for i, x in enumerate(_points(n, 0.5)):
        if not keep[i]:
            continue
        r = np.linalg.norm(xyz.astype(np.float64) - x, axis=1)
        near = r < spec.cutoff
        r, e = r[near], ext[near]
        ion = 1 / np.maximum(r, spec.ion_rmin) ** 2 - 1 / spec.cutoff ** 2
        for q in range(n_types):
            d = r - spec.rec_radius[e].astype(np.float64) - float(pot.radius[q])
            B = np.stack([gauss(d, "g1"), gauss(d, "g2"), np.minimum(np.minimum(d - p["rep_off"], 0) ** 2, 2.5),
                          ramp(d, "hyd"), ramp(d, "hb"), ion], 1)
            w = W[e, q]
            bar = 1.5e-6 * np.abs(w).sum() + 6 * len(r) * 2.0 ** -24 * (B * np.abs(w)).sum() + 1e-6
            assert abs(G[q, i] - (B * w).sum()) <= bar


@pytest.mark.parametrize("width", [0.5, 0.05])
def test_exponential_of_the_maps(width):
    """One atom, r^2 exact: r to 1 ulp, so u = (d - off) / w carries 2 ulp of 8 A over w; the exponential itself 2 ulp and its
    argument's rounding u^2 2^-22; results below 2^-126 are 0."""
    from adock_b200 import params
    from adock_b200.grid import build_grid
    sfp = dict(params.sf_params("vina"), g1_off=0.0, g1_w=width)
    at, n = np.array([[4.125, 4.625, 5.375]], np.float32), (40, 39, 41)
    g = build_grid(at, np.zeros(1, np.int64), sfp, np.zeros(3), 0.25, n, [0], per_term=True, device=DEV).cpu().numpy()[0].reshape(-1)
    r = np.linalg.norm(_points(n, 0.25) - at[0].astype(np.float64), axis=1)
    u = (r - 2 * float(np.float32(sfp["radius"][0]))) / width
    want = np.where(r < 8, np.exp(-u * u), 0.0)
    du = 2 * 8 * 2.0 ** -23 / width
    bar = want * np.expm1(2 * np.abs(u) * du + du * du + u * u * 2.0 ** -22 + 2.0 ** -22) + 2.0 ** -126
    far = np.abs(r - 8) < 1e-5
    assert (want[r < 8] < 2.0 ** -149).any() == (width < 0.1) and (np.abs(g - want) <= bar)[~far].all()


@pytest.mark.parametrize("width", [0.5, 0.05])
def test_exponential_of_the_pair_energies(width):
    """As above for a ligand of one atom on exact receptor energies; r = r^2 / sqrt(r^2) carries 4 ulp there."""
    from adock_b200 import params, synth
    from adock_b200.kernel import B200KernelProblem
    from helpers import lig_types, make_problem
    sfp = dict(params.sf_params("vina"), g1_off=0.0, g1_w=width, w_g1=1.0, w_g2=0.0, w_rep=0.0, w_hyd=0.0, w_hb=0.0)
    ligs = [synth.ligand(1, 0, 3)]
    lt = lig_types(ligs)
    at = np.zeros((1, 3), np.float32)
    rec = synth.receptor_dict(at, np.zeros(1, np.int64), np.zeros(3), np.full(3, 30.0))
    kp = B200KernelProblem(make_problem(rec, ligs, sfp, np.zeros((len(lt), 3, 3, 3), np.float32), lt, DEV))
    t = torch.zeros(2000, 3)
    t[:, 0] = torch.linspace(0.5, 7.9, 2000)
    q = torch.zeros(2000, 4)
    q[:, 0] = 1
    st = kp.pack(t.to(DEV), q.to(DEV), torch.zeros(2000, kp.KM, device=DEV))
    X = kp.rescore64(torch.zeros(2000, dtype=torch.int32, device=DEV), st)[2][:, 0].double().cpu().numpy()
    e = kp.energy_grad(torch.zeros(2000, dtype=torch.int32, device=DEV), st, exact=True)[0].double().cpu().numpy()
    rad = np.asarray(sfp["radius"], np.float32).astype(np.float64)
    r = np.linalg.norm(X, axis=1)
    u = (r - rad[0] - rad[int(ligs[0].types[0])]) / width
    want = np.exp(-u * u)
    du = 6 * 8 * 2.0 ** -23 / width
    bar = want * np.expm1(2 * np.abs(u) * du + du * du + u * u * 2.0 ** -22 + 2.0 ** -22) + 2.0 ** -126
    assert (np.abs(e - want) <= bar).all()


@pytest.mark.parametrize("n", [(13, 9, 10), (49, 50, 49)])   # one point per thread; two
@pytest.mark.parametrize("kind", ["vina", "fitted"])
def test_falling_ramps(kind, n):
    """Ramps with bad < good are 1 at large distances inside the cutoff; bars of test_gpu_map_terms.py."""
    import test_gpu_map_terms as terms
    from adock_b200 import params
    sfp = dict(params.sf_params("vina"), hyd_good=1.5, hyd_bad=0.5, hb_good=0.0, hb_bad=-0.7)
    (terms._check_vina if kind == "vina" else terms._check_fitted)(sfp, *terms._case(n), n)
