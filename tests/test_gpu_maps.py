"""Map builders at sizes around their tiles (one or two points per thread), type sets with more radii than one register
group, per-term maps, receptors that need several staging passes, and atoms on grid points, against the oracle's C
restatement at the map bar of test_gpu_parity.py (1e-5)."""
import numpy as np
import pytest
import torch

from helpers import rel_close

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _receptor(n, extent, seed, on_points=False):
    from adock_b200 import synth
    rng = np.random.default_rng(seed)
    xyz = rng.uniform(0, extent, (n, 3)).astype(np.float32)
    if on_points:
        xyz[: n // 4] = np.round(xyz[: n // 4] / 0.5) * 0.5
    return xyz, synth.MIX_TYPES[rng.integers(0, len(synth.MIX_TYPES), n)]


def _boundary(xyz, n, spacing, cutoff=8.0, band=1e-4):
    """Points where an atom lies within rounding of the cutoff: it may count on one side only."""
    from scipy.spatial import cKDTree
    pts = np.stack(np.meshgrid(*[spacing * np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3)
    t = cKDTree(xyz.astype(np.float64))
    return (t.query_ball_point(pts, cutoff + band, return_length=True) > t.query_ball_point(pts, cutoff - band,
                                                                                             return_length=True))


@pytest.mark.parametrize("n", [(1, 1, 1), (5, 4, 9), (33, 17, 8), (64, 65, 41)])
@pytest.mark.parametrize("sf,types", [("vina", list(range(18))), ("vinardo", [9]), ("vina", [0, 2, 17, 15])])
def test_vina_maps(n, sf, types):
    from adock_b200 import params
    from adock_b200.grid import build_grid
    from oracle import port
    sfp = params.sf_params(sf)
    xyz, ty = _receptor(900, 30.0, sum(n), on_points=True)
    keep = ~_boundary(xyz, n, 0.5)
    for per_term in (False, True):
        if per_term and n == (64, 65, 41):
            continue
        G = build_grid(xyz, ty, sfp, np.zeros(3), 0.5, n, types, per_term=per_term, device=DEV).cpu().numpy()
        R = port.build_grid(xyz, ty, sfp, np.zeros(3), 0.5, n, types, per_term=per_term)
        assert G.shape == R.shape
        k = G.shape[0] if not per_term else 5 * G.shape[1]
        assert rel_close(G.reshape(k, -1)[:, keep], R.reshape(k, -1)[:, keep], 1e-5) < 1e-5


@pytest.mark.parametrize("n", [(3, 3, 3), (40, 41, 47)])
@pytest.mark.parametrize("n_rec,extent,n_types", [(900, 25.0, 3), (6000, 22.0, 17)])
def test_fitted_maps(n, n_rec, extent, n_types):
    from adock_b200 import params
    from adock_b200.grid import build_grid_fit
    from oracle import port
    X = params.N_XS
    spec = params.FittedSpec("vina", buried_threshold=1, rep_cap=2.5)
    rng = np.random.default_rng(n_rec)
    pot = params.FittedPotential(spec, rng.normal(size=len(params.TERM_NAMES)).astype(np.float32),
                                 np.sort(rng.choice(3 * X, n_types, replace=False)))
    xyz, ty = _receptor(n_rec, extent, n_types, on_points=True)
    ext = ty + X * rng.integers(0, 6, n_rec)
    keep = ~_boundary(xyz, n, 0.5)
    G = build_grid_fit(xyz, ext, pot, np.zeros(3), 0.5, n, device=DEV).cpu().numpy()
    R = port.build_grid_fit(xyz, ext, pot.W, spec.rec_radius, pot.radius, spec.grid_prm(), np.zeros(3), 0.5, n)
    scale = np.abs(R).reshape(len(G), -1)[:, keep].max()
    # sums of thousands of terms of either sign: 1e-5 of the largest value where they cancel
    d = np.abs(G - R).reshape(len(G), -1)[:, keep]
    assert (d / np.maximum(np.abs(R).reshape(len(G), -1)[:, keep], 1.0)).max() < 1e-5 or d.max() < 1e-5 * scale
