"""Map terms with parameters away from the two published functions' (ramps that are steps, Gaussians of zero width), term by
term against a float64 restatement."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
SPACING = 0.5
TYPES = [0, 3, 8, 9, 12, 1]   # hydrophobic, donor, acceptor, both, hydrophobic of another radius, none of these


def _receptor(n=400, extent=14.0, seed=3):
    from adock_b200 import synth
    rng = np.random.default_rng(seed)
    return rng.uniform(0, extent, (n, 3)).astype(np.float32), synth.MIX_TYPES[rng.integers(0, len(synth.MIX_TYPES), n)]


def _terms(r, rsum, p):
    """Unweighted g1, g2, rep, hyd, hb of pairs at distances r (float64); a step is 1 below its edge, a Gaussian of zero
    width 0; pairs at or beyond the cutoff add nothing."""
    d = r - rsum
    gauss = lambda off, w: np.exp(-((d - off) / w) ** 2) if w else np.zeros_like(d)
    ramp = lambda good, bad: np.clip((bad - d) / (bad - good), 0, 1) if good != bad else (d < bad).astype(float)
    out = [gauss(p["g1_off"], p["g1_w"]), gauss(p["g2_off"], p["g2_w"]), np.minimum(d - p["rep_off"], 0) ** 2,
           ramp(p["hyd_good"], p["hyd_bad"]), ramp(p["hb_good"], p["hb_bad"])]
    return np.stack(out) * (r < p["cutoff"])


def _want(xyz, ty, sfp, n, types):
    """Term maps [5, T, points] and the points without a pair within 1e-4 A of the cutoff, a ramp's ends or a zero width's offset."""
    pts = np.stack(np.meshgrid(*[SPACING * np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3)
    r = np.linalg.norm(pts[:, None] - xyz[None].astype(np.float64), axis=2)
    rad, hyd, don, acc = (np.asarray(sfp[k]) for k in ("radius", "hydrophobic", "donor", "acceptor"))
    rad = rad.astype(np.float64)
    out, keep = [], (np.abs(r - sfp["cutoff"]) > 1e-4).all(1)
    for t in types:
        T = _terms(r, rad[ty] + rad[t], sfp)
        T[3] *= (hyd[ty] != 0) & (hyd[t] != 0)
        T[4] *= ((don[ty] != 0) & (acc[t] != 0)) | ((acc[ty] != 0) & (don[t] != 0))
        out.append(T.sum(2))
        d = r - rad[ty] - rad[t]
        edges = [sfp[k] for k in ("hyd_good", "hyd_bad", "hb_good", "hb_bad")]
        for e in edges + [sfp[g + "_off"] for g in ("g1", "g2") if sfp[g + "_w"] == 0]:
            keep &= (np.abs(d - e) > 1e-4).all(1)
    return np.stack(out, 1), keep


CHANGED = {
    "hydrophobic step": dict(hyd_good=0.7, hyd_bad=0.7),
    "bond step at contact": dict(hb_good=0.0, hb_bad=0.0),
    "both steps": dict(hyd_good=1.5, hyd_bad=1.5, hb_good=-0.3, hb_bad=-0.3),
    "first Gaussian of zero width": dict(g1_w=0.0),
    "second Gaussian of zero width": dict(g2_w=0.0),
}
# A distance of at most 8 A carries 1 ulp (5e-7) and every term of the published widths changes by less than 20 times that
# (the repulsion at 4 A overlap by 8 times), so a pair's error is below 1e-5; adding n pairs rounds n times at 2^-24 of a
# sum that is at most the sum of the absolute terms.
BAR = 1e-5


def _allowed(pairs, total):
    return BAR * (1.0 + pairs) + pairs * 2.0 ** -24 * total


def _pairs(xyz, n):
    pts = np.stack(np.meshgrid(*[SPACING * np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3)
    return (np.linalg.norm(pts[:, None] - xyz[None].astype(np.float64), axis=2) < 8.0).sum(1)


def _check_vina(sfp, xyz, ty, n):
    from adock_b200.grid import build_grid
    R, keep = _want(xyz, ty, sfp, n, TYPES)
    assert keep.mean() > 0.4
    R, pairs = R[:, :, keep], _pairs(xyz, n)[keep]
    args = (xyz, ty, sfp, np.zeros(3), SPACING, n, TYPES)
    T = build_grid(*args, per_term=True, device=DEV).cpu().numpy().reshape(R.shape[:2] + (-1,))[:, :, keep]
    assert np.isfinite(T).all() and (np.abs(T - R) <= _allowed(pairs, R)).all()
    w = np.array([sfp[k] for k in ("w_g1", "w_g2", "w_rep", "w_hyd", "w_hb")])
    G = build_grid(*args, device=DEV).cpu().numpy().reshape(len(TYPES), -1)[:, keep]
    want, total = np.einsum("m,mtp->tp", w, R), np.einsum("m,mtp->tp", np.abs(w), R)
    assert np.isfinite(G).all() and (np.abs(G - want) <= _allowed(pairs, total)).all()


def _check_fitted(sfp, xyz, ty, n):
    from adock_b200 import params
    from adock_b200.grid import build_grid_fit
    spec = params.FittedSpec("vina")
    spec.prm = {k: sfp[k] for k in spec.prm}
    pot = params.FittedPotential(spec, np.ones(len(params.TERM_NAMES), np.float32), TYPES)
    _, keep = _want(xyz, ty, sfp, n, TYPES)
    pts = np.stack(np.meshgrid(*[SPACING * np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3)
    r = np.linalg.norm(pts[:, None] - xyz[None].astype(np.float64), axis=2)
    ion = (1.0 / np.maximum(r, spec.ion_rmin) ** 2 - 1.0 / spec.cutoff ** 2) * (r < spec.cutoff)
    pairs = _pairs(xyz, n)
    G = build_grid_fit(xyz, ty, pot, np.zeros(3), SPACING, n, device=DEV).cpu().numpy().reshape(len(TYPES), -1)
    assert np.isfinite(G[:, keep]).all()
    for q in range(len(TYPES)):
        W = pot.W[ty, q].astype(np.float64)   # basis weights of each receptor atom
        assert np.abs(W).max() <= 6.0         # a weight is a sum of at most 6 ones
        B = np.concatenate([_terms(r, spec.rec_radius[ty].astype(np.float64) + float(pot.radius[q]), sfp), ion[None]])
        want, total = np.einsum("kpa,ak->p", B, W), np.einsum("kpa,ak->p", np.abs(B), np.abs(W))
        assert (np.abs(G[q] - want) <= _allowed(6 * 6 * pairs, total))[keep].all()


def _case(n):
    return _receptor(400, 6.0) if n[0] < 40 else _receptor(40, 24.0)


@pytest.mark.parametrize("n", [(13, 9, 10), (49, 50, 49)])   # one point per thread; two
@pytest.mark.parametrize("name", list(CHANGED))
def test_vina_steps_and_zero_widths(name, n):
    from adock_b200 import params
    _check_vina(dict(params.sf_params("vina"), **CHANGED[name]), *_case(n), n)


@pytest.mark.parametrize("n", [(13, 9, 10), (49, 50, 49)])
@pytest.mark.parametrize("name", list(CHANGED))
def test_fitted_steps_and_zero_widths(name, n):
    from adock_b200 import params
    _check_fitted(dict(params.sf_params("vina"), **CHANGED[name]), *_case(n), n)
