"""The ionic term of the fitted maps alone, against float64, where its rounding can be bounded: coordinates are multiples of
1/8, so that r^2 is exact in float32, and one receptor atom, so that nothing is summed."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("ion_rmin", [2.0, 0.0])
@pytest.mark.parametrize("n", [(20, 19, 21), (60, 61, 62)])   # one point per thread; two
def test_ionic_term(n, ion_rmin):
    """1 / max(r, minimum)^2 rounds once, to 1 ulp, and the difference to its value at the cutoff (a power of two) once, to
    half an ulp: 1.5 ulp of the first."""
    from adock_b200 import params
    from adock_b200.grid import build_grid_fit
    spec = params.FittedSpec("vina")
    spec.ion_rmin = ion_rmin
    pot = params.FittedPotential(spec, np.zeros(len(params.TERM_NAMES), np.float32), [0])
    pot.W = np.zeros_like(pot.W)
    pot.W[..., 5] = 1.0
    at = np.array([[4.125, 4.625, 5.375]], np.float32)
    G = build_grid_fit(at, np.zeros(1, np.int64), pot, np.zeros(3), 0.25, n, device=DEV).cpu().numpy().reshape(-1)
    pts = np.stack(np.meshgrid(*[0.25 * np.arange(k) for k in n], indexing="ij"), -1).reshape(-1, 3)
    r2 = ((pts - at[0].astype(np.float64)) ** 2).sum(1)
    near = 1.0 / np.maximum(r2, ion_rmin ** 2)
    want = np.where(r2 < spec.cutoff ** 2, near - 1.0 / spec.cutoff ** 2, 0.0)
    assert (r2 > 0).all() and (np.abs(G - want) <= 1.5 * 2.0 ** -23 * near).all()
