"""Rigid Stage-A scores where a CTA's warps share a rotation's lattice: one, two and four rotations per CTA with a last CTA
that has fewer, lattices from one point above a warp's stride on, against the oracle at the bars of test_gpu_stage_a.py."""
import pytest

import test_gpu_stage_a as lattices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Q", [7, 501, 999])   # 1, 2 and 4 rotations per CTA on a chip of 148 SMs
@pytest.mark.parametrize("NT", [32, 33, 65, 129])
def test_warps_share_a_rotation(NT, Q):
    lattices.test_stage_a_over_lattice_sizes(NT, Q, "f32")
