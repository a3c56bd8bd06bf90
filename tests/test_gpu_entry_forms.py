"""Forms of the entry points that the framework's own calls do not reach: element-wise column sums, the SiLU gradient, targets
off a 16-byte boundary, and Stage A on a grid longer than its packed index arithmetic covers."""
import numpy as np
import pytest
import torch

from helpers import lig_types, make_problem

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


@pytest.mark.parametrize("rows,cols", [(0, 5), (1, 1), (7, 3), (257, 65), (1000, 130), (33, 64), (4097, 256)])
@pytest.mark.parametrize("offset", [0, 1])
def test_column_sums(rows, cols, offset):
    """FP32 sums of at most 4,097 BF16 values: rows x 2^-24 of the sum of the absolute values."""
    from adock_b200 import _lib
    g = torch.Generator(device=DEV).manual_seed(rows + cols)
    flat = torch.randn(offset + rows * cols + 1, device=DEV, generator=g).to(torch.bfloat16)
    A = flat[offset:offset + rows * cols].view(rows, cols)
    db = torch.full((cols,), 7.0, device=DEV)
    _lib.call("adock_bias_grad", A.data_ptr() or 16, rows, cols, _lib.ptr(db), _lib.stream_ptr())
    want, size = A.double().sum(0), A.double().abs().sum(0)
    assert ((db.double() - want).abs() <= (rows + 1) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("n", [1, 255, 100003])
def test_silu_gradient(n):
    """BF16 results (2^-9) of FP32 arithmetic (1e-6 of dH per factor)."""
    from adock_b200 import _lib
    g = torch.Generator(device=DEV).manual_seed(n)
    dH, A = torch.randn(n, device=DEV, generator=g), 4 * torch.randn(n, device=DEV, generator=g)
    out = torch.empty(n, dtype=torch.bfloat16, device=DEV)
    _lib.call("adock_silu_backward", _lib.ptr(dH), _lib.ptr(A), n, _lib.ptr(out), _lib.stream_ptr())
    s = torch.sigmoid(A.double())
    want = dH.double() * s * (1 + A.double() * (1 - s))
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 4e-6 * dH.double().abs()).all()


@pytest.mark.parametrize("N,k", [(1, 1), (5, 7), (33, 12), (64, 8)])
def test_sampled_targets_off_a_16_byte_boundary(N, k):
    from adock_b200 import _lib, params, synth
    from adock_b200.kernel import B200KernelProblem
    rec = synth.receptor_dict(np.zeros((1, 3), np.float32), np.zeros(1, np.int64), np.zeros(3), np.full(3, 3.0))
    ligs = [synth.ligand(24, 5, 0)]
    lt = lig_types(ligs)
    kp = B200KernelProblem(make_problem(rec, ligs, params.sf_params("vina"), np.zeros((len(lt), 9, 9, 9), np.float32), lt, DEV))
    g = torch.Generator(device=DEV).manual_seed(N)
    out, st = torch.randn(N, 64, device=DEV, generator=g), torch.randn(N, kp.SD, device=DEV, generator=g)
    cl, ci = torch.zeros(N, dtype=torch.int32, device=DEV), torch.arange(N, dtype=torch.int32, device=DEV)
    want = kp.prop_sample(cl, ci, out, st, k, 3, 1, 3)
    flat = torch.full((N * k * 32 + 8,), 5.0, device=DEV)
    _lib.call("adock_prop_sample", kp.c_lig, kp.c_work, _lib.ptr(cl), _lib.ptr(ci), N, _lib.ptr(out), _lib.ptr(st), kp.SD, k, 3, 3, 1,
              flat.data_ptr() + 4, _lib.stream_ptr())
    assert torch.equal(flat[1:1 + N * k * 32].view(N, k, 32), want)
    assert float(flat[0]) == 5.0 and (flat[1 + N * k * 32:] == 5.0).all()


@pytest.mark.parametrize("NT", [5, 40])
def test_stage_a_on_a_long_grid(NT):
    """2^22 + 1 points along z: element indices formed from integers. The map holds the index k modulo 1,024 (exact), so a wrong
    point shows; atoms stay clear of rounding edges."""
    from adock_b200 import params, synth
    from adock_b200.grid import GridSet
    from adock_b200.kernel import B200KernelProblem
    from adock_b200.ligand import LigandBatch
    from adock_b200.problem import PairPotential, Problem
    nz = (1 << 22) + 1
    ligs = [synth.ligand(3, 0, 1)]
    lt = np.unique(np.concatenate([[0], ligs[0].types]))
    slot = -np.ones((1, params.N_XS), np.int64)
    slot[0, lt] = np.arange(len(lt))
    ramp = (torch.arange(nz, device=DEV) % 1024).float()
    maps = torch.stack([ramp + 2048 * t for t in range(len(lt))]).view(len(lt), 1, 1, nz)
    f32 = lambda a: torch.tensor([a], dtype=torch.float32, device=DEV)
    far = 1e9
    gs = GridSet([maps], f32([0.0] * 3), f32([-far] * 3), f32([far] * 3), 1.0, 10.0, slot=torch.tensor(slot, device=DEV),
                 n_types=params.N_XS)
    prob = Problem(gs, LigandBatch(ligs, DEV), torch.zeros(1, dtype=torch.long, device=DEV),
                   PairPotential(params.sf_params("vina"), DEV))
    kp = B200KernelProblem(prob)
    conf = torch.zeros(1, 1, kp.AM, 3, device=DEV)
    conf[0, 0, :3, 2] = torch.tensor([0.0, 3.0, 7.0], device=DEV)
    quats = torch.tensor([[1.0, 0, 0, 0], [0.0, 1, 0, 0]], device=DEV)   # identity; z reversed
    g = torch.Generator().manual_seed(NT)
    z = torch.randint(10, nz - 10, (NT,), generator=g).float()           # whole numbers, exact in float32
    trans = torch.zeros(1, NT, 3, device=DEV)
    trans[0, :, 2] = z.to(DEV)
    be, bi = kp.stage_a(conf, quats, trans, torch.tensor([NT], device=DEV), 1e9)
    slots = torch.tensor([int(slot[0, t]) for t in ligs[0].types], dtype=torch.float32)
    for q, sign in enumerate((1, -1)):
        e = sum(((z + sign * dz) % 1024) + 2048 * s for dz, s in zip((0.0, 3.0, 7.0), slots))
        assert float(be[0, q]) == float(e.min()) and int(bi[0, q]) == int(torch.argmin(e))
