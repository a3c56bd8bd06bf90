"""The tcgen05 GEMM over operand layouts and sizes (vector and element staging, tile edges, K split over a cluster) and the
network's forward and backward pass over odd batches, against float64.

GEMM bar: the tensor core adds at most K / 16 + 8 partial sums, each rounded at 2^-23 of a partial that is at most
sum |a b|; 3.2e-5 of that sum covers K = 4,096."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _operand(rows, cols, layout, g):
    """bf16 [rows, cols] with its strides: row-major, column-major, or row-major with an odd row stride."""
    if layout == "row":
        t = torch.randn(rows, cols, device=DEV, generator=g).to(torch.bfloat16)
    elif layout == "col":
        t = torch.randn(cols, rows, device=DEV, generator=g).to(torch.bfloat16).t()
    else:
        t = torch.randn(rows, cols + 3, device=DEV, generator=g).to(torch.bfloat16)[:, 1:1 + cols]
    return t


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (128, 64, 64), (129, 65, 72), (320, 256, 4096), (256, 64, 1000),
                                   (40, 24, 264), (4096, 256, 320), (19000, 200, 64), (128, 128, 0)])
@pytest.mark.parametrize("la,lb", [("row", "row"), ("row", "col"), ("col", "row"), ("col", "col"), ("odd", "odd")])
def test_gemm_layouts(M, N, K, la, lb):
    from adock_b200 import _lib
    g = torch.Generator(device=DEV).manual_seed(M * 7 + N * 3 + K)
    A, B = _operand(M, K, la, g), _operand(K, N, lb, g)
    bias = torch.randn(N, device=DEV, generator=g)
    C0 = torch.randn(M, N, device=DEV, generator=g)
    C, Cb = C0.clone(), torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    _lib.call("adock_gemm_bf16", M, N, K, A.data_ptr() or 16, A.stride(0), A.stride(1), B.data_ptr() or 16, B.stride(0),
              B.stride(1), _lib.ptr(C), N, 0.5, _lib.ptr(bias), 0, None, _lib.ptr(Cb), N, _lib.stream_ptr())
    want = A.double() @ B.double() + 0.5 * C0.double() + bias.double()
    scale = A.double().abs() @ B.double().abs() + 1.0
    assert float(((C.double() - want).abs() / scale).max()) < 3.2e-5
    assert float(((Cb.double() - want).abs() / (scale + want.abs())).max()) < 2 ** -8
    assert _lib.load().adock_gemm_status() == 0


@pytest.mark.parametrize("B,n_comp", [(0, 1), (1, 1), (7, 3), (130, 1), (1000, 3), (4096, 3)])
def test_loss_and_gradients_over_batch_sizes(B, n_comp):
    """Bars as in test_gpu_proposal.py: loss 1e-2, every gradient 2e-2 of its norm (BF16 activations)."""
    from oracle import mlp as O
    from adock_b200.proposal import IN, ProposalNet
    net = ProposalNet(DEV, seed=5, n_comp=n_comp)
    g = torch.Generator(device=DEV).manual_seed(B + 1)
    X = torch.randn(B, IN, device=DEV, generator=g).to(torch.bfloat16)
    Y = torch.randn(B, 32, device=DEV, generator=g) * 0.5
    Y[:, 26] = torch.randint(0, 21, (B,), device=DEV, generator=g).float()
    Y[:, 27:] = 0
    loss, grads = net.loss_grad(X, Y)
    if B == 0:
        assert all(float(v.abs().sum()) == 0.0 for v in grads)
        return
    lo, go = O.loss_and_grads([w.double().cpu().numpy() for w in net.Wb], [b.double().cpu().numpy() for b in net.b],
                              X.double().cpu().numpy(), Y.double().cpu().numpy(), n_comp=n_comp)
    assert abs(float(loss) - lo) <= 1e-2 * max(1.0, abs(lo))
    for got, want in zip(grads, go):
        assert np.linalg.norm(got.double().cpu().numpy() - want) <= 2e-2 * np.linalg.norm(want) + 1e-6
    out, saved = net.forward(X, save=True)
    assert torch.equal(out, net.forward(X)) and saved[1].shape == saved[3].shape == (B, 256)
