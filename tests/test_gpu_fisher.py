"""spi_fisher over the sizes where its staging has edges: one row block of 256 and more (W = 7 is 259 rows),
row counts off the 16-row step of the tensor-core product, one parameter and all thirteen."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tensor_cores", [False, True])
@pytest.mark.parametrize("N,W,K", [(1, 1, 1), (3, 6, 13), (2, 7, 9), (5, 14, 13), (1, 64, 8)])
def test_fisher_equals_fp64(built, N, W, K, tensor_cores):
    """F within 1e-5 of its largest entry of the FP64 sum (FP32: at most 2,368 terms of 2^-24 each, signs mixed)
    or, with BF16 operands (relative rounding 2^-9 each, two factors), of the FP64 sum over the rounded
    operands; log det and trace are the FP64 values of the F returned."""
    from spi_gb300.sensitivity import fisher
    gen = torch.Generator(device="cuda").manual_seed(N * 100 + W + K)
    J = torch.randn((N, W, 37, K), device="cuda", generator=gen)
    q = torch.rand(37, device="cuda", generator=gen) + 0.1
    F, logdet, trace = fisher(J, q, eps=1e-6, tensor_cores=tensor_cores)
    A = (torch.sqrt(q)[:, None] * J)
    A = A.to(torch.bfloat16).double() if tensor_cores else A.double()
    ref = torch.einsum("nwik,nwil->nkl", A, A)
    # a product rounded one way here and the other there moves by one BF16 step, 2^-8 of one of 37 W terms
    tol = 1e-5 if not tensor_cores else 2.0 ** -8
    assert (F.double() - ref).abs().max() <= tol * ref.abs().max()
    own = F.double()
    own = torch.tril(own) + torch.tril(own, -1).transpose(1, 2)
    eye = 1e-6 * torch.eye(K, device="cuda", dtype=torch.float64)
    assert torch.allclose(logdet, torch.logdet(own + eye), rtol=1e-9, atol=1e-9)
    assert torch.allclose(trace, torch.diagonal(own, dim1=1, dim2=2).sum(-1), rtol=1e-12)
