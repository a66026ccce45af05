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


@pytest.mark.parametrize("tensor_cores", [False, True])
@pytest.mark.parametrize("N,W,K", [(9001, 1, 13), (9001, 1, 1), (6002, 2, 5), (11000, 4, 3), (11003, 5, 8), (20001, 1, 8)])
def test_a_sample_does_not_depend_on_the_others(built, N, W, K, tensor_cores):
    """Past the numbers where the scores, and for few windows the sums, go to kernels of their own: every sample
    is, to the bit, what it is in a small call (the same operations in the same order), a zero one and one with a NaN
    among them."""
    from spi_gb300.sensitivity import fisher
    gen = torch.Generator(device="cuda").manual_seed(N + W + K)
    J = torch.randn((N, W, 37, K), device="cuda", generator=gen)
    J[7] = 0.0
    J[11, 0, 5, 0] = float("nan")
    q = torch.rand(37, device="cuda", generator=gen) + 0.1
    for weight, eps in ((q, 0.0), (None, 1e-6)):
        whole = fisher(J, weight, eps=eps, tensor_cores=tensor_cores)
        assert torch.isfinite(whole[1][20:]).all()
        for rows in (slice(0, 31), slice(N // 2, N // 2 + 2), slice(N - 3, N)):
            part = fisher(J[rows], weight, eps=eps, tensor_cores=tensor_cores)
            for a, b in zip(whole, part):
                assert torch.equal(torch.nan_to_num(a[rows], nan=-7.0), torch.nan_to_num(b, nan=-7.0))
        assert whole[1][11] == float("-inf") and (eps > 0 or whole[1][7] == float("-inf"))
