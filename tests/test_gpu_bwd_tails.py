"""Gradients where the batched gathers of the one-launch backward end: lists of every length from none to past two batches, documents of
whole and partial groups of four winners, several batches of documents per query."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,lq,nd,ld,d,dtype", [
    (128, 32, 100, 40, 128, torch.bfloat16),   # 512 threads, whole groups of four rounds, long lists
    (100, 32, 97, 300, 128, torch.float16),    # ... and partial ones, four batches of documents
    (40, 24, 33, 64, 96, torch.bfloat16),      # a batch of documents and one more
    (16, 20, 65, 17, 64, torch.float32),       # four features per load
    (20, 32, 31, 50, 256, torch.bfloat16),     # two loads per row: batches of four
])
@pytest.mark.parametrize("skew", [0, 1])
def test_lists_of_every_length(nq, lq, nd, ld, d, dtype, skew):
    """skew: most winners on few tokens, so that lists run from 0 to dozens of entries.  Bound: fp32 sums of n terms of a row's gradient differ
    from 64 bits by n * 2^-24 of their absolute sum, far below the rounding of the gradient itself: 2^-8 (bf16), 2^-11 (fp16)."""
    import late_interaction_kernels_b200 as lik

    g = torch.Generator().manual_seed(nq + skew)
    Q = torch.nn.functional.normalize(torch.randn((nq, lq, d), generator=g), dim=-1)
    D = torch.nn.functional.normalize(torch.randn((nd, ld, d), generator=g), dim=-1)
    if skew:
        D[:, ::5] *= 2.0
    Q, D = Q.cuda().to(dtype).requires_grad_(), D.cuda().to(dtype).requires_grad_()
    dm = (torch.arange(ld) < torch.randint(1, ld + 1, (nd, 1), generator=g)).cuda()
    w = torch.randn((nq, nd), generator=g).cuda()
    s = lik.maxsim(Q, D, d_mask=dm)
    gq, gd = torch.autograd.grad(s, (Q, D), w)
    x = torch.einsum("isd,jtd->ijst", Q.detach().double(), D.detach().double()).masked_fill(~dm[None, :, None, :], -torch.inf)
    win = x.argmax(-1)  # [nq, nd, lq]
    wq = torch.zeros((nq, lq, d), dtype=torch.float64, device="cuda")
    wd = torch.zeros((nd, ld, d), dtype=torch.float64, device="cuda")
    for j in range(nd):
        rows = D.detach().double()[j][win[:, j]]  # [nq, lq, d]
        wq += w[:, j, None, None].double() * rows
        wd[j].index_add_(0, win[:, j].reshape(-1), (w[:, j, None, None].double() * Q.detach().double()).reshape(-1, d))
    tol = {torch.bfloat16: 2.0**-8, torch.float16: 2.0**-10, torch.float32: 1e-5}[dtype]
    assert (gq.double() - wq).norm() < tol * wq.norm() and (gd.double() - wd).norm() < tol * wd.norm()
    again = torch.autograd.grad(lik.maxsim(Q, D, d_mask=dm), (Q, D), w)
    assert torch.equal(again[0], gq) and torch.equal(again[1], gd)
