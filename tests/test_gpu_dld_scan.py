"""GPU: the reverse scan that finishes the scalar log-decay gradient, at the edges of its tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[1], [7, 1, 300], [2047], [2048], [2049, 3], [5000, 0, 130]])
def test_scalar_decay_gradient_scan(lens):
    """dld is the reverse cumulative sum, per document, of the row dots q.dq - k.dk of the same call's
    gradients.  The sum's terms cancel, so the bound is 2^-20 of the largest partial sum's scale, sqrt(n)
    terms of the row dots' fp32 rounding."""
    from xopes_b200 import lasd_parallel_cuda
    n, h, d = sum(lens), 3, 16
    gen = torch.Generator().manual_seed(n)
    q, k, v = (torch.randn(1, n, h, d, generator=gen).cuda().requires_grad_() for _ in range(3))
    ld = (-0.05 * torch.rand(1, n, h, generator=gen)).cuda().requires_grad_()
    cu = torch.tensor([0] + lens).cumsum(0).cuda()
    do = torch.randn(1, n, h, d, generator=gen).cuda()
    o, _ = lasd_parallel_cuda(q, k, v, ld=ld, cu_seqlens=cu)
    dq, dk, _, dld = torch.autograd.grad(o, [q, k, v, ld], do)
    dots = ((q.detach().double() * dq.double()).sum(-1) - (k.detach().double() * dk.double()).sum(-1))[0].cpu()
    ref, at = torch.zeros_like(dots), 0
    for m in lens:
        ref[at:at + m] = dots[at:at + m].flip(0).cumsum(0).flip(0)
        at += m
    scale = float((q.detach().double() * dq.double()).sum(-1).abs().max()) * max(lens) ** 0.5
    assert float((ref - dld[0].double().cpu()).abs().max()) <= 2.0 ** -20 * scale
