"""GPU: the reverse scan that finishes the scalar log-decay gradient, at the edges of its tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_state", [False, True])
@pytest.mark.parametrize("d", [16, 8])  # two slots of row dots per token and one (as the tensor-core path writes them)
@pytest.mark.parametrize("lens", [[1], [7, 1, 300], [2047], [2048], [2049, 3], [5000, 0, 130]])
def test_scalar_decay_gradient_scan(lens, d, with_state):
    """dld is the reverse cumulative sum, per document, of the row dots q.dq - k.dk of the same call's
    gradients, starting from <S, dS> of the final state and its gradient.  The sum's terms cancel, so the bound
    is 2^-20 of the largest partial sum's scale: sqrt(n) terms of the row dots' fp32 rounding, and |S| |dS|."""
    from xopes_b200 import lasd_parallel_cuda
    n, h = sum(lens), 3
    gen = torch.Generator().manual_seed(n)
    q, k, v = (torch.randn(1, n, h, d, generator=gen).cuda().requires_grad_() for _ in range(3))
    ld = (-0.05 * torch.rand(1, n, h, generator=gen)).cuda().requires_grad_()
    cu = torch.tensor([0] + lens).cumsum(0).cuda()
    do = torch.randn(1, n, h, d, generator=gen).cuda()
    ds = torch.randn(len(lens), h, d, d, generator=gen).cuda()
    o, sf = lasd_parallel_cuda(q, k, v, ld=ld, cu_seqlens=cu)
    outs, gouts = ((o, sf), (do, ds)) if with_state else ((o,), (do,))
    dq, dk, _, dld = torch.autograd.grad(outs, [q, k, v, ld], gouts)
    dots = ((q.detach().double() * dq.double()).sum(-1) - (k.detach().double() * dk.double()).sum(-1))[0].cpu()
    carry = (sf.detach().double() * ds.double()).sum((-2, -1)).cpu() if with_state else torch.zeros(len(lens), h).double()
    ref, at = torch.zeros_like(dots), 0
    for i, m in enumerate(lens):
        ref[at:at + m] = dots[at:at + m].flip(0).cumsum(0).flip(0) + carry[i]
        at += m
    scale = float((q.detach().double() * dq.double()).sum(-1).abs().max()) * max(lens) ** 0.5
    if with_state:
        scale += float((sf.detach().double().norm(dim=(-2, -1)) * ds.double().norm(dim=(-2, -1))).max())
    assert float((ref - dld[0].double().cpu()).abs().max()) <= 2.0 ** -20 * scale
