"""GPU: vector-decay calls that overlap on several streams, with decays that stay on the first set of kernels
and decays that need the second, give what they give one after the other."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(n, h, strong, seed):
    gen = torch.Generator().manual_seed(seed)
    q, k, v = (torch.randn(1, n, h, 128, generator=gen).mul(0.1).bfloat16().cuda() for _ in range(3))
    ldk = torch.nn.functional.logsigmoid(torch.randn(1, n, h, 128, generator=gen)).div(1 if strong else 16).cuda()
    return q, k, v, ldk


@pytest.mark.parametrize("graphs", [False, True])
def test_vector_decay_calls_overlap(graphs):
    """graphs: a stream's calls are replayed from a graph, back to back, so that those of the streams interleave
    densely."""
    from xopes_b200 import lightning_attn_func
    n, h, rounds = 512, 4, 40
    inputs = [_call(n, h, False, 0), _call(n, h, True, 1), _call(n, h, True, 2), _call(n, h, False, 3)]

    def call(x):
        with torch.no_grad():
            return lightning_attn_func(*x[:3], ldk=x[3], decay_type="vector")[0]

    ref = [call(x) for x in inputs]
    streams = [torch.cuda.Stream() for _ in inputs]
    torch.cuda.synchronize()
    out = [[] for _ in inputs]
    if graphs:
        held = []
        for x, o in zip(inputs, out):
            held.append(torch.cuda.CUDAGraph())
            with torch.cuda.graph(held[-1]):
                o.extend(call(x) for _ in range(rounds))
    wrong = [0] * len(inputs)
    for _ in range(5):
        if graphs:
            for os in out:  # outputs that a call leaves unwritten stay NaN
                for o in os:
                    o.fill_(float("nan"))
            torch.cuda.synchronize()
            for g, s in zip(held, streams):
                with torch.cuda.stream(s):
                    g.replay()
        else:
            out = [[] for _ in inputs]
            for s in streams:
                with torch.cuda.stream(s):
                    torch.full((rounds * n * h * 128 * 2,), float("nan"), dtype=torch.bfloat16, device="cuda")
            for _ in range(rounds):
                for x, s, o in zip(inputs, streams, out):
                    with torch.cuda.stream(s):
                        o.append(call(x))
        torch.cuda.synchronize()
        for i, (r, os) in enumerate(zip(ref, out)):
            wrong[i] += sum(not torch.equal(r, o) for o in os)
    assert wrong == [0] * len(inputs)
