"""GPU: the memory pool and the side streams, which the library makes on first need, may be needed first under
stream capture (after one tensor-core call outside): the capture goes on and the results are the same."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HEAD = """
import torch
from xopes_b200 import _lib, lightning_attn_func
torch.manual_seed(0)
def rand(b, n, h):
    q, k, v = (torch.randn(b, n, h, 128, device="cuda").mul(128 ** -0.5).bfloat16() for _ in range(3))
    return q, k, v, torch.nn.functional.logsigmoid(torch.randn(b, n, h, device="cuda"))
q, k, v, ld = rand(1, 256, 4)  # needs neither
lightning_attn_func(q, k, v, ld=ld, decay_type="scalar")
torch.cuda.synchronize()
"""

CALLS = {
    # more pairs than SMs: the even split of the chunks, with scratch from the pool
    "scalar": """
q, k, v, ld = rand(10, 256, 16)
call = lambda: lightning_attn_func(q, k, v, ld=ld, decay_type="scalar")
""",
    # few pairs: dq on a side stream
    "backward": """
q, k, v, ld = rand(1, 256, 4)
do = torch.randn_like(v)
lib = _lib.load()
def call():
    dq, dk, dv, dld = (torch.empty_like(t) for t in (q, k, v, ld))
    ws = torch.empty(lib.la_lasd_bwd_workspace_bytes(1, 256, 4, 128, 128, 0, 1), dtype=torch.uint8, device="cuda")
    rc = lib.la_lasd_bwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), ld.data_ptr(), *ld.stride(), None, do.data_ptr(), None,
                         None, dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dld.data_ptr(), None, ws.data_ptr(),
                         ws.numel(), 1, 256, 4, 128, 128, 0, 1, 0, torch.cuda.current_stream().cuda_stream)
    assert rc == 0, (rc, lib.la_debug_last_cuda_error())
    return dq, dk, dv, dld
""",
}

TAIL = """
with torch.no_grad():
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = call()
    graph.replay()
    ref = call()
    torch.cuda.synchronize()
for o, r in zip(out, ref):
    assert torch.isfinite(o.float()).all() and torch.equal(o, r), float((o.float() - r.float()).abs().max())
"""


@pytest.mark.parametrize("which", sorted(CALLS))
def test_first_need_under_capture(which):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", HEAD + CALLS[which] + TAIL], cwd=root, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
