"""The first no-allocation call of a process, which writes the list areas that
the kernels read, on streams that do not wait for the default one."""
import os
import re
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FIRST = """
import numpy as np, torch
from adds_b200 import _lib as L, graphs as G
from oracle import oracle as O
g = G.rmat(13, 16, seed=2)
row = torch.from_numpy(g.row.astype(np.uint32).view(np.int32)).cuda()
edges = torch.from_numpy(np.stack([g.dst, g.w], 1).astype(np.uint32).view(np.int32).copy()).cuda()
out = torch.empty(g.n, dtype=torch.int32, device="cuda")
busy = torch.zeros(1 << 26, device="cuda")
torch.cuda.synchronize()
for src in (3, 4, 5):
    st = torch.cuda.Stream()  # non-blocking
    for _ in range(20):
        busy += 1.0  # the default stream has work of its own
    rc = L.lib().adds_sssp_noalloc(g.n, g.m, row.data_ptr(), edges.data_ptr(), g.wtype, src,
                                   out.data_ptr(), st.cuda_stream)
    L.check(rc, "adds_sssp_noalloc")
    with torch.cuda.stream(st):
        got = out.cpu().numpy().view(np.uint32)
    assert np.array_equal(got, O.dijkstra(g, src)[0]), src
"""


def test_every_step_is_on_the_callers_stream():
    """Nothing of the call goes to the default stream: no copy, no fill and no
    launch that names no stream."""
    text = open(os.path.join(ROOT, "adds_b200", "csrc", "noalloc.cu")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    assert not re.findall(r"\bcuda(?:Memcpy|Memset)(?:ToSymbol|FromSymbol)?\s*\(", text)
    launches = re.findall(r"<<<(.*?)>>>", text, flags=re.S)
    assert launches and all(x.replace(" ", "").endswith(",st") for x in launches)


@pytest.mark.gpu
def test_first_call_on_a_stream_of_its_own():
    r = subprocess.run([sys.executable, "-c", FIRST], cwd=ROOT, capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
