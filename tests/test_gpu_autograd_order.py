"""The autograd entry point on weights that are still being computed: the
graphs and the batch run on streams of their own and must wait for them."""
import numpy as np
import pytest

import adds_b200 as A
from adds_b200 import graphs as G
from oracle import oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("side", [40, 300])
def test_forward_waits_for_its_weights(side):
    from adds_b200.autograd import batched_sssp
    g = G.grid(side, side, 0.0, 8, wtype=G.F32, seed=side)
    dg = A.Graph.from_csr(g)
    b = A.Batch([dg, dg], [0, side * side // 2])
    x = torch.randn(4096, 4096, device="cuda")
    base = torch.from_numpy(g.w.view(np.float32).copy()).cuda()
    for turn in range(3):
        scale = float(turn + 1)
        y = x
        for _ in range(20):  # some milliseconds of work before the weights are there
            y = (y @ x) * 1e-3
        w = base * scale + 0.0 * torch.nan_to_num(y.sum(), 0.0, 0.0, 0.0)
        flat = batched_sssp(b, [dg], [w])
        want = (g.w.view(np.float32) * np.float32(scale)).astype(np.float32)
        ref = O.dijkstra(G.CSR(g.n, g.row, g.dst, want.view(np.uint32), G.F32), 0)[0]
        assert np.array_equal(flat[: g.n].cpu().numpy().view(np.uint32), ref)
    b.close()
    dg.close()


def test_forward_takes_host_weights():
    """Weights that lie in host memory: the distances come back there too."""
    from adds_b200.autograd import batched_sssp
    g = G.grid(40, 40, 0.0, 8, wtype=G.F32, seed=3)
    dg = A.Graph.from_csr(g)
    b = A.Batch([dg], [5])
    flat = batched_sssp(b, [dg], [torch.from_numpy(g.w.view(np.float32) * np.float32(2))])
    n = G.CSR(g.n, g.row, g.dst, (g.w.view(np.float32) * np.float32(2)).view(np.uint32), G.F32)
    assert flat.device.type == "cpu"
    assert np.array_equal(flat[: g.n].numpy().view(np.uint32), O.dijkstra(n, 5)[0])
    b.close()
    dg.close()
