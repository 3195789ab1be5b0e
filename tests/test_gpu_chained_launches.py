"""Products and V-cycles begin before the kernel ahead of them has finished and wait for
its writes: back-to-back calls, with torch kernels writing their inputs in between, in
plain streams and inside a captured graph, give the bits of calls synchronised one by
one."""
import numpy as np
import pytest
import torch

from helpers import jittered_box, tet10_box

pytestmark = pytest.mark.gpu


def _setup(kind, n):
    import exfem_b200 as xf
    X, c = (jittered_box if kind == "hex" else tet10_box)(*[float(k) for k in n], *n, 0.1, 1)
    m = xf.Model(X)
    b = m.add_block(c, xf.HEX8 if kind == "hex" else xf.TET10, xf.LinearElastic(1.0, 0.3))
    fixed = np.zeros((len(X), 3), bool)
    fixed[X[:, 0] < 1e-9] = True
    b.set_fixed(fixed.reshape(-1))
    zero = torch.zeros(m.ndof, dtype=torch.float64, device="cuda")
    return m, b, xf.DeviceAMG(b, b.stiffness(zero, b.init_state()), max_coarse=60, keep_level0=True)


def _chain(b, amg, v, steps, sync):
    out = []
    d = torch.full_like(v, 0.5)
    for k in range(steps):
        v = v * 0.5 + 1.0
        if sync:
            torch.cuda.synchronize()
        y = b.tangent_matvec(v)
        if sync:
            torch.cuda.synchronize()
        v = amg.vcycle(y, level0=b, dinv0=d) * 0.25
        if sync:
            torch.cuda.synchronize()
        out.append(y)
        out.append(v)
    return out


@pytest.mark.parametrize("kind,n", [("hex", (5, 4, 3)), ("hex", (40, 12, 12)), ("tet", (4, 3, 3)), ("tet", (12, 10, 9))])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
def test_back_to_back_calls_give_the_same_bits(cuda, kind, n, dtype):
    m, b, amg = _setup(kind, n)
    v = torch.randn(m.ndof, dtype=dtype, device="cuda", generator=torch.Generator("cuda").manual_seed(2))
    want = _chain(b, amg, v, 12, True)
    got = _chain(b, amg, v, 12, False)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        on_side = _chain(b, amg, v, 12, False)
    torch.cuda.synchronize()
    for g in (got, on_side):
        assert all(torch.equal(a, w) for a, w in zip(g, want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        in_graph = _chain(b, amg, v, 4, False)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, w) for a, w in zip(in_graph, want))
