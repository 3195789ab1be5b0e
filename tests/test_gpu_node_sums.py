"""Node sums of the multi-right-hand-side products in every form their count and alignment
select (whole 16-byte groups, pairs of them, a node's three rows at a time, single values):
the bits of the single-column product of the same matrices, whose sums have the same order."""
import numpy as np
import pytest
import torch

from helpers import jittered_box, tet10_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["hex", "tet"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 6, 8, 9, 10, 12, 14, 15, 16])
def test_columns_do_not_depend_on_their_number(cuda, kind, dtype, nrhs):
    import exfem_b200 as xf
    X, c = jittered_box(5, 4, 3, 5, 4, 3, 0.1, 2) if kind == "hex" else tet10_box(3, 2, 2, 3, 2, 2, 0.1, 2)
    m = xf.Model(X)
    b = m.add_block(c, xf.HEX8 if kind == "hex" else xf.TET10, xf.LinearElastic(1.0, 0.3))
    fixed = np.zeros(m.ndof, bool)
    fixed[1::5] = True
    b.set_fixed(fixed)
    g = torch.Generator("cuda").manual_seed(nrhs)
    K = torch.randn(b.ne, b.etype.nd, b.etype.nd, dtype=dtype, device="cuda", generator=g)
    V = torch.randn(m.ndof, nrhs, dtype=dtype, device="cuda", generator=g)
    off = torch.zeros(V.numel() + 1, dtype=dtype, device="cuda")[1:].view(m.ndof, nrhs)
    off.copy_(V)
    assert V.data_ptr() % 16 == 0 and off.data_ptr() % 16 != 0
    Y = b.ebe_matvec_multi(K, V)
    assert torch.equal(b.ebe_matvec_multi(K, off), Y)
    for j in range(nrhs):
        assert torch.equal(b.ebe_matvec_multi(K, V[:, j:j + 1].contiguous())[:, 0], Y[:, j])
