"""Stored-Ke products at the sizes and forms their kernels treat differently: element
counts around a thread block's share, element matrices off a 16-byte boundary, and
prescribed DOFs, against the product of the same matrices in plain FP64 on the CPU."""
import numpy as np
import pytest
import torch

from helpers import jittered_box, rel_err, tet10_box

pytestmark = pytest.mark.gpu


def _block(kind, ne):
    import exfem_b200 as xf
    X, c = jittered_box(9, 2, 2, 9, 2, 2, 0.15, 2) if kind == "hex" else tet10_box(4, 1, 2, 4, 1, 2, 0.1, 2)
    m = xf.Model(X)
    return m, m.add_block(c[:ne], xf.HEX8 if kind == "hex" else xf.TET10, xf.LinearElastic(210000.0, 0.3))


def _reference(b, K, v, fixed):
    """free K (free v) + fixed v, v (ndof, k), in FP64 on the CPU."""
    dofs = (torch.as_tensor(b.conn).long()[:, :, None] * 3 + torch.arange(3)).reshape(b.ne, -1)
    fr = torch.as_tensor(~fixed).double()[:, None]
    ye = torch.einsum("eij,ejk->eik", K, (fr * v)[dofs])
    y = torch.zeros_like(v).index_add_(0, dofs.reshape(-1), ye.reshape(-1, v.shape[1]))
    return torch.where(fr > 0, y, v)


@pytest.mark.parametrize("kind", ["hex", "tet"])
@pytest.mark.parametrize("ne", [1, 2, 7, 8, 9, 31, 33])
@pytest.mark.parametrize("offset", [0, 1])
def test_single_product(cuda, kind, ne, offset):
    """Bar 1e-13 of the largest entry: sums of up to 30 products per row and 8 to 24 rows
    per node in FP64."""
    m, b = _block(kind, ne)
    g = torch.Generator().manual_seed(ne)
    nd = b.etype.nd
    K = torch.randn(ne, nd, nd, dtype=torch.float64, generator=g)
    v = torch.randn(m.ndof, dtype=torch.float64, generator=g)
    fixed = np.zeros(m.ndof, bool)
    fixed[::5] = True
    Kd = torch.zeros(K.numel() + offset, dtype=torch.float64, device="cuda")[offset:].view(ne, nd, nd)
    Kd.copy_(K)
    assert Kd.data_ptr() % 16 == 8 * offset
    for fx, bc in ((fixed, True), (np.zeros(m.ndof, bool), False)):
        b.set_fixed(fixed)
        y = b.ebe_matvec(Kd, v.cuda(), apply_bc=bc)
        assert rel_err(y, _reference(b, K, v[:, None], fx)[:, 0]) < 1e-13


@pytest.mark.parametrize("kind", ["hex", "tet"])
@pytest.mark.parametrize("nrhs", [1, 2, 3, 4, 5, 7, 8, 11, 13, 16])
@pytest.mark.parametrize("ne", [1, 2, 15, 16, 17, 33])
def test_products_of_several_right_hand_sides(cuda, kind, nrhs, ne):
    """FP64 bar as above; FP32 accumulation of up to 30 products per row and 24 rows per
    node: 24 roundings of 6e-8 on sums of unit-variance products, bar 3e-6."""
    m, b = _block(kind, ne)
    g = torch.Generator().manual_seed(100 * nrhs + ne)
    nd = b.etype.nd
    K = torch.randn(ne, nd, nd, dtype=torch.float64, generator=g)
    v = torch.randn(m.ndof, nrhs, dtype=torch.float64, generator=g)
    fixed = np.zeros(m.ndof, bool)
    fixed[1::5] = True
    b.set_fixed(fixed)
    assert rel_err(b.ebe_matvec_multi(K.cuda(), v.cuda()), _reference(b, K, v, fixed)) < 1e-13
    v32 = v.float()
    for dt in (torch.float32, torch.bfloat16):
        Kt = K.to(dt)
        y = b.ebe_matvec_multi(Kt.cuda(), v32.cuda())
        assert rel_err(y, _reference(b, Kt.double(), v32.double(), fixed)) < 3e-6
    none = np.zeros(m.ndof, bool)
    assert rel_err(b.ebe_matvec_multi(K.cuda(), v.cuda(), apply_bc=False), _reference(b, K, v, none)) < 1e-13
