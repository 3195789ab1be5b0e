"""Elastic forces on both sides of the mesh size at which their form changes (12,000 C3D8)
against the stored element matrices' product, with stiffness scales, per-element moduli,
element forces and the state copy; elastic stresses against the oracle.  Bar 1e-12 relative
(FP64 sums of a few hundred terms)."""
import numpy as np
import pytest
import torch

from helpers import jittered_box, rel_err, smooth_field, tet10_box
from oracle import fem as ofem

pytestmark = pytest.mark.gpu

E, NU = 210000.0, 0.3


@pytest.mark.parametrize("n", [(30, 20, 20), (31, 20, 20), (26, 21, 23)])
@pytest.mark.parametrize("field", ["none", "scale", "lame"])
def test_forces_on_both_sides_of_the_line(cuda, n, field):
    import exfem_b200 as xf
    from exfem_b200 import _lib
    from exfem_b200._lib import check, lib, ptr, stream_ptr
    X, c = jittered_box(*[float(k) for k in n], *n, 0.1, 1)
    X = X + np.array([300.0, -200.0, 100.0])
    m = xf.Model(X)
    b = m.add_block(c, xf.HEX8, xf.LinearElastic(E, NU))
    rng = np.random.default_rng(3)
    if field == "scale":
        b.set_scale(np.exp(rng.uniform(-1, 1, b.ne)))
    if field == "lame":
        Es, nus = rng.uniform(1e4, 3e5, b.ne), rng.uniform(0.05, 0.45, b.ne)
        b.set_lame(Es * nus / ((1 + nus) * (1 - 2 * nus)), Es / (2 * (1 + nus)))
    u = torch.randn(m.ndof, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    st = torch.rand(b.ne * 8, dtype=torch.float64, device="cuda")
    new, fe, f = torch.empty_like(st), torch.empty(b.ne, 24, dtype=torch.float64, device="cuda"), torch.empty_like(u)
    check(lib.exfem_internal_force(b.handle, ptr(u), ptr(st), ptr(new), ptr(fe), ptr(f), _lib.ASSEMBLE_GATHER,
                                   stream_ptr()))
    K = b.stiffness(torch.zeros_like(u), b.init_state())
    dofs = (torch.as_tensor(b.conn).long().cuda()[:, :, None] * 3 + torch.arange(3, device="cuda")).reshape(b.ne, 24)
    assert rel_err(fe, torch.einsum("eij,ej->ei", K, u[dofs])) < 1e-12
    assert rel_err(f, b.ebe_matvec(K, u, apply_bc=False)) < 1e-12
    assert torch.equal(new, st)


@pytest.mark.parametrize("kind,n", [("hex", (1, 1, 1)), ("hex", (8, 4, 4)), ("hex", (9, 5, 3)),
                                    ("tet", (1, 1, 1)), ("tet", (4, 3, 3))])
def test_stresses_match_the_oracle(cuda, kind, n):
    import exfem_b200 as xf
    X, c = (jittered_box if kind == "hex" else tet10_box)(*[float(k) for k in n], *n, 0.1, 1)
    om, pm = ofem.Model(X), xf.Model(X)
    om.add_block(c, ofem.HEX8 if kind == "hex" else ofem.TET10, ofem.LinearElastic(E, NU))
    pm.add_block(c, xf.HEX8 if kind == "hex" else xf.TET10, xf.LinearElastic(E, NU))
    u = torch.as_tensor(smooth_field(X, 2e-3, seed=3))
    ro, rp = om.stresses(u, om.init_state())[0], pm.stresses(u.cuda(), pm.init_state())[0]
    assert rel_err(rp["S"], ro["S"]) < 1e-12
    assert rel_err(rp["MISES"], ro["MISES"]) < 1e-12
    assert not rp["PEEQ"].any()
