"""FP64 tangent products on both sides of the line between their two forms (one lane per
Gauss point up to 120,000 C3D8 or 350,000 C3D10, tiles above) and over the inputs both
take: prescribed DOFs, per-element scale and moduli, elastic and J2 tangents."""
import numpy as np
import pytest
import torch

from helpers import jittered_box, rel_err, smooth_field, tet10_box
from oracle import fem as ofem

pytestmark = pytest.mark.gpu

E, NU = 210000.0, 0.3
TABLE = [[250.0, 0.0], [1250.0, 1.0]]


@pytest.mark.parametrize("kind", ["hex", "tet"])
@pytest.mark.parametrize("mat", ["el", "j2"])
@pytest.mark.parametrize("ne", [1, 4, 7, 9, 33])
def test_small_products_match_the_oracle(cuda, kind, mat, ne):
    """Bar 1e-12 relative (FP64 rounding)."""
    import exfem_b200 as xf
    X, c = jittered_box(9, 2, 2, 9, 2, 2, 0.15, 2) if kind == "hex" else tet10_box(4, 1, 2, 4, 1, 2, 0.1, 2)
    c = c[:ne]
    args = (E, NU) if mat == "el" else (E, NU, TABLE)
    om, pm = ofem.Model(X), xf.Model(X)
    om.add_block(c, ofem.HEX8 if kind == "hex" else ofem.TET10,
                 (ofem.LinearElastic if mat == "el" else ofem.J2Plasticity)(*args))
    b = pm.add_block(c, xf.HEX8 if kind == "hex" else xf.TET10,
                     (xf.LinearElastic if mat == "el" else xf.J2Plasticity)(*args))
    rng = np.random.default_rng(ne)
    sc = rng.uniform(0.5, 4.0, ne)
    u, s = torch.as_tensor(smooth_field(X, 4e-3, seed=1)), om.init_state()
    v = torch.as_tensor(rng.standard_normal(pm.ndof))
    fixed = np.zeros(pm.ndof, bool)
    fixed[2::5] = True
    free = torch.as_tensor((~fixed).astype(float))
    b.set_fixed(fixed)
    for scale in (None, sc):
        b.set_scale(scale)
        b.tangent_update(u.cuda(), pm.init_state()[0])
        kw = {} if scale is None else dict(scale=[scale])
        assert rel_err(b.tangent_matvec(v.cuda(), apply_bc=False), om.tangent_jvp(u, s, v, **kw)) < 1e-12
        ref = free * om.tangent_jvp(u, s, free * v, **kw) + (1 - free) * v
        assert rel_err(b.tangent_matvec(v.cuda()), ref) < 1e-12


def test_per_element_moduli(cuda):
    import exfem_b200 as xf
    X, c = jittered_box(3, 3, 2, 3, 3, 2, 0.1, 1)
    m = xf.Model(X)
    b = m.add_block(c, xf.HEX8, xf.LinearElastic(E, NU))
    rng = np.random.default_rng(3)
    Es, nus = rng.uniform(1e4, 3e5, b.ne), rng.uniform(0.05, 0.45, b.ne)
    b.set_lame(Es * nus / ((1 + nus) * (1 - 2 * nus)), Es / (2 * (1 + nus)))
    v = torch.as_tensor(rng.standard_normal(m.ndof), device="cuda")
    K = b.stiffness(torch.zeros_like(v), b.init_state())
    assert rel_err(b.tangent_matvec(v, apply_bc=False), b.ebe_matvec(K, v, apply_bc=False)) < 1e-12


@pytest.mark.parametrize("kind,n", [("hex", (100, 40, 30)), ("hex", (101, 40, 30)),
                                    ("tet", (39, 38, 39)), ("tet", (39, 39, 39))])
def test_both_sides_of_the_line(cuda, kind, n):
    """An elastic product is the internal force of v (1e-12)."""
    import exfem_b200 as xf
    X, c = jittered_box(*[float(k) for k in n], *n, 0.1, 1) if kind == "hex" else \
        tet10_box(*[float(k) for k in n], *n, 0.1, 1)
    assert (len(c) <= (120000 if kind == "hex" else 350000)) == (n in ((100, 40, 30), (39, 38, 39)))
    m = xf.Model(X)
    b = m.add_block(c, xf.HEX8 if kind == "hex" else xf.TET10, xf.LinearElastic(E, NU))
    v = torch.randn(m.ndof, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    f, _ = b.internal_force(v, b.init_state())
    assert rel_err(b.tangent_matvec(v, apply_bc=False), f) < 1e-12
    fixed = np.zeros(m.ndof, bool)
    fixed[::7] = True
    fx = torch.as_tensor(fixed, device="cuda")
    b.set_fixed(fixed)
    f, _ = b.internal_force(torch.where(fx, 0.0, v), b.init_state())
    assert rel_err(b.tangent_matvec(v), torch.where(fx, v, f)) < 1e-12


@pytest.mark.parametrize("n", [(100, 40, 30), (101, 40, 30)])
def test_both_sides_of_the_line_j2(cuda, n):
    """The J2 product against the stored element tangents' (1e-12)."""
    import exfem_b200 as xf
    X, c = jittered_box(*[float(k) for k in n], *n, 0.1, 1)
    m = xf.Model(X)
    b = m.add_block(c, xf.HEX8, xf.J2Plasticity(E, NU, TABLE))
    u = torch.as_tensor(smooth_field(X, 3e-3, seed=1), device="cuda")
    s = b.init_state()
    v = torch.randn(m.ndof, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    y = m.tangent_jvp(u, [s], v)
    assert rel_err(y, b.ebe_matvec(b.stiffness(u, s), v, apply_bc=False)) < 1e-12
