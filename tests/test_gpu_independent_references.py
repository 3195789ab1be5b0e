"""FP64 products, elastic stresses and V-cycle steps against references that share no kernel
with them.  Bars: FP64 sums of a few hundred terms, 1e-12 relative; solves to a residual of
1e-11 with condition numbers below 1e3 of the preconditioned systems, 1e-8."""
import numpy as np
import pytest
import torch

from helpers import jittered_box, rel_err, tet10_box

pytestmark = pytest.mark.gpu

E, NU = 210000.0, 0.3


def _mesh(kind, n):
    return (jittered_box if kind == "hex" else tet10_box)(*[float(k) for k in n], *n, 0.1, 1)


def _block(xf, X, c, kind):
    m = xf.Model(X)
    return m, m.add_block(c, xf.HEX8 if kind == "hex" else xf.TET10, xf.LinearElastic(E, NU))


@pytest.mark.parametrize("kind,n", [("hex", (100, 40, 30)), ("hex", (101, 40, 30)),
                                    ("tet", (39, 38, 39)), ("tet", (39, 39, 39))])
def test_elastic_products_match_stored_matrices(cuda, kind, n):
    """The elastic FP64 product on both sides of the size at which its form changes."""
    import exfem_b200 as xf
    X, c = _mesh(kind, n)
    m, b = _block(xf, X, c, kind)
    v = torch.randn(m.ndof, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    K = b.stiffness(torch.zeros_like(v), b.init_state())
    fixed = np.zeros(m.ndof, bool)
    fixed[::7] = True
    b.set_fixed(fixed)
    for bc in (False, True):
        assert rel_err(b.tangent_matvec(v, apply_bc=bc), b.ebe_matvec(K, v, apply_bc=bc)) < 1e-12


@pytest.mark.parametrize("kind,n", [("hex", (3, 2, 2)), ("tet", (2, 2, 1))])
def test_elastic_plastic_strain_is_zero(cuda, kind, n):
    import exfem_b200 as xf
    X, c = _mesh(kind, n)
    m, b = _block(xf, X, c, kind)
    u = torch.randn(m.ndof, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    assert not m.stresses(u, m.init_state())[0]["PEEQ"].any()


def test_vcycle_of_a_long_prolongation_matches_scalar_matrices(cuda):
    """More prolongation rows than four lanes each would fit on the chip at once."""
    import exfem_b200 as xf
    X, c = _mesh("tet", (22, 22, 21))
    m, b = _block(xf, X, c, "tet")
    fixed = np.zeros((len(X), 3), bool)
    fixed[X[:, 0] < 1e-9] = True
    b.set_fixed(fixed.reshape(-1))
    zero = torch.zeros(m.ndof, dtype=torch.float64, device="cuda")
    amg = xf.DeviceAMG(b, b.stiffness(zero, b.init_state()), keep_level0=True)
    setup = amg.to_setup()
    P = setup["levels"][0]["P"]
    assert len(X) > 148 * 512 and P.nnz / 18 <= 4 * len(X)
    ref = xf.AMG.from_setup(setup)
    r = torch.randn(m.ndof, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    r[torch.as_tensor(fixed.reshape(-1), device="cuda")] = 0.0
    z = ref.vcycle(r)
    assert rel_err(amg.vcycle(r), z) < 1e-12
    assert rel_err(amg.vcycle(r.float()), z) < 2e-5


@pytest.mark.parametrize("count", [1, 2])
@pytest.mark.parametrize("op", ["mf64", "ebe64", "csr64", "mf32"])
def test_right_hand_side_on_prescribed_dofs(cuda, op, count):
    """opA is the identity on prescribed DOFs and couples them to nothing: with a
    right-hand side that is not zero there, the solution is that of the masked one plus the
    right-hand side's prescribed entries, in the same iterations and at most a few more
    (one further eigenvalue, 1)."""
    import exfem_b200 as xf
    X, c = _mesh("hex", (16, 6, 5))
    m = xf.Model(X)
    for part in np.array_split(np.arange(len(c)), count):
        m.add_block(c[part], xf.HEX8, xf.LinearElastic(E, NU))
    fixed = np.zeros((len(X), 3), bool)
    fixed[X[:, 0] < 1e-9] = True
    for b in m.blocks:
        b.set_fixed(fixed.reshape(-1))
    zero = torch.zeros(m.ndof, dtype=torch.float64, device="cuda")
    Kes = [b.stiffness(zero, b.init_state()) for b in m.blocks]
    amg = xf.DeviceAMG(m.blocks, Kes)
    ns = xf.NativeSolver(m.blocks, op, "amg", amg)
    if op in ("ebe64", "csr64"):
        ns.set_ke(Kes)
    fx = torch.as_tensor(fixed.reshape(-1), device="cuda")
    rhs = torch.randn(m.ndof, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    masked = torch.where(fx, 0.0, rhs)
    solve = (lambda f: ns.mixed(f, tol=1e-11)) if op == "mf32" else (lambda f: ns.pcg(f, tol=1e-11))
    x0, k0 = solve(masked)[:2]
    x1, k1 = solve(rhs)[:2]
    assert not x0[fx].any()
    assert rel_err(x1[fx], rhs[fx]) < 1e-8
    assert rel_err(x1[~fx], x0[~fx]) < 1e-8
    assert k1 <= k0 + 3, (k1, k0)
