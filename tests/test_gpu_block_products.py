"""Block-sparse level products at every lane count their rows select (1 to 256 lanes per
block row): a V-cycle of the device set-up, whose matrices are block-sparse, against the
same hierarchy uploaded as scalar CSR matrices.  Bars: FP64 1e-12, FP32 2e-5 relative
(a few hundred products of rounding error 1e-16 / 6e-8 through two smoothed levels)."""
import numpy as np
import pytest
import torch

from helpers import jittered_box, rel_err, tet10_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n", [("hex", (6, 3, 2)), ("hex", (20, 6, 5)), ("hex", (12, 12, 11)),
                                    ("tet", (5, 4, 4)), ("tet", (11, 9, 8))])
@pytest.mark.parametrize("max_coarse", [30, 300])
def test_vcycle_matches_scalar_matrices(cuda, kind, n, max_coarse):
    import exfem_b200 as xf
    X, c = (jittered_box if kind == "hex" else tet10_box)(*[float(k) for k in n], *n, 0.1, 1)
    m = xf.Model(X)
    b = m.add_block(c, xf.HEX8 if kind == "hex" else xf.TET10, xf.LinearElastic(210000.0, 0.3))
    fixed = np.zeros((len(X), 3), bool)
    fixed[X[:, 0] < 1e-9] = True
    b.set_fixed(fixed.reshape(-1))
    zero = torch.zeros(m.ndof, dtype=torch.float64, device="cuda")
    amg = xf.DeviceAMG(b, b.stiffness(zero, b.init_state()), max_coarse=max_coarse, keep_level0=True)
    ref = xf.AMG.from_setup(amg.to_setup())
    r = torch.randn(m.ndof, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    r[torch.as_tensor(fixed.reshape(-1), device="cuda")] = 0.0
    z = ref.vcycle(r)
    assert rel_err(amg.vcycle(r), z) < 1e-12
    assert rel_err(amg.vcycle(r.float()), z) < 2e-5
    d = 1.0 / b.tangent_diagonal()
    assert rel_err(amg.vcycle(r, level0=b, dinv0=d), ref.vcycle(r, level0=b, dinv0=d)) < 1e-12
