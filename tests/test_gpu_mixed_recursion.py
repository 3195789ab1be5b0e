"""The FP32 recursion of the mixed solver on meshes whose moduli spread over a decade (the
V-cycle is indefinite on some vectors there): it converges in about the FP64 PCG's
iterations, restarted or with replaced residuals, and does not stall."""
import numpy as np
import pytest
import torch

from helpers import tet10_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,seed", [(28, 8), (32, 7)])
def test_fp32_recursion_keeps_up_with_fp64(cuda, n, seed):
    from exfem_b200 import elements, linalg
    from exfem_b200.materials import LinearElastic
    from exfem_b200.model import Block
    X, c = tet10_box(1.0, 1.0, 1.0, n, n, n, 0.1, 0)
    b = Block(c, elements.TET10, LinearElastic(1000.0, 0.3), X=X)
    fixed = np.zeros((len(X), 3), bool)
    fixed[X[:, 2] < 1e-9] = True
    b.set_fixed(fixed.reshape(-1))
    b.set_scale(np.exp(np.random.default_rng(seed).uniform(0.0, np.log(10.0), size=len(c))))
    f = np.zeros((len(X), 3))
    f[X[:, 2] > 1.0 - 1e-9, 2] = 1.0
    f = torch.as_tensor(f.reshape(-1), device="cuda")
    zero = torch.zeros(b.nn * 3, dtype=torch.float64, device="cuda")
    amg = linalg.DeviceAMG(b, b.stiffness(zero, b.init_state()))
    x64, k64, _ = linalg.NativeSolver(b, "mf64", "amg", amg).pcg(f, tol=1e-8)
    for mode in ("reliable", "restart"):
        x, k, passes, rel = linalg.NativeSolver(b, "mf32", "amg", amg, mixed_mode=mode).mixed(f, tol=1e-8)
        assert rel <= 1e-8
        # a restart gives up the Krylov space of the pass before: at most the FP64 count again
        assert k <= 2 * k64, (mode, k, k64)
        assert float((x - x64).norm() / x64.norm()) < 1e-5
