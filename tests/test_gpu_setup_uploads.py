"""The device set-up's index arrays are in place before its kernels read them: set-ups on
the default stream and on a side stream, with the device memory they are handed holding
NaN bit patterns, all give the same hierarchy."""
import numpy as np
import pytest
import torch

from helpers import jittered_box

pytestmark = pytest.mark.gpu


def test_setups_on_used_memory_agree(cuda):
    import exfem_b200 as xf
    X, c = jittered_box(20.0, 6.0, 5.0, 20, 6, 5, 0.1, 1)
    fixed = np.zeros((len(X), 3), bool)
    fixed[X[:, 0] < 1e-9] = True

    def setup():
        old = [torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
               for n in (1 << 20, 1 << 17, 1 << 14, 1 << 12) for _ in range(3)]
        torch.cuda.synchronize()
        del old
        torch.cuda.empty_cache()                 # the library's allocations get these pages
        m = xf.Model(X)
        b = m.add_block(c, xf.HEX8, xf.LinearElastic(210000.0, 0.3))
        b.set_fixed(fixed.reshape(-1))
        K = b.stiffness(torch.zeros(m.ndof, dtype=torch.float64, device="cuda"), b.init_state())
        return xf.DeviceAMG(b, K, max_coarse=30, keep_level0=True).to_setup()

    want = setup()
    for k in range(6):
        with torch.cuda.stream(torch.cuda.Stream() if k % 2 else torch.cuda.current_stream()):
            got = setup()
        for a, w in zip(got["levels"], want["levels"]):
            assert a["rho"] == w["rho"]
            for name in ("A", "P", "R"):
                np.testing.assert_array_equal(a[name].indices, w[name].indices)
                np.testing.assert_array_equal(a[name].data, w[name].data)
        np.testing.assert_array_equal(got["coarse_inv"], want["coarse_inv"])
