"""Element tangents at the sizes and forms their kernel treats differently: element
counts around a warp's share (4 C3D8 or 8 C3D10) and a thread block's, every stored
precision, matrices that do not start on a 16-byte boundary, per-element scale and
Lame parameters, and the diagonal-only form."""
import numpy as np
import pytest
import torch

from helpers import jittered_box, rel_err, smooth_field, tet10_box
from oracle import fem as ofem

pytestmark = pytest.mark.gpu

E, NU = 210000.0, 0.3
TABLE = [[250.0, 0.0], [1250.0, 1.0]]


def _models(kind, mat, ne):
    import exfem_b200 as xf
    X, c = jittered_box(9, 2, 2, 9, 2, 2, 0.15, 2) if kind == "hex" else tet10_box(4, 1, 2, 4, 1, 2, 0.1, 2)
    c = c[:ne]
    args = (E, NU) if mat == "el" else (E, NU, TABLE)
    om, pm = ofem.Model(X), xf.Model(X)
    om.add_block(c, ofem.HEX8 if kind == "hex" else ofem.TET10,
                 (ofem.LinearElastic if mat == "el" else ofem.J2Plasticity)(*args))
    pm.add_block(c, xf.HEX8 if kind == "hex" else xf.TET10, (xf.LinearElastic if mat == "el" else xf.J2Plasticity)(*args))
    return X, om, pm


@pytest.mark.parametrize("kind", ["hex", "tet"])
@pytest.mark.parametrize("mat", ["el", "j2"])
@pytest.mark.parametrize("ne", [1, 3, 4, 5, 8, 9, 16, 17, 33])
def test_ragged_element_counts(cuda, kind, mat, ne):
    """FP64 1e-12 (rounding); FP32 6e-8 and BF16 4e-3 of the largest entry (half a unit
    in the last place of each format, plus the FP64 difference)."""
    X, om, pm = _models(kind, mat, ne)
    _, s1 = om.internal_force(torch.as_tensor(smooth_field(X, 2e-3, seed=3)), om.init_state())
    u = torch.as_tensor(smooth_field(X, 4e-3, seed=1))
    Ko = om.element_stiffness(u, s1)[0]
    sp = [s.cuda() for s in s1]
    for dtype, bar in ((torch.float64, 1e-12), (torch.float32, 6.1e-8), (torch.bfloat16, 4e-3)):
        Kp = pm.element_stiffness(u.cuda(), sp, dtype=dtype)[0]
        assert Kp.dtype == dtype and rel_err(Kp.double(), Ko) < bar
    b = pm.blocks[0]
    b.tangent_update(u.cuda(), sp[0])
    d = pm.diagonal([b.stiffness(u.cuda(), sp[0])])
    assert rel_err(b.tangent_diagonal(), d) < 1e-12


@pytest.mark.parametrize("kind", ["hex", "tet"])
def test_unaligned_scaled_and_per_element_moduli(cuda, kind):
    from exfem_b200 import _lib
    X, om, pm = _models(kind, "el", 21)
    b = pm.blocks[0]
    u = torch.as_tensor(smooth_field(X, 1e-3), device="cuda")
    K = b.stiffness(u, b.init_state())
    nd = b.etype.nd
    buf = torch.zeros(1 + K.numel(), dtype=torch.float64, device="cuda")[1:]
    assert buf.data_ptr() % 16 == 8
    _lib.check(_lib.lib.exfem_element_stiffness(b.handle, u.data_ptr(), None, _lib.F64, buf.data_ptr(),
                                                _lib.stream_ptr()))
    torch.testing.assert_close(buf.reshape(-1, nd, nd), K, rtol=0, atol=0)
    rng = np.random.default_rng(4)
    sc = rng.uniform(0.5, 4.0, b.ne)
    b.set_scale(sc)
    assert rel_err(b.stiffness(u, b.init_state()), K * torch.as_tensor(sc, device="cuda")[:, None, None]) < 1e-14
    b.set_scale(None)
    Es, nus = rng.uniform(1e4, 3e5, b.ne), rng.uniform(0.05, 0.45, b.ne)
    b.set_lame(Es * nus / ((1 + nus) * (1 - 2 * nus)), Es / (2 * (1 + nus)))
    got = b.stiffness(u, b.init_state())
    import exfem_b200 as xf
    for e in (0, 7, 20):
        m = xf.Model(X)
        one = m.add_block(b.conn[e:e + 1], b.etype, xf.LinearElastic(Es[e], nus[e]))
        assert rel_err(got[e], one.stiffness(u, one.init_state())[0]) < 1e-12
    d = pm.diagonal([got])
    assert rel_err(b.tangent_diagonal(), d) < 1e-12
    b.set_lame(None, None)
