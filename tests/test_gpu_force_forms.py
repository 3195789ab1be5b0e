"""Internal force, states and stresses at the sizes and forms their kernel treats
differently: element counts around a warp's share (4 C3D8, 8 C3D10) and a thread
block's, states updated in place, states and element forces that do not start on a
16-byte boundary, and the state copy of elastic blocks."""
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
    """Bar 1e-12 relative (FP64 rounding), forces, states, stresses and the product with
    the tangent data the force call leaves behind."""
    X, om, pm = _models(kind, mat, ne)
    _, s1 = om.internal_force(torch.as_tensor(smooth_field(X, 2e-3, seed=3)), om.init_state())
    u = torch.as_tensor(smooth_field(X, 4e-3, seed=1))
    fo, so = om.internal_force(u, s1)
    sp = [s.cuda() for s in s1]
    fp, sn = pm.internal_force(u.cuda(), sp)
    assert rel_err(fp, fo) < 1e-12
    if mat == "j2":
        assert rel_err(sn[0], so[0]) < 1e-12
    ro, rp = om.stresses(u, s1)[0], pm.stresses(u.cuda(), sp)[0]
    for k in ("S", "MISES", "PEEQ"):
        assert rel_err(rp[k], ro[k]) < 1e-12 or float(ro[k].abs().max()) == 0.0
    v = torch.randn(pm.ndof, dtype=torch.float64, generator=torch.Generator().manual_seed(1))
    y = pm.blocks[0].tangent_matvec(v.cuda(), apply_bc=False)
    assert rel_err(y, om.tangent_jvp(u, s1, v)) < 1e-12


@pytest.mark.parametrize("kind", ["hex", "tet"])
def test_states_in_place_and_unaligned(cuda, kind):
    from exfem_b200 import _lib
    from exfem_b200._lib import check, lib, ptr, stream_ptr
    X, om, pm = _models(kind, "j2", 21)
    b = pm.blocks[0]
    u = torch.as_tensor(smooth_field(X, 4e-3, seed=1), device="cuda")
    s0 = b.init_state()
    f, s1 = b.internal_force(u, s0)
    f2 = torch.empty_like(f)
    place = s0.clone()
    check(lib.exfem_internal_force(b.handle, ptr(u), ptr(place), ptr(place), None, ptr(f2), _lib.ASSEMBLE_GATHER,
                                   stream_ptr()))
    torch.testing.assert_close(place, s1, rtol=0, atol=0)
    torch.testing.assert_close(f2, f, rtol=0, atol=0)
    fe = torch.empty(21 * b.etype.nd, dtype=torch.float64, device="cuda")
    check(lib.exfem_internal_force(b.handle, ptr(u), ptr(s0), None, ptr(fe), ptr(f2), _lib.ASSEMBLE_GATHER,
                                   stream_ptr()))
    bufs = [torch.zeros(1 + n, dtype=torch.float64, device="cuda")[1:] for n in (s0.numel(), s0.numel(), fe.numel())]
    bufs[0].copy_(s0.reshape(-1))
    assert all(t.data_ptr() % 16 == 8 for t in bufs)
    check(lib.exfem_internal_force(b.handle, ptr(u), *[t.data_ptr() for t in bufs], ptr(f2), _lib.ASSEMBLE_GATHER,
                                   stream_ptr()))
    torch.testing.assert_close(bufs[1].reshape(s1.shape), s1, rtol=0, atol=0)
    torch.testing.assert_close(bufs[2], fe, rtol=0, atol=0)
    torch.testing.assert_close(f2, f, rtol=0, atol=0)


def test_elastic_state_is_copied(cuda):
    from exfem_b200 import _lib
    from exfem_b200._lib import check, lib, ptr, stream_ptr
    X, om, pm = _models("hex", "el", 9)
    b = pm.blocks[0]
    u = torch.as_tensor(smooth_field(X, 1e-3), device="cuda")
    old = torch.rand(9, 8, 1, dtype=torch.float64, device="cuda")
    new, f = torch.full_like(old, -1.0), torch.empty(pm.ndof, dtype=torch.float64, device="cuda")
    check(lib.exfem_internal_force(b.handle, ptr(u), ptr(old), ptr(new), None, ptr(f), _lib.ASSEMBLE_GATHER,
                                   stream_ptr()))
    torch.testing.assert_close(new, old, rtol=0, atol=0)
