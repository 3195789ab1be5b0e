"""J2 return map over hardening tables of one to many rows against the CPU oracle's
25-iteration local Newton: forces, states, stresses and tangents where the return
crosses several table segments, on perfect plasticity, softening and past the table's
last row.  Bar 1e-12 relative (FP64 rounding of the same formulas)."""
import pytest
import torch

from helpers import jittered_box, rel_err, smooth_field, tet10_box
from oracle import fem as ofem

pytestmark = pytest.mark.gpu

TABLES = {
    "perfect": ([[250.0, 0.0]], 0.0),
    "segments": ([[250.0, 0.0], [262.0, 0.001], [300.0, 0.006], [305.0, 0.02], [360.0, 0.08]], 1500.0),
    "softening": ([[250.0, 0.0], [262.0, 0.002], [240.0, 0.03]], 800.0),
    "flat_start": ([[250.0, 0.0], [250.0, 0.004], [300.0, 0.02]], 0.0),
}


@pytest.mark.parametrize("kind", ["hex", "tet"])
@pytest.mark.parametrize("name", sorted(TABLES))
@pytest.mark.parametrize("amp", [1.5e-3, 4e-2])
def test_return_map_over_tables(cuda, kind, name, amp):
    import exfem_b200 as xf
    table, hk = TABLES[name]
    X, c = jittered_box(3, 2, 2, 3, 2, 2, 0.15, 1) if kind == "hex" else tet10_box(2, 1, 1, 2, 1, 1, 0.1, 1)
    om, pm = ofem.Model(X), xf.Model(X)
    om.add_block(c, ofem.HEX8 if kind == "hex" else ofem.TET10, ofem.J2Plasticity(210000.0, 0.3, table, Hk=hk))
    pm.add_block(c, xf.HEX8 if kind == "hex" else xf.TET10, xf.J2Plasticity(210000.0, 0.3, table, Hk=hk))
    _, s1 = om.internal_force(torch.as_tensor(smooth_field(X, 0.6 * amp, seed=3)), om.init_state())
    u = torch.as_tensor(smooth_field(X, amp, seed=5))
    fo, so = om.internal_force(u, s1)
    sp = [s.cuda() for s in s1]
    fp, sn = pm.internal_force(u.cuda(), sp)
    assert float(so[0][..., 9].max()) > 0
    assert rel_err(fp, fo) < 1e-12
    assert rel_err(sn[0], so[0]) < 1e-12
    assert rel_err(pm.element_stiffness(u.cuda(), sp)[0], om.element_stiffness(u, s1)[0]) < 1e-12
    ro, rp = om.stresses(u, s1)[0], pm.stresses(u.cuda(), sp)[0]
    for k in ("S", "MISES", "PEEQ"):
        assert rel_err(rp[k], ro[k]) < 1e-12
