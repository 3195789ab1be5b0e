"""A bounded device wait that gave up in any block of a synchronising call makes that call
report EXFEM_ERR_TIMEOUT, once: the flag is set by the self-test wait (nothing faults), the
call that follows raises and the next one succeeds."""
import numpy as np
import pytest
import torch

from helpers import cantilever_bcs, jittered_box

pytestmark = pytest.mark.gpu


def _blocks(xf, count):
    X, c = jittered_box(50.0, 20.0, 20.0, 10, 4, 4, 0.1, 1)
    m = xf.Model(X)
    for part in np.array_split(np.arange(len(c)), count):
        m.add_block(c[part], xf.HEX8, xf.LinearElastic(210e3, 0.3))
    fixed = np.zeros((len(X), 3), bool)
    fixed[X[:, 0] < 1e-9] = True
    for b in m.blocks:
        b.set_fixed(fixed.reshape(-1))
    f = np.zeros((len(X), 3))
    f[X[:, 0] > 50.0 - 1e-9, 2] = -1.0
    return X, m, torch.as_tensor(f.reshape(-1), device="cuda")


def _multi_pcg(xf):
    X, m, f = _blocks(xf, 1)
    b = m.blocks[0]
    Ke = b.stiffness(torch.zeros_like(f), b.init_state())
    return m.blocks, lambda: b.multi_pcg(Ke, torch.stack([f, 2 * f], 1))


def _solver(op, call):
    def make(xf):
        X, m, f = _blocks(xf, 2)
        Kes = [b.stiffness(torch.zeros_like(f), b.init_state()) for b in m.blocks]
        ns = xf.NativeSolver(m.blocks, op, "jacobi")
        if op == "ebe64":
            ns.set_ke(Kes)
        return m.blocks, lambda: getattr(ns, call)(f)
    return make


def _newton(xf):
    X, m, f = _blocks(xf, 2)
    fix, tip, bcs, loads = cantilever_bcs(X, 50.0)
    s = xf.StaticSolver(m, rtol=1e-6, linear_solver="mixed", tangent="mf", verbose=False)
    assert s._device_increment_ok()
    return m.blocks, lambda: s.solve(xf.Step(bcs=bcs, loads=loads))


def _batch(xf):
    from exfem_b200 import batch
    p = batch.cantilever(6, 2, 2, 5.0, xf.LinearElastic(210e3, 0.3), [[0.0, 0.0, -10.0]])
    S = batch.BatchSolver([p], workers=0, amg_setup="host")
    return [S.block], lambda: S.solve()


def _modal(xf):
    X, m, f = _blocks(xf, 2)
    fix, tip, bcs, loads = cantilever_bcs(X, 50.0)
    from exfem_b200 import eigen
    return m.blocks, lambda: eigen.modal_lobpcg(m, xf.Step(bcs=bcs), 2, tol=1e-4)


CALLS = dict(multi_pcg=_multi_pcg, ebe64=_solver("ebe64", "pcg"), mf64=_solver("mf64", "pcg"),
             mixed=_solver("mf32", "mixed"), newton=_newton, batch=_batch, modal=_modal)


@pytest.mark.parametrize("call", sorted(CALLS))
def test_a_failed_wait_in_any_block_is_reported_once(cuda, call):
    import exfem_b200 as xf
    from exfem_b200 import _lib
    blocks, run = CALLS[call](xf)
    run()
    for b in blocks:
        assert _lib.lib.exfem_selftest_block_wait(b.handle, 1 << 10, _lib.stream_ptr()) == _lib.OK
        with pytest.raises(_lib.ExfemError, match="bounded device wait gave up"):
            run()
        run()
        assert _lib.lib.exfem_block_status(b.handle, _lib.stream_ptr()) == _lib.OK
