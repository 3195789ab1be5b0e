"""A J2 request among saturating linear requests is served beside them: it shares the GPU
with the running solves and does not wait until they leave it idle."""
import numpy as np
import pytest

from exfem_b200 import batch, elements, mesh, serve
from exfem_b200.materials import J2Plasticity, LinearElastic
from exfem_b200.solvers import Step

pytestmark = pytest.mark.gpu

MESHES, ROUNDS = 12, 40


def _linear_spec(i):
    et = elements.HEX8 if i % 2 else elements.TET10
    n = (64, 16, 16) if i % 2 else (32, 8, 8)                      # 56,355 DOF either way
    p = batch.cantilever(*n, 5.0, LinearElastic(210e3, 0.3), [[0.0, 0.0, -500.0]], etype=et)
    return serve.MeshSpec(f"lin{i}", p.X, p.conn, et, p.material, p.fixed), p.rhs[0]


def _j2_spec():
    L = 160.0
    X, c = mesh.box_hex(L, 40.0, 40.0, 32, 8, 8)
    fix = mesh.nodes_where(X, lambda x, y, z: x < 1e-9)
    tip = mesh.nodes_where(X, lambda x, y, z: x > L - 1e-9)
    fixed = np.zeros(3 * len(X), bool)
    for d in range(3):
        fixed[3 * fix + d] = True
    step = Step(bcs=[(fix, d, 0.0) for d in range(3)] + [(tip, 2, -L / 400.0)], dt_init=0.2, dt_max=0.2)
    mat = J2Plasticity(210e3, 0.3, [[250.0, 0.0], [1250.0, 1.0]])
    return serve.MeshSpec("j2", X, c, elements.HEX8, mat, fixed), step


def test_j2_request_is_served_during_a_linear_backlog(cuda):
    linear = [_linear_spec(i) for i in range(MESHES)]
    j2, step = _j2_spec()
    with serve.SolveServer(slots=MESHES + 1) as srv:
        srv.warm([sp for sp, _ in linear] + [j2])
        for f in [srv.submit(serve.SolveRequest(sp, rhs=r)) for sp, r in linear]:
            f.result(timeout=300)
        srv.submit(serve.SolveRequest(j2, step=step)).result(timeout=300)
        backlog = [serve.SolveRequest(sp, rhs=r) for _ in range(ROUNDS) for sp, r in linear]
        futs = [srv.submit(q) for q in backlog]
        q = serve.SolveRequest(j2, step=step)
        srv.submit(q).result(timeout=300)
        for f in futs:
            f.result(timeout=300)
    # thirteen slots share the GPU: a J2 request's work, a few linear solves' worth, takes a
    # fraction of the 40 rounds however the slots are served; one that waits for an idle GPU
    # ends with the last round
    total = max(b.t_done for b in backlog) - q.t_start
    assert q.t_done - q.t_start < 0.5 * total, (q.t_done - q.t_start, total)
