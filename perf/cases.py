"""The measured work of the framework, through its public entry points.

Residual (internal force), tangent (element stiffness), stress recovery, tangent
products (matrix-free and stored) and linear solves, on the meshes the repository
itself uses: C3D8 cantilever beams from the 1,575-DOF one to the 133,623-DOF
100 x 20 x 20 elastoplastic one, and C3D10 unit cubes split into 6 Kuhn tetrahedra
per hexahedron.  Interior nodes are jittered by 10% of the spacing.  Materials are
steel-like (E = 210 GPa, nu = 0.3); J2 blocks carry a plastic history near the
clamped end, and the displacement field loads about a third of the Gauss points
plastically, the rest elastically.
"""
import math

import numpy as np
import torch

import exfem_b200 as xf
from exfem_b200 import mesh

E, NU = 210000.0, 0.3
MU = E / (2 * (1 + NU))
LAM = E * NU / ((1 + NU) * (1 - 2 * NU))
BULK = LAM + 2 * MU / 3
HARDENING = {                                    # hardening tables and kinematic moduli
    "bilinear": ([[250.0, 0.0], [1250.0, 1.0]], 0.0),
    "table": ([[250.0, 0.0], [290.0, 0.01], [330.0, 0.05], [380.0, 0.2]], 500.0),
}
F64 = torch.float64
DTYPES = {"f64": torch.float64, "f32": torch.float32, "bf16": torch.bfloat16}


def _case(name, op, etype, material, n, **more):
    c = dict(op=op, etype=etype, material=material, nx=n[0], ny=n[1], nz=n[2], **more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the residual of the 1,575-DOF cantilever: the smallest call, launches and host only
        _case("force_c3d8_small", "force", "C3D8", "elastic", (20, 4, 4)),
        # Newton residual and state update of the elastoplastic beam (133,623 DOF)
        _case("force_c3d8_j2_beam", "force", "C3D8", "bilinear", (100, 20, 20)),
        # the same on a quadratic tetrahedral part, odd sizes, longer hardening table
        _case("force_c3d10_j2", "force", "C3D10", "table", (31, 27, 25)),
        # stress recovery after a converged increment
        _case("stress_c3d8_j2_beam", "stress", "C3D8", "bilinear", (100, 20, 20)),
        # Newton tangent of the elastoplastic beam (plain FP64 method, AMG set-up)
        _case("tangent_c3d8_j2_beam", "tangent", "C3D8", "bilinear", (100, 20, 20)),
        # element matrices of a linear quadratic-tetrahedron part (AMG set-up)
        _case("tangent_c3d10", "tangent", "C3D10", "elastic", (25, 23, 21)),
        # FP32 product of the mixed-precision solver, streaming size
        _case("product_c3d10_f32", "product", "C3D10", "elastic", (48, 48, 48), dtype="f32"),
        # tangent linearisation and FP64 product of the elastoplastic beam
        _case("product_c3d8_j2_f64", "product", "C3D8", "bilinear", (100, 20, 20), dtype="f64"),
        # stored-Ke FP64 product of the plain method, odd sizes
        _case("stored_c3d8_f64", "stored", "C3D8", "elastic", (93, 23, 19), dtype="f64", nrhs=1),
        # four load cases at once on BF16 element matrices
        _case("multi_c3d8_bf16", "stored", "C3D8", "elastic", (128, 32, 32), dtype="bf16", nrhs=4),
        # whole linear solve of the small cantilever, plain FP64 AMG-PCG
        _case("solve_small_f64", "solve", "C3D8", "elastic", (20, 4, 4), dtype="f64"),
        # whole linear solve of a 481,000-DOF quadratic part, FP32 inside FP64
        _case("solve_c3d10_mixed", "solve", "C3D10", "elastic", (27, 27, 26), dtype="f32"),
    ]


# largest element counts drawn per operation: those of the listed cases
_MOST = {("force", "C3D8"): 40000, ("force", "C3D10"): 125550, ("stress", "C3D8"): 40000, ("stress", "C3D10"): 60000,
         ("tangent", "C3D8"): 40000, ("tangent", "C3D10"): 72450, ("product", "C3D8"): 130000,
         ("product", "C3D10"): 660000, ("stored", "C3D8"): 130000, ("stored", "C3D10"): 60000,
         ("solve", "C3D8"): 40000, ("solve", "C3D10"): 110000}


def draw(rng):
    op = rng.choice(["force", "stress", "tangent", "product", "stored", "solve"])
    etype = rng.choice(["C3D8", "C3D10"])
    material = "elastic"
    if op in ("force", "stress", "tangent", "product"):
        material = rng.choice(["elastic", "bilinear"] if op == "product" else ["elastic", "bilinear", "table"])
    per = 1 if etype == "C3D8" else 6
    most = _MOST[op, etype] if material == "elastic" else min(_MOST[op, etype], 125550)
    hexes = math.exp(rng.uniform(math.log(60), math.log(most / per)))
    aspect = rng.uniform(1.5, 5.0) if etype == "C3D8" else rng.uniform(1.0, 2.0)
    side = (hexes / aspect) ** (1.0 / 3.0)
    ny = max(2, int(side * rng.uniform(0.85, 1.15)))
    nz = max(2, int(side * rng.uniform(0.85, 1.15)))
    n = (max(2, int(hexes / (ny * nz))), ny, nz)
    if op in ("force", "stress", "tangent"):
        return _case(None, op, etype, material, n)
    if op == "product":
        return _case(None, op, etype, material, n, dtype=rng.choice(["f32", "f64"]))
    if op == "stored":
        dtype = rng.choice(["f64", "f64", "f32", "bf16"])
        nrhs = rng.choice([1, 2, 3, 4, 8, 16] if dtype == "f64" else [2, 3, 4, 8, 16])
        return _case(None, op, etype, "elastic", n, dtype=dtype, nrhs=nrhs)
    return _case(None, op, etype, "elastic", n, dtype=rng.choice(["f32", "f64"]))


# ------------------------------------------------------------------ inputs
def _mesh(case, seed):
    n = (case["nx"], case["ny"], case["nz"])
    size = [5.0 * k for k in n] if case["etype"] == "C3D8" else [k / max(n) for k in n]
    X, c = mesh.box_hex(*size, *n)
    X = mesh.jitter_interior(X, [s / k for s, k in zip(size, n)], 0.1, seed)
    if case["etype"] == "C3D10":
        X, c = mesh.tet4_to_tet10(*mesh.hex_to_tet4(X, c))
    return X, np.ascontiguousarray(c, dtype=np.int32), size


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _bending(X, size, amp):
    """Displacement of a cantilever in bending, strain amp (1 - x / L) eta."""
    x, y = X[:, 0], X[:, 1]
    L, H = size[0], size[1]
    eta = 2.0 * y / H - 1.0
    u = torch.zeros_like(X)
    u[:, 0] = amp * (x - x * x / (2 * L)) * eta
    u[:, 1] = -(2 * amp / H) * (x * x / 2 - x ** 3 / (6 * L))
    return u


def _fields(case, seed):
    """Mesh, displacement, and (J2) Gauss-point state of a case, as CUDA tensors."""
    X, c, size = _mesh(case, seed)
    g = _gen(seed)
    Xd = torch.as_tensor(X, device="cuda")
    cd = torch.as_tensor(c, device="cuda").long()
    amp = 5e-3 if case["material"] != "elastic" else 1e-3
    h = size[0] / case["nx"]
    u = _bending(Xd, size, amp) + 2e-5 * h * torch.randn(Xd.shape, dtype=F64, device="cuda", generator=g)
    state = None
    if case["material"] != "elastic":
        ngp = 8 if case["etype"] == "C3D8" else 4
        hk = HARDENING[case["material"]][1]
        xc = Xd[cd].mean(1)
        strain = amp * (1 - xc[:, 0] / size[0]) * (2 * xc[:, 1] / size[1] - 1)
        past = (0.85 * strain.abs() - 1.6e-3).clamp(min=0) * torch.sign(strain)
        past = past[:, None] * (1 + 0.05 * torch.randn((len(c), ngp), dtype=F64, device="cuda", generator=g))
        state = torch.zeros((len(c), ngp, 19), dtype=F64, device="cuda")
        for k, w in ((0, 1.0), (4, -0.5), (8, -0.5)):
            state[..., k] = w * past
            state[..., 10 + k] = 2.0 / 3.0 * hk * w * past
        state[..., 9] = past.abs()
    return X, c, size, Xd, cd, u.reshape(-1), state


def _clamped(X):
    fixed = np.zeros((len(X), 3), bool)
    fixed[X[:, 0] < 1e-9] = True
    return fixed.reshape(-1)


def _tip_load(X, size, seed):
    tip = np.nonzero(X[:, 0] > size[0] * (1 - 1e-9))[0]
    rng = np.random.default_rng(seed)
    f = np.zeros((len(X), 3))
    f[tip] = rng.uniform(-1, 1, 3) * 100.0 / len(tip) * (1 + 0.2 * rng.standard_normal((len(tip), 1)))
    return torch.as_tensor(f.reshape(-1), device="cuda")


def _material(case):
    if case["material"] == "elastic":
        return xf.LinearElastic(E, NU)
    table, hk = HARDENING[case["material"]]
    return xf.J2Plasticity(E, NU, table, Hk=hk)


def prepare(case, seed):
    X, c, size, Xd, cd, u, state = _fields(case, seed)
    m = xf.Model(X)
    b = m.add_block(c, xf.ELEMENTS[case["etype"]], _material(case))
    s = dict(case=case, model=m, block=b, u=u, states=[state if state is not None else b.init_state()])
    if case["op"] == "product":
        s["v"] = torch.randn(m.ndof, dtype=DTYPES[case["dtype"]], device="cuda", generator=_gen(seed + 1))
        if case["dtype"] == "f32":               # the solver's operator: prescribed DOFs, current tangent
            b.set_fixed(_clamped(X))
            m.tangent_update(u, s["states"])
    elif case["op"] == "stored":
        s["Ke"] = _element_matrices(case, Xd, cd, u, state).to(DTYPES[case["dtype"]])
        vt = F64 if case["dtype"] == "f64" else torch.float32
        shape = (m.ndof, case["nrhs"]) if case["nrhs"] > 1 else (m.ndof,)
        s["v"] = torch.randn(shape, dtype=vt, device="cuda", generator=_gen(seed + 1))
        b.set_fixed(_clamped(X))
    elif case["op"] == "solve":
        b.set_fixed(_clamped(X))
        amg = xf.DeviceAMG(b, b.stiffness(torch.zeros_like(u), s["states"][0]))
        s["solver"] = xf.NativeSolver(b, op="mf64" if case["dtype"] == "f64" else "mf32", pc="amg", amg=amg)
        s["rhs"] = _tip_load(X, size, seed)
    return s


def run(s):
    case, m, b = s["case"], s["model"], s["block"]
    op = case["op"]
    if op == "force":
        f, new = m.internal_force(s["u"], s["states"])
        return [f] if case["material"] == "elastic" else [f, new[0]]
    if op == "stress":
        return m.stresses(s["u"], s["states"])[0]
    if op == "tangent":
        return m.element_stiffness(s["u"], s["states"])
    if op == "product":
        return b.tangent_matvec(s["v"]) if case["dtype"] == "f32" else m.tangent_jvp(s["u"], s["states"], s["v"])
    if op == "stored":
        return b.ebe_matvec(s["Ke"], s["v"]) if case["nrhs"] == 1 else b.ebe_matvec_multi(s["Ke"], s["v"])
    if case["dtype"] == "f64":
        return s["solver"].pcg(s["rhs"], tol=1e-11)[0]
    return s["solver"].mixed(s["rhs"], tol=1e-11)[0]


# ------------------------------------------------------------------ work
def _counts(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["etype"] == "C3D8":
        return nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1), 8, 8
    # corners, and one mid-node per distinct edge of the Kuhn split
    corners = (nx + 1) * (ny + 1) * (nz + 1)
    edges = (nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
             + nx * ny * (nz + 1) + nx * (ny + 1) * nz + (nx + 1) * ny * nz + nx * ny * nz)
    return 6 * nx * ny * nz, corners + edges, 10, 4


def work(case):
    """Mesh (FP64 coordinates, int32 connectivity), inputs and outputs once each; the
    arithmetic of one strain, stress and force (or tangent) evaluation per Gauss point."""
    ne, nn, nnode, ngp = _counts(case)
    j2 = case["material"] != "elastic"
    topo, vec = 4 * ne * nnode, 24 * nn
    states = 8 * 19 * ne * ngp if j2 else 0
    point = 36 * nnode + 120 + (200 if j2 else 0)
    nd = 3 * nnode
    op = case["op"]
    if op == "force":
        return dict(bytes=topo + 3 * vec + 2 * states, flops=ne * ngp * (point + 18 * nnode))
    if op == "stress":
        return dict(bytes=topo + 2 * vec + states + 88 * ne, flops=ne * ngp * point)
    if op == "tangent":
        return dict(bytes=topo + 2 * vec + states + 8 * ne * nd * nd, flops=ne * ngp * (point + 18 * nnode * nnode))
    if op == "product":
        w = 4 if case["dtype"] == "f32" else 8
        # vector in and out, connectivity, coordinates; FP32: the J2 tangent kept (6 + 2 a point)
        data = 8 * 4 * ne * ngp if j2 and w == 4 else states
        return dict(bytes=6 * w * nn + topo + (12 if w == 4 else 24) * nn + data, flops=ne * ngp * 54 * nnode)
    if op == "stored":
        w = {"f64": 8, "f32": 4, "bf16": 2}[case["dtype"]]
        vw = 8 if case["dtype"] == "f64" else 4
        return dict(bytes=ne * nd * nd * w + topo + 6 * vw * nn * case["nrhs"], flops=2 * ne * nd * nd * case["nrhs"])
    # solve: the preconditioned iteration to 1e-11 applies the operator about 100 times
    # (25 iterations, each one product and four in the smoother)
    w = 4 if case["dtype"] == "f32" else 8
    return dict(bytes=100 * (6 * w * nn + topo + 12 * nn), flops=100 * ne * ngp * 54 * nnode)


# ------------------------------------------------------------------ values in 64 bits
def _tables(etype):
    """dN/dxi at the Gauss points (ngp, nnode, 3), weights, and at the centre (C3D8)."""
    if etype == "C3D8":
        sg = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], float)

        def grad(p):
            f = 1 + sg * p
            return 0.125 * np.stack([sg[:, 0] * f[:, 1] * f[:, 2], f[:, 0] * sg[:, 1] * f[:, 2], f[:, 0] * f[:, 1] * sg[:, 2]], 1)
        dN = np.stack([grad(p / math.sqrt(3.0)) for p in sg])
        w, dN0 = 1.0, grad(np.zeros(3))
    else:
        a, b = 0.5854101966249685, 0.1381966011250105
        dL = np.array([[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]])
        out = []
        for p in ([b, b, b], [a, b, b], [b, a, b], [b, b, a]):
            L = np.array([1 - sum(p), *p])
            d = [(4 * L[k] - 1) * dL[k] for k in range(4)]
            d += [4 * (L[i] * dL[j] + L[j] * dL[i]) for i, j in ((0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3))]
            out.append(np.stack(d))
        dN, w, dN0 = np.stack(out), 1.0 / 24.0, None
    t = lambda v: None if v is None else torch.as_tensor(v, dtype=F64, device="cuda")  # noqa: E731
    return t(dN), w, t(dN0)


def _geometry(case, Xe):
    """Shape-function gradients (ne, ngp, nnode, 3), volumes, centre gradients."""
    dN, w, dN0 = _tables(case["etype"])
    J = torch.einsum("ean,gai->egni", Xe, dN)
    G = torch.einsum("gai,egij->egaj", dN, torch.linalg.inv(J))
    G0 = None
    if dN0 is not None:
        G0 = torch.einsum("ai,eij->eaj", dN0, torch.linalg.inv(torch.einsum("ean,ai->eni", Xe, dN0)))
    return G, w * torch.linalg.det(J), G0


def _strain(G, G0, ue):
    H = torch.einsum("eac,egaj->egcj", ue, G)
    eye = torch.eye(3, dtype=F64, device=H.device)
    if G0 is not None:
        tr0 = torch.einsum("eac,eac->e", ue, G0)
        H = H + ((tr0[:, None] - H.diagonal(dim1=-2, dim2=-1).sum(-1)) / 3)[..., None, None] * eye
    return 0.5 * (H + H.transpose(-1, -2))


def _radial_return(case, eps, state):
    """Stress, new state and (n, c1, c2) of the consistent tangent."""
    eye = torch.eye(3, dtype=F64, device=eps.device)
    tr = eps.diagonal(dim1=-2, dim2=-1).sum(-1)
    if state is None:
        return LAM * tr[..., None, None] * eye + 2 * MU * eps, None, None
    hk = HARDENING[case["material"]][1]
    mat = _material(case)
    ep, sy = (torch.as_tensor(v, dtype=F64, device=eps.device) for v in (mat.ep_tab, mat.sy_tab))
    slopes = (sy[1:] - sy[:-1]) / (ep[1:] - ep[:-1])

    def table(x):
        i = torch.searchsorted(ep, x.contiguous(), right=True).clamp(1, len(ep) - 1) - 1
        s = torch.where((x < ep[0]) | (x > ep[-1]), torch.zeros_like(x), slopes[i])
        return sy[i] + (x.clamp(ep[0], ep[-1]) - ep[i]) * slopes[i], s

    e0, a0, be = state[..., :9].unflatten(-1, (3, 3)), state[..., 9], state[..., 10:].unflatten(-1, (3, 3))
    ee = eps - e0
    tre = ee.diagonal(dim1=-2, dim2=-1).sum(-1)
    s_tr = 2 * MU * (ee - tre[..., None, None] / 3 * eye)
    xi = s_tr - be
    q = math.sqrt(1.5) * torch.sqrt((xi * xi).sum((-1, -2)) + 1e-30)
    plastic = q > table(a0)[0]
    dg, slope = torch.zeros_like(q), torch.zeros_like(q)
    for _ in range(25):
        syv, slope = table(a0 + dg)
        dg = (dg + (q - (3 * MU + hk) * dg - syv) / (3 * MU + hk + slope)).clamp(min=0)
    dg = torch.where(plastic, dg, torch.zeros_like(dg))
    n = 1.5 * xi / (q + 1e-30)[..., None, None]
    d = dg[..., None, None]
    sig = s_tr - 2 * MU * d * n + BULK * tre[..., None, None] * eye
    new = torch.cat([(e0 + d * n).flatten(-2), (a0 + dg)[..., None], (be + 2.0 / 3.0 * hk * d * n).flatten(-2)], -1)
    c1 = torch.where(plastic, 1 - 3 * MU * dg / q, torch.ones_like(q))
    c2 = torch.where(plastic, 4 * MU * MU * (dg / q - 1 / (3 * MU + hk + slope)), torch.zeros_like(q))
    return sig, new, (n, c1, c2)


def _stress_force(case, Xd, cd, u, state):
    """Per element: nodal forces, new states, averaged stress, Mises, averaged plastic strain."""
    G, vol, G0 = _geometry(case, Xd[cd])
    sig, new, _ = _radial_return(case, _strain(G, G0, u.reshape(-1, 3)[cd]), state)
    p = sig.diagonal(dim1=-2, dim2=-1).sum(-1) / 3
    if G0 is None:
        fe = torch.einsum("eg,egcj,egaj->eac", vol, sig, G)
    else:
        dev = sig - p[..., None, None] * torch.eye(3, dtype=F64, device=sig.device)
        fe = torch.einsum("eg,egcj,egaj->eac", vol, dev, G) + (vol * p).sum(1)[:, None, None] * G0
    V = vol.sum(1)
    S = (vol[..., None, None] * sig).sum(1) / V[:, None, None]
    dev = S - S.diagonal(dim1=-2, dim2=-1).sum(-1)[:, None, None] / 3 * torch.eye(3, dtype=F64, device=S.device)
    peeq = torch.zeros_like(V) if new is None else (vol * new[..., 9]).sum(1) / V
    return fe, new, dict(S=S, MISES=torch.sqrt(1.5 * (dev * dev).sum((-1, -2))), PEEQ=peeq)


def _element_matrices(case, Xd, cd, u, state, chunk=8192):
    """Element tangents by chunks: sum over Gauss points of vol dE_i : C : dE_j."""
    out = []
    ue = u.reshape(-1, 3)
    eye = torch.eye(3, dtype=F64, device=Xd.device)
    for k in range(0, len(cd), chunk):
        c = cd[k:k + chunk]
        st = None if state is None else state[k:k + chunk]
        G, vol, G0 = _geometry(case, Xd[c])
        ne, ngp, nnode, _ = G.shape
        H = torch.einsum("ck,egaj->egakcj", eye, G)                    # gradient of unit displacement k at node a
        if G0 is not None:
            H = H + torch.einsum("egak,cj->egakcj", (G0[:, None] - G) / 3, eye)
        B = (0.5 * (H + H.transpose(-1, -2))).reshape(ne, ngp, 3 * nnode, 3, 3)
        tr = B.diagonal(dim1=-2, dim2=-1).sum(-1)
        dS = 2 * MU * B + LAM * tr[..., None, None] * eye
        if st is not None:
            _, _, (n, c1, c2) = _radial_return(case, _strain(G, G0, ue[c]), st)
            dev = B - tr[..., None, None] / 3 * eye
            nb = torch.einsum("egcj,egicj->egi", n, dev)
            dS = BULK * tr[..., None, None] * eye + 2 * MU * c1[..., None, None, None] * dev \
                + (c2[..., None] * nb)[..., None, None] * n[:, :, None]
        wB = (vol[..., None, None, None] * B).flatten(-2)
        out.append(torch.matmul(wB.transpose(1, 2).flatten(2), dS.flatten(-2).transpose(1, 2).flatten(2).transpose(1, 2)))
    return torch.cat(out)


def _assemble(cd, fe, nn):
    out = torch.zeros((nn,) + fe.shape[2:], dtype=F64, device="cuda")
    return out.index_add_(0, cd.reshape(-1), fe.flatten(0, 1))


def _times(K, cd, v, free, nn):
    """free K (free v) + (1 - free) v for v (ndof, k)."""
    k = v.shape[1]
    ve = (free[:, None] * v).reshape(nn, 3 * k)[cd].reshape(len(cd), -1, k)
    y = _assemble(cd, torch.matmul(K, ve).reshape(len(cd), cd.shape[1], 3 * k), nn).reshape(-1, k)
    return torch.where(free[:, None] > 0, y, v)


def _solve(K, cd, b, free, nn):
    """Jacobi-preconditioned conjugate gradients to the rounding level, with the
    residual recomputed and the iteration restarted until it no longer improves."""
    d = torch.diagonal(K, dim1=1, dim2=2).reshape(len(cd), -1, 3)
    dinv = torch.where(free > 0, 1.0 / _assemble(cd, d, nn).reshape(-1), torch.ones_like(free))[:, None]
    x, bn, best = torch.zeros_like(b), float(b.norm()), math.inf
    for _ in range(6):
        r = b - _times(K, cd, x, free, nn)
        rn = float(r.norm())
        if rn >= 0.3 * best or rn <= 1e-15 * bn:
            break
        best, dx, z = rn, torch.zeros_like(b), dinv * r
        p, rz = z.clone(), (r * z).sum()
        for it in range(6000):
            q = _times(K, cd, p, free, nn)
            al = rz / (p * q).sum()
            dx += al * p
            r -= al * q
            if it % 25 == 24 and float(r.norm()) <= 1e-9 * rn:
                break
            z = dinv * r
            rz, old = (r * z).sum(), rz
            p = z + (rz / old) * p
        x += dx
    return x


def exact(case, seed):
    X, c, size, Xd, cd, u, state = _fields(case, seed)
    nn, op = len(X), case["op"]
    if op in ("force", "stress"):
        fe, new, rec = _stress_force(case, Xd, cd, u, state)
        if op == "stress":
            return rec
        f = _assemble(cd, fe, nn).reshape(-1)
        return [f] if new is None else [f, new]
    K = _element_matrices(case, Xd, cd, u, state)
    if op == "tangent":
        return [K]
    free = torch.as_tensor(1.0 - _clamped(X), dtype=F64, device="cuda")
    if op == "solve":
        return _solve(K, cd, _tip_load(X, size, seed)[:, None], free, nn)[:, 0]
    dtype = DTYPES[case["dtype"]]
    if op == "product":
        v = torch.randn(3 * nn, dtype=dtype, device="cuda", generator=_gen(seed + 1)).to(F64)[:, None]
        return _times(K, cd, v, free if case["dtype"] == "f32" else torch.ones_like(free), nn)[:, 0]
    shape = (3 * nn, case["nrhs"]) if case["nrhs"] > 1 else (3 * nn,)
    v = torch.randn(shape, dtype=F64 if case["dtype"] == "f64" else torch.float32, device="cuda", generator=_gen(seed + 1))
    y = _times(K.to(dtype).to(F64), cd, v.to(F64).reshape(3 * nn, -1), free, nn)
    return y.reshape(shape)
