"""Performance cases of the assembly library: what a finite-element program has it do.

A case is one assembly of a plane-stress quadrilateral mesh through the public Python
interface (`Plan`, `Batch`, `run_residual_kernel`, `run_jacobian_kernel`), at the sizes
of this repository's own workloads (`mesh.py`, `bench.py`) and their ragged
neighbours.  Meshes are structured, with the node placement of `mesh.py`: element
vertices perturbed by up to 0.15-0.2 h, higher-order nodes at the cosine knots of the
element's bilinear map, displacements in [-1e-3, 1e-3].  Coordinates, displacements
and material come from the seed.

Kinds:
  plan      Newton iteration: residual and Jacobian from an assembly plan
  residual  residual alone from the plan (line search, load step, explicit dynamics)
  driver    the reference driver's sequence on its own data format: zero the outputs,
            run the residual kernel, run the Jacobian kernel through the element map
  batch     many small meshes of mixed orders, one captured graph
"""
import math

import numpy as np
import torch

import fem_pkg

DEV = "cuda"
THICK = 1.0

# 1D Gauss points and weights (order + 1 of them) and the monomial coefficients,
# highest power first, of the 1D basis on the cosine knots: the element's definition.
GAUSS = {
    1: ([-0.577350269189626, 0.577350269189626], [1.0, 1.0]),
    2: ([-0.774596669241483, 0.0, 0.774596669241483], [5.0 / 9.0, 8.0 / 9.0, 5.0 / 9.0]),
    3: ([-0.861136311594053, -0.339981043584856, 0.339981043584856, 0.861136311594053],
        [0.347854845137454, 0.652145154862546, 0.652145154862546, 0.347854845137454]),
    4: ([-0.906179845938664, -0.538469310105683, 0.0, 0.538469310105683, 0.906179845938664],
        [0.236926885056189, 0.478628670499366, 0.568888888888889, 0.478628670499366, 0.236926885056189]),
}
BASIS = {
    1: [[-0.5, 0.5], [0.5, 0.5]],
    2: [[0.5, -0.5, 0.0], [-1.0, 0.0, 1.0], [0.5, 0.5, 0.0]],
    3: [[-2.0 / 3.0, 2.0 / 3.0, 1.0 / 6.0, -1.0 / 6.0], [4.0 / 3.0, -2.0 / 3.0, -4.0 / 3.0, 2.0 / 3.0],
        [-4.0 / 3.0, -2.0 / 3.0, 4.0 / 3.0, 2.0 / 3.0], [2.0 / 3.0, 2.0 / 3.0, -1.0 / 6.0, -1.0 / 6.0]],
    4: [[1.0, -1.0, -0.5, 0.5, 0.0], [-2.0, 1.41421356237310, 2.0, -1.41421356237310, 0.0],
        [2.0, 0.0, -3.0, 0.0, 1.0], [-2.0, -1.41421356237310, 2.0, 1.41421356237310, 0.0],
        [1.0, 1.0, -0.5, -0.5, 0.0]],
}


def _case(name, kind, order, nx, ny, shape="square", precision="fp64", strain="linear"):
    return {"name": name, "kind": kind, "order": order, "nx": nx, "ny": ny, "shape": shape, "precision": precision,
            "strain": strain}


def listed():
    return [
        # the smallest call: one launch over 4096 bilinear elements, bound by latency
        _case("plan_p1_64", "plan", 1, 64, 64),
        # the largest bilinear mesh of the benchmark, one Newton iteration
        _case("plan_p1_2048", "plan", 1, 2048, 2048),
        # curved geometry, periodic numbering: the benchmark's annulus
        _case("plan_p2_annulus", "plan", 2, 512, 2048, "annulus"),
        # a small ragged mesh of the server's and batch's lower range, alone on the GPU
        _case("plan_p3_small", "plan", 3, 43, 37),
        # the headline workload, and the largest case: 18.9 M unknowns, 7.55 GB of matrix
        _case("plan_p3_1024", "plan", 3, 1024, 1024),
        # the highest order, ragged sides
        _case("plan_p4_ragged", "plan", 4, 381, 379),
        # reduced-precision element stiffness
        _case("mixed_p3", "plan", 3, 515, 509, precision="mixed"),
        # finite strain: a tangent that depends on the state
        _case("nonlinear_p3", "plan", 3, 400, 397, strain="nonlinear"),
        # residual evaluations of a line search
        _case("residual_p3", "residual", 3, 600, 590),
        # the reference driver's calls on the reference's data format
        _case("driver_p2", "driver", 2, 501, 500),
        _case("driver_p4", "driver", 4, 200, 201),
        # 12 meshes of 1e3 to 6e4 elements, every order, one graph launch
        {"name": "batch_mixed", "kind": "batch", "meshes": 12, "most": 60000, "mix": 4, "precision": "fp64"},
    ]


def draw(rng):
    def log_size(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["plan", "plan", "plan", "residual", "driver", "batch"])
    if kind == "batch":
        return {"kind": "batch", "meshes": rng.randint(4, 24), "most": int(log_size(4e3, 8e4)), "mix": rng.randint(0, 10**6),
                "precision": "fp64"}
    order = rng.randint(1, 4)
    # up to a quarter of a million elements, a million bilinear ones
    count = log_size(1e3, {1: 1e6, 2: 4e5, 3: 2.5e5, 4: 1.2e5}[order])
    aspect = log_size(0.25, 4.0)
    nx = max(3, int(round(math.sqrt(count * aspect))))
    ny = max(3, int(round(count / nx)))
    shape = rng.choice(["square", "square", "annulus"])
    precision, strain = "fp64", "linear"
    if kind == "plan" and order >= 2:
        u = rng.random()
        if u < 0.2:
            precision = "mixed"
        elif u < 0.4:
            strain = "nonlinear"
    c = _case("", kind, order, nx, ny, shape, precision, strain)
    del c["name"]
    return c


def batch_parts(case):
    """The meshes of a batch case: log-uniform element counts, orders 1 to 4."""
    r = np.random.default_rng(case["mix"])
    parts = []
    for i in range(case["meshes"]):
        count = math.exp(r.uniform(math.log(1e3), math.log(case["most"])))
        ny = max(3, int(round(math.sqrt(count))))
        parts.append({"kind": "plan", "order": 1 + i % 4, "nx": max(3, int(round(count / ny))), "ny": ny,
                      "shape": "square", "precision": case["precision"], "strain": "linear"})
    return parts


def _knots(p):
    k = -np.cos(np.pi / 2 * (2.0 * np.arange(p + 1) / p))
    k[0], k[-1] = -1.0, 1.0
    return (k + 1.0) / 2.0


def _axis(n_el, p):
    """(element, fraction within it) of the n_el * p + 1 nodes of one axis."""
    i = np.arange(n_el * p + 1)
    e = np.minimum(i // p, n_el - 1)
    return torch.from_numpy(e).to(DEV), torch.from_numpy(_knots(p)[i - e * p]).to(DEV)


def _conn(case):
    """Element connectivity (host, int32 [elements, nodes]) and the node count."""
    p, nx, ny = case["order"], case["nx"], case["ny"]
    wrap = case["shape"] == "annulus"
    nxn, nyn = nx * p + 1, ny * p + (0 if wrap else 1)
    a = np.arange(p + 1)
    i = (np.arange(nx)[:, None] * p + a[None, :]).astype(np.int32)
    j = (np.arange(ny)[:, None] * p + a[None, :]).astype(np.int32)
    if wrap:
        j %= nyn
    return (j[:, None, :, None] * nxn + i[None, :, None, :]).reshape(nx * ny, (p + 1) ** 2), nxn * nyn


def _inputs(case, seed):
    """Coordinates and displacements (device, float64 [nodes, 2]), E and nu."""
    p, nx, ny = case["order"], case["nx"], case["ny"]
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    r = np.random.default_rng(seed)
    E, nu = float(r.uniform(50e9, 210e9)), float(r.uniform(0.25, 0.35))

    def uniform(*shape):
        return 2.0 * torch.rand(*shape, dtype=torch.float64, device=DEV, generator=g) - 1.0

    ex, fx = _axis(nx, p)
    ey, fy = _axis(ny, p)
    if case["shape"] == "annulus":
        ey, fy = ey[:-1], fy[:-1]
        rad = (1.0 + (ex + fx) / nx)[None, :].expand(ey.numel(), -1)
        th = (2.0 * math.pi * (ey + fy) / ny)[:, None].expand(-1, ex.numel())
        xy = torch.stack([rad * torch.cos(th), rad * torch.sin(th)], -1)
        wave = 1e-3 * torch.sin(int(r.integers(1, 9)) * th) * rad
        u = torch.stack([wave, wave], -1) + 1e-5 * uniform(*xy.shape)
    else:
        v = torch.empty(ny + 1, nx + 1, 2, dtype=torch.float64, device=DEV)
        v[:, :, 0] = torch.linspace(0.0, 10.0, nx + 1, dtype=torch.float64, device=DEV)[None, :]
        v[:, :, 1] = torch.linspace(0.0, 10.0, ny + 1, dtype=torch.float64, device=DEV)[:, None]
        h = torch.tensor([10.0 / nx, 10.0 / ny], dtype=torch.float64, device=DEV)
        v[1:-1, 1:-1] += 0.15 * h * uniform(ny - 1, nx - 1, 2)
        fx, fy = fx[None, :, None], fy[:, None, None]
        lo, hi = v[ey], v[ey + 1]
        xy = (1 - fy) * ((1 - fx) * lo[:, ex] + fx * lo[:, ex + 1]) + fy * ((1 - fx) * hi[:, ex] + fx * hi[:, ex + 1])
        u = 1e-3 * uniform(*xy.shape)
    return xy.reshape(-1, 2).contiguous(), u.reshape(-1, 2).contiguous(), E, nu


def _mesh_state(fem, case, seed):
    conn, nodes = _conn(case)
    nn = conn.shape[1]
    ptr = np.arange(conn.shape[0] + 1, dtype=np.int32) * nn
    xy, u, E, nu = _inputs(case, seed)
    s = {"case": case, "xy": xy, "u": u, "E": E, "nu": nu, "elements": conn.shape[0]}
    if case["kind"] == "driver":
        rowp, cols = fem.build_bsr_pattern(nodes, ptr, conn.reshape(-1))
        emap = fem.build_element_bsr_map(ptr, conn.reshape(-1), nn, rowp, cols)
        s["ptr"], s["conn"] = torch.from_numpy(ptr).to(DEV), torch.from_numpy(conn.reshape(-1)).to(DEV)
        s["map"] = torch.from_numpy(emap).to(DEV)
        blocks = int(cols.size)
    else:
        s["plan"] = fem.Plan(case["order"], nodes, ptr, conn.reshape(-1))
        blocks = s["plan"].nnzb
    s["res"] = torch.zeros(2 * nodes, dtype=torch.float64, device=DEV)
    if case["kind"] != "residual":
        s["mat"] = torch.zeros(4 * blocks, dtype=torch.float64, device=DEV)
    return s


def prepare(case, seed):
    fem = fem_pkg.load()
    if case["kind"] != "batch":
        s = _mesh_state(fem, case, seed)
        s["fem"] = fem
        return s
    parts = [_mesh_state(fem, c, seed * 64 + i) for i, c in enumerate(batch_parts(case))]
    batch = fem.Batch([q["plan"] for q in parts])
    for i, q in enumerate(parts):
        batch.bind(i, q["u"], q["xy"], q["E"], q["nu"], THICK, q["res"], q["mat"])
    batch.capture(precision=case["precision"])
    return {"case": case, "parts": parts, "batch": batch}


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].replay()
        return [[q["res"], q["mat"]] for q in state["parts"]]
    xy, u, E, nu, res = state["xy"], state["u"], state["E"], state["nu"], state["res"]
    if case["kind"] == "residual":
        state["plan"].assemble(u, xy, E, nu, THICK, res)
        return [res]
    mat = state["mat"]
    if case["kind"] == "plan":
        state["plan"].assemble(u, xy, E, nu, THICK, res, mat, precision=case["precision"], strain=case["strain"])
        return [res, mat]
    fem = state["fem"]
    mesh = (case["order"], state["ptr"], state["conn"], state["elements"], u, xy, E, nu, THICK)
    res.zero_()
    fem.run_residual_kernel(*mesh, res, timed=False)
    mat.zero_()
    fem.run_jacobian_kernel(*mesh, state["map"], None, mat, timed=False)
    return [res, mat]


def work(case):
    if case["kind"] == "batch":
        w = [work(c) for c in batch_parts(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    p, nx, ny = case["order"], case["nx"], case["ny"]
    n = (p + 1) ** 2
    wrap = case["shape"] == "annulus"
    nodes = (nx * p + 1) * (ny * p + (0 if wrap else 1))
    blocks = (nx * (p * p + 2 * p) + 1) * (ny * (p * p + 2 * p) + (0 if wrap else 1))
    elements = nx * ny
    size = 32 * nodes + 4 * n * elements + 16 * nodes  # coordinates and states, connectivity, residual
    # per quadrature point: J and grad u, the nodal gradients, the residual
    flops = n * (16 * n + 6 * n + 8 * n + 60)
    if case["kind"] != "residual":
        size += 32 * blocks
        if case["kind"] == "driver":
            size += 4 * n * n * elements  # the element map
        # the symmetric element matrix: (2n)(2n + 1)/2 entries of n products each
        flops += n * 2 * n * (2 * n + 1) * (2 if case["strain"] == "nonlinear" else 1)
    return {"bytes": float(size), "flops": float(flops * elements)}


def _table(p):
    """dN [points, nodes, 2], its sum over the nodes [points, 2] (zero but for the
    rounding of the table) and the quadrature weights, on the device."""
    gp, gw = GAUSS[p]
    N = np.array([[np.polyval(c, x) for c in BASIS[p]] for x in gp])
    D = np.array([[np.polyval(np.polyder(np.array(c)), x) for c in BASIS[p]] for x in gp])
    n = (p + 1) ** 2
    dx = (N[:, None, :, None] * D[None, :, None, :]).reshape(n, n)  # q = qy (p + 1) + qx, a likewise
    dy = (D[:, None, :, None] * N[None, :, None, :]).reshape(n, n)
    w = (np.array(gw)[:, None] * np.array(gw)[None, :]).reshape(-1)
    dN = np.stack([dx, dy], -1)
    total = np.array([[math.fsum(dN[q, :, d]) for d in range(2)] for q in range(n)])
    return tuple(torch.from_numpy(v).to(DEV) for v in (dN, total, w))


def _exact_mesh(case, seed):
    conn, nodes = _conn(case)
    xy, u, E, nu = _inputs(case, seed)
    dN, total, w = _table(case["order"])
    c = torch.from_numpy(conn).to(DEV).long()
    nE, nn = conn.shape
    mu = 0.5 * E / (1.0 + nu)
    lam = 2.0 * mu * nu / (1.0 - nu)
    eye = torch.eye(2, dtype=torch.float64, device=DEV)
    res = torch.zeros(nodes, 2, dtype=torch.float64, device=DEV)
    jac = case["kind"] != "residual"
    step = max(1, int(6e7) // (4 * nn * nn))
    if jac:
        keys = torch.empty(0, dtype=torch.int64, device=DEV)
        for e0 in range(0, nE, 4 * step):
            k = c[e0:e0 + 4 * step]
            k = torch.unique((k[:, :, None] * nodes + k[:, None, :]).reshape(-1))
            keys = torch.cat([keys, k])
        keys = torch.unique(keys)
        mat = torch.zeros(keys.numel(), 4, dtype=torch.float64, device=DEV)
    for e0 in range(0, nE, step):
        k = c[e0:e0 + step]
        X = xy[k]
        J = torch.einsum("eai,qaj->eqij", X - X[:, :1], dN) + torch.einsum("ei,qj->eqij", X[:, 0], total)
        det = J[..., 0, 0] * J[..., 1, 1] - J[..., 0, 1] * J[..., 1, 0]
        inv = torch.stack([torch.stack([J[..., 1, 1], -J[..., 0, 1]], -1),
                           torch.stack([-J[..., 1, 0], J[..., 0, 0]], -1)], -2) / det[..., None, None]
        G = torch.einsum("qaj,eqji->eqai", dN, inv)
        s = w * det * THICK
        g = torch.einsum("eai,eqaj->eqij", u[k], G)
        if case["strain"] == "nonlinear":
            F = eye + g
            C = 0.5 * (g + g.transpose(-1, -2) + g.transpose(-1, -2) @ g)
            S = 2 * mu * C + lam * (C[..., 0, 0] + C[..., 1, 1])[..., None, None] * eye
            P = F @ S
        else:
            P = mu * (g + g.transpose(-1, -2)) + lam * (g[..., 0, 0] + g[..., 1, 1])[..., None, None] * eye
        R = torch.einsum("eqij,eqaj->eai", s[..., None, None] * P, G)
        res.index_add_(0, k.reshape(-1), R.reshape(-1, 2))
        if not jac:
            continue
        if case["strain"] == "nonlinear":
            A = (torch.einsum("ik,eqln->eqilkn", eye, S) + mu * torch.einsum("eqin,eqkl->eqilkn", F, F)
                 + mu * torch.einsum("eqik,ln->eqilkn", F @ F.transpose(-1, -2), eye)
                 + lam * torch.einsum("eqil,eqkn->eqilkn", F, F))
            B = torch.einsum("eqilkn,eqbn->eqlikb", A * s[..., None, None, None, None], G)
            K = torch.einsum("eqal,eqlx->eax", G, B.reshape(*B.shape[:3], -1)).reshape(-1, nn, 2, 2, nn)
            K = K.permute(0, 1, 4, 2, 3)
        else:
            H = (s[..., None, None] * G).reshape(k.shape[0], nn, 2 * nn)
            M = (H.transpose(1, 2) @ G.reshape(k.shape[0], nn, 2 * nn)).reshape(-1, nn, 2, nn, 2).permute(0, 1, 3, 2, 4)
            K = lam * M + mu * M.transpose(-1, -2) + mu * (M[..., 0, 0] + M[..., 1, 1])[..., None, None] * eye
        pos = torch.searchsorted(keys, (k[:, :, None] * nodes + k[:, None, :]).reshape(-1))
        mat.index_add_(0, pos, K.reshape(-1, 4))
    return [res.reshape(-1), mat.reshape(-1)] if jac else [res.reshape(-1)]


def exact(case, seed):
    if case["kind"] == "batch":
        return [_exact_mesh(c, seed * 64 + i) for i, c in enumerate(batch_parts(case))]
    return _exact_mesh(case, seed)
