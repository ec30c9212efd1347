"""GPU: the strip layout of order-3 plans (a warp assembles a strip of right
neighbours; an edge's blocks are carried to the next element, a strip's first edge is
completed by a halo element).  Against the FP64 oracle at 1e-12 and the colour layout to
rounding, in every mode, for chains whose length leaves every remainder of a strip,
meshes closed along the other axis (odd ring: three colours) and scrambled numbering;
deterministic; equal to the host-buffer assembly bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODES = [("fp64", "linear", True, True), ("fp64", "linear", True, False), ("fp64", "linear", False, True),
         ("fp64", "nonlinear", True, True), ("fp64", "nonlinear", True, False), ("fp64", "nonlinear", False, True),
         ("mixed", "linear", True, True), ("mixed", "linear", False, True)]


def _scramble(fem, m, seed):
    rng = np.random.default_rng(seed)
    nn = (m.order + 1) ** 2
    pe, pn = rng.permutation(m.num_elements), rng.permutation(m.num_nodes)
    inv = np.empty_like(pn)
    inv[pn] = np.arange(pn.size)
    conn = pn[m.conn.reshape(-1, nn)[pe]].reshape(-1).astype(np.int32)
    return fem.Mesh(m.order, m.coords[inv], np.arange(0, conn.size + 1, nn, dtype=np.int32), conn, m.states[inv],
                    m.E, m.nu, m.t)


def _mirror(m):
    """Every element's local nodes mirrored along x: all det J negative."""
    nn, p1 = (m.order + 1) ** 2, m.order + 1
    a = np.arange(nn)
    m.conn = np.ascontiguousarray(m.conn.reshape(-1, nn)[:, (a // p1) * p1 + (p1 - 1 - a % p1)].reshape(-1))
    return m


MESHES = {f"chain{nx}": (lambda f, nx=nx: f.square_mesh(nx, -(-16500 // nx), 3, 1.0, 1.0, 0.15, seed=nx))
          for nx in (4, 8, 9, 14, 15, 16, 17, 18, 19, 128)}
MESHES.update({f"small{nx}x{ny}": (lambda f, nx=nx, ny=ny: f.square_mesh(nx, ny, 3, 1.0, 1.0, 0.15, seed=nx))
               for nx, ny in ((4, 1), (5, 2), (11, 8), (43, 37), (90, 91))})
MESHES["ring"] = lambda f: f.annulus_mesh(17, 981, 3, seed=81)
MESHES["scrambled"] = lambda f: _scramble(f, f.square_mesh(129, 131, 3, 1.0, 1.0, 0.15, seed=82), 82)
MESHES["negative_det"] = lambda f: _mirror(f.square_mesh(30, 560, 3, 1.0, 1.0, 0.15, seed=83))


def _run(cuda, m, plan, d, prec, strain, res_on, mat_on):
    import torch
    res = torch.full((m.num_nodes * 2,), float("nan"), dtype=torch.float64, device=cuda) if res_on else None
    mat = torch.full((plan.nnzb * 4,), float("nan"), dtype=torch.float64, device=cuda) if mat_on else None
    plan.assemble(d.states, d.coords, m.E, m.nu, m.t, res, mat, precision=prec, strain=strain)
    return res, mat


@pytest.mark.parametrize("name", list(MESHES))
def test_strips_match_oracle_and_colours(fem, orc, cuda, name):
    import torch
    m = MESHES[name](fem)
    plan = fem.Plan(3, m.num_nodes, m.conn_ptr, m.conn)
    d = fem.DeviceMesh(m, cuda)
    try:
        assert plan.layout()[0] == "pairs" and plan.strips()[0] > 0 and plan.launches() <= 3
        got = {k: _run(cuda, m, plan, d, *k) for k in MODES}
        again = _run(cuda, m, plan, d, *MODES[0])
        assert all(torch.equal(x, y) for x, y in zip(again, got[MODES[0]]))
        rowp, cols = plan.pattern()
        orc.set_extended_j(True)  # thin elements: the plain sum of J cancels by 1 / h (up to 4000 here)
        try:
            R0, A0 = orc.assemble(m, orc.element_bsr_map(m.conn_ptr, m.conn, 16, rowp, cols), cols.size)
        finally:
            orc.set_extended_j(False)
        for x, y in zip(got[MODES[0]], (R0, A0)):
            x = x.cpu().numpy()
            assert not np.isnan(x).any() and np.abs(x - y).max() <= 1e-12 * np.abs(y).max()
        plan.set_layout("colours")
        assert plan.launches() == plan.num_colours
        for k in MODES:
            for x, y in zip(got[k], _run(cuda, m, plan, d, *k)):
                if x is not None:
                    assert not torch.isnan(x).any(), k
                    assert (x - y).abs().max() <= (1e-6 if k[0] == "mixed" else 1e-14) * y.abs().max(), k
    finally:
        plan.close()


@pytest.mark.parametrize("name,precision,strain,bands", [("chain128", "fp64", "linear", 8), ("chain9", "mixed", "linear", 5),
                                                         ("ring", "fp64", "nonlinear", 32), ("scrambled", "fp64", "linear", 4)])
def test_strips_host_assembly_equals_device_assembly(fem, cuda, name, precision, strain, bands):
    import torch
    m = MESHES[name](fem)
    plan = fem.Plan(3, m.num_nodes, m.conn_ptr, m.conn)
    d = fem.DeviceMesh(m, cuda)
    res0, mat0 = _run(cuda, m, plan, d, precision, strain, True, True)
    h_states = torch.from_numpy(np.ascontiguousarray(m.states).reshape(-1)).pin_memory()
    h_res = torch.full((m.num_nodes * 2,), float("nan"), dtype=torch.float64).pin_memory()
    states, res, mat = torch.zeros_like(d.states), torch.full_like(res0, float("nan")), torch.full_like(mat0, float("nan"))
    plan.assemble_host(h_states, states, d.coords, m.E, m.nu, m.t, h_res, res, mat, precision=precision, strain=strain,
                       bands=bands, timed=True)
    torch.cuda.synchronize()
    assert torch.equal(h_res, res0.cpu()) and torch.equal(mat, mat0)
    plan.close()
