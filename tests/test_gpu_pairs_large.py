"""GPU: pair launches that run as pairs: more than 7104 elements, orders 2 to 4, at order 3
meshes without strips (rings closed along the local x axis, chains of two and three, elements
turned at random).  A warp's second element adds to the edge that its first one stored, and
both may add to what an earlier colour stored.  Against the colour layout to rounding, FP64
LINEAR and NONLINEAR against the FP64 oracle at 1e-12, deterministic, and path() at every
switch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _turn(m, mask, quarters):
    g = m.conn.reshape(-1, m.order + 1, m.order + 1).copy()
    for q in (1, 2, 3):
        i = np.nonzero(mask & (quarters == q))[0]
        g[i] = np.rot90(g[i], q, axes=(1, 2))
    m.conn = np.ascontiguousarray(g.reshape(-1))
    return m


def _square(f, nx, ny, p):
    return f.square_mesh(nx, ny, p, 1.0, 1.0, 0.15, seed=40 + p)


def _rings(f, p, nr, nth):
    """An annulus whose elements' local x axis runs around it."""
    m = f.annulus_mesh(nr, nth, p, seed=50 + p)
    return _turn(m, np.ones(m.num_elements, bool), np.ones(m.num_elements, int))


def _chains(f, n, w):
    """Chains of w elements: every other block w wide has its axes crossed."""
    ex, ey = (a.reshape(-1) for a in np.meshgrid(np.arange(n), np.arange(n)))
    return _turn(_square(f, n, n, 3), (ex // w + ey // w) % 2 == 1, np.ones(n * n, int))


def _random(f, nx, ny, p):
    r = np.random.default_rng(60)
    return _turn(_square(f, nx, ny, p), r.random(nx * ny) < 0.5, r.integers(1, 4, nx * ny))


MESHES = {
    "square_p2": lambda f: _square(f, 97, 89, 2),
    "annulus_p2": lambda f: f.annulus_mesh(24, 311, 2, seed=74),
    "random_p2": lambda f: _random(f, 121, 119, 2),
    "square_p4": lambda f: _square(f, 91, 83, 4),
    "random_p4": lambda f: _random(f, 87, 85, 4),
    "rings_p3": lambda f: _rings(f, 3, 20, 401),
    "chains2_p3": lambda f: _chains(f, 90, 2),
    "chains3_p3": lambda f: _chains(f, 99, 3),
    "random_p3": lambda f: _random(f, 130, 127, 3),
}


def _run(cuda, m, plan, d, prec, strain, res_on, mat_on):
    import torch
    res = torch.full((m.num_nodes * 2,), float("nan"), dtype=torch.float64, device=cuda) if res_on else None
    mat = torch.full((plan.nnzb * 4,), float("nan"), dtype=torch.float64, device=cuda) if mat_on else None
    plan.assemble(d.states, d.coords, m.E, m.nu, m.t, res, mat, precision=prec, strain=strain)
    return res, mat


@pytest.mark.parametrize("name", list(MESHES))
def test_pairs_match_oracle_and_colours(fem, orc, cuda, name):
    import torch
    m = MESHES[name](fem)
    plan = fem.Plan(m.order, m.num_nodes, m.conn_ptr, m.conn)
    d = fem.DeviceMesh(m, cuda)
    modes = [("fp64", "linear", True, True), ("fp64", "linear", True, False), ("fp64", "linear", False, True)]
    if m.order < 4:
        modes += [("fp64", "nonlinear", True, True), ("fp64", "nonlinear", True, False), ("mixed", "linear", True, True)]
    try:
        assert m.num_elements > 7104 and plan.layout()[0] == "pairs"
        for prec, strain, _, jac in modes:
            assert plan.path(strain, prec, jac) == "pairs"
        assert plan.launches() == plan.layout()[2]
        got = {k: _run(cuda, m, plan, d, *k) for k in modes}
        for _ in range(3):
            for k in modes:
                if k[3]:
                    assert torch.equal(_run(cuda, m, plan, d, *k)[1], got[k][1]), k
        plan.set_layout("colours")
        assert plan.path() == "colours"
        for k in modes:
            for x, y in zip(got[k], _run(cuda, m, plan, d, *k)):
                if x is not None:
                    assert not torch.isnan(x).any(), k
                    assert (x - y).abs().max() <= (1e-6 if k[0] == "mixed" else 1e-14) * y.abs().max(), k
        rowp, cols = plan.pattern()
        emap = orc.element_bsr_map(m.conn_ptr, m.conn, m.nodes_per_element, rowp, cols)
        orc.set_extended_j(True)
        try:
            for k in modes:
                if k[0] == "fp64" and k[2] and k[3]:
                    for x, y in zip(got[k], orc.assemble(m, emap, cols.size, strain=k[1])):
                        assert np.abs(x.cpu().numpy() - y).max() <= 1e-12 * np.abs(y).max(), k
        finally:
            orc.set_extended_j(False)
        plan.set_layout("pairs")
        assert plan.path() == "pairs"
        plan.set_schedule()
        assert plan.path() == "ordered" and plan.launches() == 1
    finally:
        plan.close()


def test_path_of_other_plans(fem, cuda):
    def path(m, *args):
        plan = fem.Plan(m.order, m.num_nodes, m.conn_ptr, m.conn)
        try:
            return plan.path(*args)
        finally:
            plan.close()

    assert path(fem.square_mesh(4, 4, 1)) == "rows" and path(fem.square_mesh(4, 4, 1), "nonlinear") == "colours"
    assert path(fem.square_mesh(9, 9, 2)) == "colours" and path(fem.square_mesh(9, 9, 4)) == "colours"
    s = fem.square_mesh(9, 9, 3)
    assert path(s) == "strips" and path(s, "linear", "mixed") == "strips"
    assert path(s, "linear", "fp64", False) == "colours" and path(s, "nonlinear") == "colours"
