"""GPU: which order-3 plans run strips.  Meshes whose elements do not all have their axes
along one grid: elements turned at random, blocks with crossed axes.  Their chains of right
neighbours cross and need many colours; such a plan runs its pairs (or colours), unless it
is large and up to seven colours do, where FP64 runs strips and MIXED the pairs.  Every
mode against the colour layout to rounding, the small ones against the FP64 oracle at
1e-12, host-buffer assembly bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _turn(m, mask, quarters):
    """The masked elements' local axes turned by quarter turns (det J stays positive)."""
    g = m.conn.reshape(-1, m.order + 1, m.order + 1).copy()
    for q in (1, 2, 3):
        i = np.nonzero(mask & (quarters == q))[0]
        g[i] = np.rot90(g[i], q, axes=(1, 2))
    m.conn = np.ascontiguousarray(g.reshape(-1))
    return m


def _turned(fem, nx, ny, fraction, seed):
    r = np.random.default_rng(seed)
    return _turn(fem.square_mesh(nx, ny, 3, 1.0, 1.0, 0.15, seed=seed), r.random(nx * ny) < fraction,
                 r.integers(1, 4, nx * ny))


def _crossed(fem, nx, ny, w, seed):
    """Blocks w elements wide, every other one with its axes crossed."""
    ex, ey = (a.reshape(-1) for a in np.meshgrid(np.arange(nx), np.arange(ny)))
    return _turn(fem.square_mesh(nx, ny, 3, 1.0, 1.0, 0.15, seed=seed), (ex // w + ey // w) % 2 == 1, np.ones(nx * ny, int))


MODES = [("fp64", "linear", True, True), ("fp64", "linear", False, True), ("fp64", "linear", True, False),
         ("fp64", "nonlinear", True, True), ("mixed", "linear", True, True)]


def _run(cuda, m, plan, d, prec, strain, res_on, mat_on):
    import torch
    res = torch.full((m.num_nodes * 2,), float("nan"), dtype=torch.float64, device=cuda) if res_on else None
    mat = torch.full((plan.nnzb * 4,), float("nan"), dtype=torch.float64, device=cuda) if mat_on else None
    plan.assemble(d.states, d.coords, m.E, m.nu, m.t, res, mat, precision=prec, strain=strain)
    return res, mat


def _check(fem, cuda, m, plan, d):
    """Every mode against the colour layout; host assembly bit for bit; the default's FP64 result."""
    import torch
    got = {k: _run(cuda, m, plan, d, *k) for k in MODES}
    hs = torch.from_numpy(np.ascontiguousarray(m.states).reshape(-1)).pin_memory()
    for k in (MODES[0], MODES[-1]):
        hr = torch.empty(m.num_nodes * 2, dtype=torch.float64).pin_memory()
        res, mat = torch.full_like(got[k][0], float("nan")), torch.full_like(got[k][1], float("nan"))
        plan.assemble_host(hs, torch.zeros_like(d.states), d.coords, m.E, m.nu, m.t, hr, res, mat, precision=k[0], bands=6,
                           timed=True)
        assert torch.equal(hr, got[k][0].cpu()) and torch.equal(mat, got[k][1]), k
    plan.set_layout("colours")
    for k in MODES:
        for x, y in zip(got[k], _run(cuda, m, plan, d, *k)):
            if x is not None:
                assert not torch.isnan(x).any(), k
                assert (x - y).abs().max() <= (1e-6 if k[0] == "mixed" else 1e-14) * y.abs().max(), k
    plan.set_layout("pairs")
    return got[MODES[0]]


@pytest.mark.parametrize("make", [lambda f: _turned(f, 43, 37, 0.05, 5), lambda f: _turned(f, 97, 89, 0.05, 6),
                                  lambda f: _turned(f, 97, 89, 0.15, 7), lambda f: _crossed(f, 46, 40, 23, 8),
                                  lambda f: _crossed(f, 128, 96, 64, 9), lambda f: _crossed(f, 120, 96, 8, 10)],
                         ids=["small-turned", "turned5", "turned15", "small-crossed", "crossed", "blocks8"])
def test_crossing_chains_run_no_strips(fem, orc, cuda, make):
    m = make(fem)
    plan = fem.Plan(3, m.num_nodes, m.conn_ptr, m.conn)
    d = fem.DeviceMesh(m, cuda)
    try:
        assert plan.strips() == (0, 0)
        assert plan.launches() == (plan.layout()[2] if m.num_elements > 7104 else plan.num_colours)
        R, A = _check(fem, cuda, m, plan, d)
        rowp, cols = plan.pattern()
        orc.set_extended_j(True)
        try:
            R0, A0 = orc.assemble(m, orc.element_bsr_map(m.conn_ptr, m.conn, 16, rowp, cols), cols.size)
        finally:
            orc.set_extended_j(False)
        for x, y in ((R, R0), (A, A0)):
            assert np.abs(x.cpu().numpy() - y).max() <= 1e-12 * np.abs(y).max()
    finally:
        plan.close()


@pytest.mark.parametrize("make", [lambda f: _crossed(f, 461, 457, 230, 11), lambda f: _turned(f, 461, 457, 0.02, 12)],
                         ids=["crossed", "turned2"])
def test_large_crossing_chains(fem, cuda, make):
    m = make(fem)
    plan = fem.Plan(3, m.num_nodes, m.conn_ptr, m.conn)
    d = fem.DeviceMesh(m, cuda)
    try:
        strips, colours = plan.strips()
        assert strips > 0 and 4 <= colours <= 7
        assert plan.launches() == colours and plan.launches(precision="mixed") == plan.layout()[2]
        _check(fem, cuda, m, plan, d)
    finally:
        plan.close()
