"""GPU: the plan writers of orders 2 and 4 over many steps of one warp.  A warp stages the
blocks it adds in a few slots and refills them while earlier reductions may still read
them, so each mesh here gives every resident warp several steps, most of them with bulk
groups of both elements, and an odd last element.  Against the FP64 oracle at 1e-12, in
both layouts, as one dependency-ordered launch and band by band; deterministic."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# resident warps: 148 SMs x 16 at order 2, x 12 at order 4; a colour holds a quarter of the elements
CASES = [(2, "nonlinear", 141, 139), (2, "nonlinear", 251, 239), (2, "linear", 251, 239), (4, "linear", 171, 169)]


@pytest.mark.parametrize("order,strain,nx,ny", CASES)
def test_many_steps_match_oracle(fem, orc, cuda, order, strain, nx, ny):
    import torch
    m = fem.square_mesh(nx, ny, order, 1.0, 1.0, 0.15, seed=17 + order)
    plan = fem.Plan(order, m.num_nodes, m.conn_ptr, m.conn)
    d = fem.DeviceMesh(m, cuda)
    rowp, cols = plan.pattern()
    orc.set_extended_j(True)  # the plain sum of J cancels by 1 / h
    try:
        R0, A0 = orc.assemble(m, orc.element_bsr_map(m.conn_ptr, m.conn, m.nodes_per_element, rowp, cols), cols.size,
                              strain=strain)
    finally:
        orc.set_extended_j(False)
    scale = np.abs(R0).max(), np.abs(A0).max()
    R0, A0 = torch.from_numpy(R0).to(cuda).reshape(-1), torch.from_numpy(A0).to(cuda).reshape(-1)

    def outputs():
        return (torch.full((m.num_nodes * 2,), float("nan"), dtype=torch.float64, device=cuda),
                torch.full((plan.nnzb * 4,), float("nan"), dtype=torch.float64, device=cuda))

    def check(res, mat, what):
        assert not torch.isnan(res).any() and not torch.isnan(mat).any(), what
        assert float((res - R0).abs().max()) <= 1e-12 * scale[0], what
        assert float((mat - A0).abs().max()) <= 1e-12 * scale[1], what

    try:
        for layout in ("pairs", "colours"):
            plan.set_layout(layout)
            res, mat = outputs()
            plan.assemble(d.states, d.coords, m.E, m.nu, m.t, res, mat, strain=strain)
            check(res, mat, layout)
            for _ in range(3):
                again = outputs()
                plan.assemble(d.states, d.coords, m.E, m.nu, m.t, *again, strain=strain)
                assert torch.equal(again[0], res) and torch.equal(again[1], mat), layout
            hs = torch.from_numpy(np.ascontiguousarray(m.states).reshape(-1)).pin_memory()
            hr = torch.empty(m.num_nodes * 2, dtype=torch.float64).pin_memory()
            again = outputs()
            plan.assemble_host(hs, torch.zeros_like(d.states), d.coords, m.E, m.nu, m.t, hr, *again, strain=strain, bands=5,
                               timed=True)
            assert torch.equal(hr, res.cpu()) and torch.equal(again[1], mat), layout
        plan.set_schedule()
        again = outputs()
        plan.assemble(d.states, d.coords, m.E, m.nu, m.t, *again, strain=strain)
        assert plan.wait_status() == 0
        check(*again, "ordered")
    finally:
        plan.close()
