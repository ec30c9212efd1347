"""GPU: material and thickness of either sign, or zero, at every order: the kernels fold mu
and t into the gradients as a square root and carry the sign apart.  Plans (residual +
Jacobian, residual alone) and the drop-in calls against the FP64 oracle at 1e-12."""
import dataclasses

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E,t", [(70e9, -0.5), (-70e9, 2.0), (-70e9, -1.0), (70e9, 0.0), (0.0, 1.0)])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_signs(fem, orc, cuda, order, E, t):
    import torch
    m = dataclasses.replace(fem.square_mesh(9, 5, order, 1.0, 1.0, 0.15, seed=40 + order), E=E, t=t)
    plan = fem.Plan(order, m.num_nodes, m.conn_ptr, m.conn)
    rowp, cols = plan.pattern()
    emap = fem.build_element_bsr_map(m.conn_ptr, m.conn, m.nodes_per_element, rowp, cols)
    R0, A0 = orc.assemble(m, emap, cols.size)
    d = fem.DeviceMesh(m, cuda)

    def close(x, y):
        return np.abs(x.cpu().numpy() - y).max() <= 1e-12 * np.abs(y).max()

    res = torch.full((m.num_nodes * 2,), float("nan"), dtype=torch.float64, device=cuda)
    mat = torch.full((cols.size * 4,), float("nan"), dtype=torch.float64, device=cuda)
    plan.assemble(d.states, d.coords, E, m.nu, t, res, mat)
    assert close(res, R0) and close(mat, A0)
    res.fill_(float("nan"))
    plan.assemble(d.states, d.coords, E, m.nu, t, res)
    assert close(res, R0)
    mesh = (order, d.conn_ptr, d.conn, m.num_elements, d.states, d.coords, E, m.nu, t)
    res.zero_()
    fem.run_residual_kernel(*mesh, res)
    assert close(res, R0)
    res.zero_()
    mat.zero_()
    fem.run_jacobian_kernel(*mesh, torch.from_numpy(emap).to(cuda), res, mat)
    assert close(res, R0) and close(mat, A0)
    plan.close()
