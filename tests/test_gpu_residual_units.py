"""GPU: the residual alone takes two elements per step also in launches that leave warps
idle: both are rows of the same products, so a mesh in the colour layout (independent
elements) takes no longer than in the pair layout, and the values are the oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_colours_take_no_longer_than_pairs(fem, orc, cuda):
    import torch
    m = fem.square_mesh(90, 89, 2, 1.0, 1.0, 0.1, seed=3)
    plan = fem.Plan(2, m.num_nodes, m.conn_ptr, m.conn)
    d = fem.DeviceMesh(m, cuda)
    rowp, cols = plan.pattern()
    orc.set_extended_j(True)  # the plain sum of J cancels by 1 / h
    try:
        R0, _ = orc.assemble(m, orc.element_bsr_map(m.conn_ptr, m.conn, 9, rowp, cols), cols.size)
    finally:
        orc.set_extended_j(False)
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = {}
    for layout in ("pairs", "colours"):
        plan.set_layout(layout)
        res = torch.full((m.num_nodes * 2,), float("nan"), dtype=torch.float64, device=cuda)
        plan.assemble(d.states, d.coords, m.E, m.nu, m.t, res)
        assert np.abs(res.cpu().numpy() - R0).max() <= 1e-12 * np.abs(R0).max()
        times = []
        for _ in range(20):
            a.record()
            for _ in range(20):
                plan.assemble(d.states, d.coords, m.E, m.nu, m.t, res)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        best[layout] = min(times[5:])
    plan.close()
    assert best["colours"] <= 1.2 * best["pairs"]  # 1.42 with one element per warp
