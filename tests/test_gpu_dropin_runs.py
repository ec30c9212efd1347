"""GPU: the drop-in Jacobian of orders 2 to 4, whose lanes add stretches of blocks that are
adjacent in the matrix: numberings that make every stretch length, a matrix that is only
8-byte aligned (atomics), odd element counts, with and without the residual, LINEAR and
NONLINEAR (orders 2, 3); accumulated into a matrix that is not zero.  Against the FP64
oracle at 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _renumbered(fem, m, how):
    """Nodes numbered along y (no x-neighbours adjacent), at random, or as they are."""
    n = m.num_nodes
    if how == "grid":
        return m
    if how == "columns":
        key = np.lexsort((m.coords[:, 1].round(3), m.coords[:, 0].round(3)))
    else:
        key = np.random.default_rng(3).permutation(n)
    new = np.empty(n, np.int64)
    new[key] = np.arange(n)
    return fem.Mesh(m.order, np.ascontiguousarray(m.coords[key]), m.conn_ptr, new[m.conn].astype(np.int32),
                    np.ascontiguousarray(m.states[key]), m.E, m.nu, m.t)


@pytest.mark.parametrize("offset", [0, 1], ids=["aligned", "8-byte"])
@pytest.mark.parametrize("how", ["grid", "columns", "random"])
@pytest.mark.parametrize("order,strain", [(2, "linear"), (2, "nonlinear"), (3, "linear"), (3, "nonlinear"), (4, "linear")])
def test_dropin_stretches(fem, orc, cuda, order, strain, how, offset):
    import torch
    m = _renumbered(fem, fem.square_mesh(7, 5, order, 1.0, 1.0, 0.1, seed=90 + order), how)
    rowp, cols = fem.build_bsr_pattern(m.num_nodes, m.conn_ptr, m.conn)
    emap = fem.build_element_bsr_map(m.conn_ptr, m.conn, m.nodes_per_element, rowp, cols)
    R0, A0 = orc.assemble(m, emap, cols.size, strain=strain)
    d = fem.DeviceMesh(m, cuda)
    dmap = torch.from_numpy(emap).to(cuda)
    for with_res in (True, False):
        buf = torch.full((cols.size * 4 + 2,), 1.0, dtype=torch.float64, device=cuda)
        mat = buf[offset:offset + cols.size * 4]
        res = torch.zeros(m.num_nodes * 2, dtype=torch.float64, device=cuda)
        fem.run_jacobian_kernel(order, d.conn_ptr, d.conn, m.num_elements, d.states, d.coords, m.E, m.nu, m.t, dmap,
                                res if with_res else None, mat, strain=strain)
        A = mat.cpu().numpy() - 1.0
        assert np.abs(A - A0).max() <= 1e-12 * np.abs(A0).max()
        assert float(buf[0]) == 1.0 or offset == 0
        assert torch.all(buf[offset + cols.size * 4:] == 1.0)
        if with_res:
            assert np.abs(res.cpu().numpy() - R0).max() <= 1e-12 * np.abs(R0).max()
        else:
            assert torch.all(res == 0.0)
