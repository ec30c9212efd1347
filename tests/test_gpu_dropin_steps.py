"""GPU: the drop-in kernels of orders 2 to 4 over several steps of a warp: pairs of elements,
staging slots refilled after their reductions, the next pair's map rows, and a last pair of
one element.  Grid and random numbering, a matrix that is 16-byte and one that is 8-byte
aligned; added to what the outputs hold.  Against the FP64 oracle at 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# odd element counts; resident warps: 2368 at order 2, 1184 at orders 3 and 4, two elements each
CASES = [(2, "linear", 131, 115), (2, "nonlinear", 131, 115), (3, "linear", 97, 79), (3, "nonlinear", 97, 79),
         (4, "linear", 91, 83)]


def _scrambled(fem, m):
    r = np.random.default_rng(7)
    pe, key = r.permutation(m.num_elements), r.permutation(m.num_nodes)
    new = np.empty(m.num_nodes, np.int64)
    new[key] = np.arange(m.num_nodes)
    conn = new[m.conn.reshape(-1, m.nodes_per_element)[pe]].reshape(-1).astype(np.int32)
    return fem.Mesh(m.order, np.ascontiguousarray(m.coords[key]), m.conn_ptr, conn, np.ascontiguousarray(m.states[key]),
                    m.E, m.nu, m.t)


@pytest.mark.parametrize("scrambled", [False, True], ids=["grid", "random"])
@pytest.mark.parametrize("order,strain,nx,ny", CASES)
def test_dropin_many_steps(fem, orc, cuda, order, strain, nx, ny, scrambled):
    import torch
    m = fem.square_mesh(nx, ny, order, 1.0, 1.0, 0.15, seed=30 + order)
    if scrambled:
        m = _scrambled(fem, m)
    rowp, cols = fem.build_bsr_pattern(m.num_nodes, m.conn_ptr, m.conn)
    emap = fem.build_element_bsr_map(m.conn_ptr, m.conn, m.nodes_per_element, rowp, cols)
    orc.set_extended_j(True)  # the plain sum of J cancels by 1 / h
    try:
        R0, A0 = orc.assemble(m, emap, cols.size, strain=strain)
    finally:
        orc.set_extended_j(False)
    d = fem.DeviceMesh(m, cuda)
    dmap = torch.from_numpy(emap).to(cuda)
    mesh = (order, d.conn_ptr, d.conn, m.num_elements, d.states, d.coords, m.E, m.nu, m.t)
    for offset in (0, 1):
        buf = torch.full((cols.size * 4 + 2,), 1.0, dtype=torch.float64, device=cuda)
        mat = buf[offset:offset + cols.size * 4]
        res = torch.full((m.num_nodes * 2,), 1.0, dtype=torch.float64, device=cuda)
        fem.run_jacobian_kernel(*mesh, dmap, res, mat, strain=strain)
        assert np.abs(mat.cpu().numpy() - 1.0 - A0).max() <= 1e-12 * np.abs(A0).max()
        assert np.abs(res.cpu().numpy() - 1.0 - R0).max() <= 1e-12 * np.abs(R0).max()
        assert torch.all(buf[offset + cols.size * 4:] == 1.0) and (offset == 0 or float(buf[0]) == 1.0)
        buf.fill_(1.0)
        fem.run_jacobian_kernel(*mesh, dmap, None, mat, strain=strain)
        assert np.abs(mat.cpu().numpy() - 1.0 - A0).max() <= 1e-12 * np.abs(A0).max()
        res.fill_(1.0)
        fem.run_residual_kernel(*mesh, res, strain=strain)
        assert np.abs(res.cpu().numpy() - 1.0 - R0).max() <= 1e-12 * np.abs(R0).max()
