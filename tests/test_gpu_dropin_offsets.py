"""GPU: the drop-in Jacobian through a caller's map whose blocks stand at odd offsets, so that
half of them are 8-byte aligned only (FP64 atomics) and no two are adjacent; order 4 at sizes
that run the element kernel and the fragment kernel.  Against the FP64 oracle at 1e-12; the
gaps between the blocks keep their value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,strain,nx,ny", [(2, "linear", 7, 5), (2, "nonlinear", 7, 5), (3, "linear", 7, 5),
                                                (3, "nonlinear", 7, 5), (4, "linear", 7, 5), (4, "linear", 34, 34)])
def test_dropin_odd_offsets(fem, orc, cuda, order, strain, nx, ny):
    import torch
    m = fem.square_mesh(nx, ny, order, 1.0, 1.0, 0.1, seed=60 + order)
    rowp, cols = fem.build_bsr_pattern(m.num_nodes, m.conn_ptr, m.conn)
    emap = fem.build_element_bsr_map(m.conn_ptr, m.conn, m.nodes_per_element, rowp, cols)
    R0, A0 = orc.assemble(m, emap, cols.size, strain=strain)
    d = fem.DeviceMesh(m, cuda)
    dmap = torch.from_numpy(emap // 4 * 5 + 1).to(cuda)  # blocks five doubles apart from offset 1
    mat = torch.full((cols.size * 5 + 1,), 1.0, dtype=torch.float64, device=cuda)
    res = torch.zeros(m.num_nodes * 2, dtype=torch.float64, device=cuda)
    fem.run_jacobian_kernel(order, d.conn_ptr, d.conn, m.num_elements, d.states, d.coords, m.E, m.nu, m.t, dmap, res, mat,
                            strain=strain)
    got = mat.cpu().numpy()
    A = got[1:].reshape(-1, 5)
    assert np.abs(A[:, :4].reshape(-1) - 1.0 - A0.reshape(-1)).max() <= 1e-12 * np.abs(A0).max()
    assert got[0] == 1.0 and (A[:, 4] == 1.0).all()
    assert np.abs(res.cpu().numpy() - R0).max() <= 1e-12 * np.abs(R0).max()
