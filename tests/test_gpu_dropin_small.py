"""GPU: the order-4 drop-in Jacobian where it changes between the element and the fragment
kernel (a step of the fragment kernel's 1184 resident warps holds 1, 2, 4, 6 elements per
warp), against the FP64 oracle at 1e-12; and that a mesh of a few elements does not pay
the fragment kernel's whole step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dropin(fem, cuda, m):
    import torch
    rowp, cols = fem.build_bsr_pattern(m.num_nodes, m.conn_ptr, m.conn)
    emap = fem.build_element_bsr_map(m.conn_ptr, m.conn, m.nodes_per_element, rowp, cols)
    d = fem.DeviceMesh(m, cuda)
    dmap = torch.from_numpy(emap).to(cuda)
    mat = torch.zeros(cols.size * 4, dtype=torch.float64, device=cuda)
    res = torch.zeros(m.num_nodes * 2, dtype=torch.float64, device=cuda)

    def run(with_res):
        fem.run_jacobian_kernel(4, d.conn_ptr, d.conn, m.num_elements, d.states, d.coords, m.E, m.nu, m.t, dmap,
                                res if with_res else None, mat, timed=False)
    return run, emap, cols.size, res, mat


# products of elements either side of 1147, 1184, 2220, 4144, 5772
@pytest.mark.parametrize("nx,ny", [(2, 573), (31, 37), (37, 32), (79, 15), (317, 7), (60, 37), (2071, 2), (56, 74), (29, 199),
                                   (74, 78)])
def test_sizes_where_the_kernel_changes(fem, orc, cuda, nx, ny):
    m = fem.square_mesh(nx, ny, 4, 0.01 * nx, 0.01 * ny, 0.1, seed=nx)
    run, emap, nnzb, res, mat = _dropin(fem, cuda, m)
    orc.set_extended_j(True)
    try:
        R0, A0 = orc.assemble(m, emap, nnzb)
    finally:
        orc.set_extended_j(False)
    run(True)
    assert np.abs(res.cpu().numpy() - R0).max() <= 1e-12 * np.abs(R0).max()
    assert np.abs(mat.cpu().numpy() - A0).max() <= 1e-12 * np.abs(A0).max()


def test_few_elements_take_less_than_a_full_step(fem, cuda):
    import torch

    def best(nx, ny):
        run = _dropin(fem, cuda, fem.square_mesh(nx, ny, 4, 1.0, 1.0, 0.1, seed=1))[0]
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        times = []
        for _ in range(25):
            a.record()
            for _ in range(20):
                run(False)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[5:])

    # 64 and 256 elements against 1184: 12 and 12 us against 26 (23 with the fragment kernel)
    full = best(37, 32)
    assert best(8, 8) < 0.7 * full and best(16, 16) < 0.7 * full
