"""GPU: the batch tuner starts from what the batch has and does not replace it by something
slower: the captured graph's replay after tuning takes no longer than before, whichever
tile lengths, launch forms and kernels were fastest order by order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _replay_seconds(batch):
    import torch
    batch.capture()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    times = []
    for _ in range(15):
        a.record()
        for _ in range(5):
            batch.replay()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    return min(times[3:])


@pytest.mark.parametrize("specs", [[(60, 60, 2)] * 10, [(31, 30, 1 + i % 4) for i in range(12)], [(60, 61, 3), (40, 41, 4)]],
                         ids=["order2", "mixed", "two"])
@pytest.mark.parametrize("tiles", [None, [16, 6, 6, 6]], ids=["default", "six"])
def test_tuning_never_costs(fem, cuda, specs, tiles):
    import torch
    meshes = [fem.square_mesh(nx, ny, p, 1.0, 1.0, 0.15, seed=i) for i, (nx, ny, p) in enumerate(specs)]
    plans = [fem.Plan(m.order, m.num_nodes, m.conn_ptr, m.conn) for m in meshes]
    batch = fem.Batch(plans)
    out = []
    for i, m in enumerate(meshes):
        d = fem.DeviceMesh(m, cuda)
        out.append((d, torch.zeros(m.num_nodes * 2, dtype=torch.float64, device=cuda),
                    torch.zeros(plans[i].nnzb * 4, dtype=torch.float64, device=cuda)))
        batch.bind(i, d.states, d.coords, m.E, m.nu, m.t, out[i][1], out[i][2])
    if tiles:
        batch.set_tiles(tiles)
    before = _replay_seconds(batch)
    ref = [(r.clone(), a.clone()) for _, r, a in out]
    assert batch.tune(reps=3) > 0.0
    after = _replay_seconds(batch)
    # two timings of one configuration differ by about 2 %; the former tuner cost 27 % ("order2")
    assert after <= 1.1 * before, batch.info()
    for (r0, a0), (_, r, a) in zip(ref, out):
        assert (r - r0).abs().max() <= 1e-13 * r0.abs().max() and (a - a0).abs().max() <= 1e-13 * a0.abs().max()
