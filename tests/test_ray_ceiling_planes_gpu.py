"""The ceiling planes on the device against the numpy construction of
``test_ray_ceiling``: not only bounds, but as low as it makes them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# ends inside a scan segment, a batch of eight steps and a block of 32 lines
@pytest.mark.parametrize("rows,cols", [(7, 90), (90, 7), (33, 65), (64, 64), (129, 71), (300, 280)])
@pytest.mark.parametrize("doy,lat", [(172, 53.0), (355, -35.0)])
def test_planes_follow_the_construction(cuda, rows, cols, doy, lat):
    """The window maximum is a maximum of float32 heights: equal.  The ceiling is
    a chain of at most nx + 16 float32 subtractions rounded up (and the carries'
    products): from 0 to 4 (nx + 16) roundings above the float64 chain."""
    import torch
    from test_ray_ceiling import ceiling_planes
    from solweig_cuda_b200 import batched, engine, synthetic
    sc = synthetic.make_scene(rows, cols, seed=rows)
    scene = engine.Scene(sc.dsm, sc.trees, sc.dem, 1.0, landcover=sc.landcover)
    met = synthetic.make_met(doy=doy, latitude=lat, longitude=0.0, seed=4)
    day = batched.ChosenDay(scene, lat, 0.0, 3.0, 0.0, use_graph=False)
    plan = day.plan(met)
    day._part(0, 0, 24)
    torch.cuda.synchronize()
    at, n = day.work_offsets()["gvf"], rows * cols
    planes = day.work[at:at + 8 * n * 24].view(torch.float32).cpu().numpy().reshape(24, rows, cols, 2)
    H = scene.geo32.cpu().numpy().reshape(rows, cols, 4)[..., :3].max(axis=2).astype(np.float64)
    checked = 0
    for hr, (record, ray, _) in enumerate(plan):
        if not record.daytime or ray.steps < 5:
            continue
        C, f, M = ceiling_planes(H, ray.dxdy, ray.dz)
        ceiling = planes[hr, ..., 0].astype(np.float64)
        nx = rows if f["rows_major"] else cols
        slack = 4 * (nx + 16) * 2.0 ** -24 * (H.max() + nx * f["delta"])
        assert np.array_equal(planes[hr, ..., 1], M), hr
        assert (ceiling >= C).all() and (ceiling - C).max() <= slack, hr
        checked += 1
    assert checked >= 3
