"""Ray ceilings of the sweep: upper bounds along every ray, at raster sizes that
end inside a scan segment, a batch of eight steps and a block of 32 lines."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(7, 90), (90, 7), (33, 65), (64, 64), (129, 71)])
@pytest.mark.parametrize("doy,lat", [(172, 53.0), (355, -35.0)])
def test_ceilings_bound_the_heights_ahead(rows, cols, doy, lat):
    """At step k of a pixel's ray the plane holds at least what any later sample
    presents there, max_j H_j - (dz_{j-1} - dz_{k-1}), and the maximum of the next
    eight samples."""
    import torch
    from solweig_cuda_b200 import batched, engine, synthetic
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sc = synthetic.make_scene(rows, cols, seed=rows)
    scene = engine.Scene(sc.dsm, sc.trees, sc.dem, 1.0, landcover=sc.landcover)
    met = synthetic.make_met(doy=doy, latitude=lat, longitude=0.0, seed=4)
    day = batched.ChosenDay(scene, lat, 0.0, 3.0, 0.0, use_graph=False)
    plan = day.plan(met)
    day._part(0, 0, 24)
    torch.cuda.synchronize()
    at = day.work_offsets()["gvf"]
    n = rows * cols
    planes = day.work[at:at + 8 * n * 24].view(torch.float32).cpu().numpy().reshape(24, rows, cols, 2)
    geo = scene.geo32.cpu().numpy().reshape(rows, cols, 4)
    H = geo[..., :3].max(axis=2).astype(np.float64)
    checked = 0
    for hr, (record, table, _) in enumerate(plan):
        if not record.daytime or table.steps < 5:
            continue
        dxdy, dz = np.asarray(table.dxdy).reshape(-1, 2), np.asarray(table.dz, dtype=np.float64)
        later = np.full((rows, cols), -np.inf)           # suffix maximum of H_j - dz_{j-1}
        window = [np.full((rows, cols), -np.inf)] * 8    # H of the steps k .. k + 7
        for k in range(table.steps - 1, 0, -1):
            dr, dc = int(dxdy[k, 0]), int(dxdy[k, 1])
            r0, r1, c0, c1 = max(0, -dr), min(rows, rows - dr), max(0, -dc), min(cols, cols - dc)
            h = np.full((rows, cols), -np.inf)
            if r0 >= r1 or c0 >= c1:
                window = [h] + window[:-1]
                continue
            here = (slice(r0, r1), slice(c0, c1))
            there = (slice(r0 + dr, r1 + dr), slice(c0 + dc, c1 + dc))
            h[here] = H[there]
            later = np.maximum(later, h - dz[k - 1])
            window = [h] + window[:-1]
            ceiling, ahead = planes[hr][there][..., 0], planes[hr][there][..., 1]
            assert (ceiling - dz[k - 1] >= later[here]).all(), (hr, k)
            assert (ahead >= np.max(window, axis=0)[here]).all(), (hr, k)
            checked += int(np.isfinite(ceiling).sum())
    assert checked
