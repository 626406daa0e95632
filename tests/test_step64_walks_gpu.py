"""The float64 step's GVF walks by walk words, by walk lengths and by the ground
bits: the same sums in the same order, at rasters that end inside a tile, and in
launches of one hour and of several that begin at night."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(5, 40), (33, 31), (64, 65)])
@pytest.mark.parametrize("grouped", [True, False])
def test_walks_are_identical(rows, cols, grouped, monkeypatch):
    import torch
    from solweig_cuda_b200 import engine, synthetic
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sc = synthetic.make_scene(rows, cols, seed=rows)
    scene = engine.Scene(sc.dsm, sc.trees, sc.dem, 1.0, landcover=sc.landcover)
    assert scene.struct.gvf_walks and scene.struct.gvf_hits
    met = synthetic.make_met(doy=172, latitude=53.0, longitude=0.0, seed=4)
    if not grouped:
        monkeypatch.setattr(engine.DayRunner64, "GROUP_BYTES", 1)
    saved = scene.struct.gvf_walks, scene.struct.gvf_hits
    res = []
    try:
        for walks, hits in (saved, (None, saved[1]), (None, None)):
            scene.struct.gvf_walks, scene.struct.gvf_hits = walks, hits
            out = engine.DayRunner64(scene, 53.0, 0.0, 3.0, 0.0).run_day(met)
            torch.cuda.synchronize()
            res.append({k: v.clone() for k, v in out.items()})
    finally:
        scene.struct.gvf_walks, scene.struct.gvf_hits = saved
    for other in res[1:]:
        for k, v in res[0].items():
            a, b = v.cpu().numpy(), other[k].cpu().numpy()
            assert np.array_equal(a, b, equal_nan=True), k
