"""Walk words that a day makes in its work buffer: days too short to hold them among
the patch sums and days that do, rasters that end inside a tile."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(33, 31), (64, 65), (5, 70)])
@pytest.mark.parametrize("hours", [1, 4, 5, 6, 24])
def test_words_made_by_the_day_equal_the_scenes(cuda, rows, cols, hours):
    """The same planes, and nothing written behind the buffer."""
    import torch
    from solweig_cuda_b200 import batched, engine, synthetic
    s = synthetic.make_scene(rows, cols, seed=rows)
    scene = engine.Scene(s.dsm, s.trees, s.dem, 1.0, landcover=s.landcover)
    met = synthetic.make_met(doy=172, latitude=53.0, longitude=0.0, seed=2)
    met = met if hours == 24 else met[9:9 + hours]
    res = []
    for own in (False, True):
        if own:
            scene.struct.gvf_walks = None
        day = batched.ChosenDay(scene, 53.0, 0.0, 3.0, 0.0, hours=hours, outputs=("tmrt", "kup", "lup"))
        guarded = torch.full((day.work_bytes + 4096,), 0x5a, dtype=torch.uint8, device=cuda)
        guarded[:day.work_bytes] = 0
        day.work = guarded
        res.append([v.clone() for v in day.run_day(met).values()])
        torch.cuda.synchronize()
        assert bool((guarded[day.work_bytes:] == 0x5a).all())
    for a, b in zip(*res):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
