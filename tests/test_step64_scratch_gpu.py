"""The float64 step with scratch on an odd multiple of 8 bytes: the same results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(33, 31), (40, 64)])
@pytest.mark.parametrize("grouped", [True, False])
def test_scratch_needs_the_alignment_of_a_double(cuda, rows, cols, grouped, monkeypatch):
    import torch
    from solweig_cuda_b200 import engine, synthetic
    sc = synthetic.make_scene(rows, cols, seed=rows)
    scene = engine.Scene(sc.dsm, sc.trees, sc.dem, 1.0, landcover=sc.landcover)
    met = synthetic.make_met(doy=172, latitude=53.0, longitude=0.0, seed=4)
    if not grouped:
        monkeypatch.setattr(engine.DayRunner64, "GROUP_BYTES", 1)
    runner = engine.DayRunner64(scene, 53.0, 0.0, 3.0, 0.0)
    want = {k: v.cpu().numpy() for k, v in runner.run_day(met).items()}
    odd = torch.empty(runner.scratch.numel() + 1, dtype=torch.float64, device=cuda)[1:]
    assert odd.data_ptr() % 16 == 8
    runner.scratch = odd.view(runner.scratch.shape)
    for k, v in runner.run_day(met).items():
        assert np.array_equal(v.cpu().numpy(), want[k], equal_nan=True), k
