"""A scene's walk words, lengths and albedo-without-shadow plane under another step
table than theirs: the day and the float64 step do without them."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _steps(scene, scale):
    from solweig_cuda_b200 import rays
    scene.gvf_dxdy_host, scene.first_steps, scene.second_steps = rays.gvf_offsets(scale)
    scene.gvf_host_ptr = scene.gvf_dxdy_host.ctypes.data_as(ctypes.c_void_p)


def _runs(scene, met):
    import torch
    from solweig_cuda_b200 import batched, engine
    out = batched.ChosenDay(scene, 53.0, 0.0, 3.0, 0.0, outputs=("tmrt", "kup", "lup")).run_day(met)
    res = [v.clone() for v in out.values()]
    out = engine.DayRunner64(scene, 53.0, 0.0, 3.0, 0.0).run_day(met, outputs=("tmrt", "kup", "lup"))
    res += [v.clone() for v in out.values()]
    torch.cuda.synchronize()
    return [v.cpu().numpy() for v in res]


# words of 22 steps under a table of 11, words of 11 under a table of 22, and of
# 22 under another table of 22 (its directions in reverse)
@pytest.mark.parametrize("made,used", [(1.0, 0.5), (0.5, 1.0), (1.0, None)])
def test_other_tables_do_without_the_words(cuda, made, used):
    from solweig_cuda_b200 import engine, synthetic
    s = synthetic.make_scene(45, 70, seed=9, building_cover=0.2)
    scene = engine.Scene(s.dsm, s.trees, s.dem, 1.0, landcover=s.landcover)
    met = synthetic.make_met(doy=172, latitude=53.0, longitude=0.0, seed=4)
    _steps(scene, made)
    scene._gvf_statics(engine.stream_handle())
    assert scene.struct.gvf_walks and scene.struct.gvf_table
    if used is not None:
        _steps(scene, used)
    else:
        scene.gvf_dxdy_host = np.ascontiguousarray(scene.gvf_dxdy_host[::-1])
        scene.gvf_host_ptr = scene.gvf_dxdy_host.ctypes.data_as(ctypes.c_void_p)
    got = _runs(scene, met)
    scene.struct.gvf_walks = scene.struct.gvf_hits = scene.struct.gvf_nosh = None
    for a, b in zip(got, _runs(scene, met)):
        assert np.array_equal(a, b, equal_nan=True)
