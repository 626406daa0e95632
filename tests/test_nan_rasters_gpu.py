"""Rasters with a cell that is not a number: the highest object is then unknown and
the rays run to the raster's edge."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAN = float("nan")


@pytest.mark.parametrize("option", [1, 2])
@pytest.mark.parametrize("shape,scale", [((40, 50), 1.0), ((1, 1), 1.0), ((3, 300), 0.5)])
def test_rays_without_a_highest_object(cuda, option, shape, scale):
    from solweig_cuda_b200 import engine, rays
    dxdy, dz, lengths, _ = rays.svf_rays(option, shape, NAN, scale)
    t_dxdy, t_dz, t_len, cap = engine.svf_ray_tables(option, shape, NAN, scale, cuda)
    assert np.array_equal(t_len.cpu().numpy(), lengths) and lengths.max() <= cap
    for p, n in enumerate(lengths):
        assert np.array_equal(t_dxdy[p, :n].cpu().numpy(), dxdy[p, :n]), p
        assert np.array_equal(t_dz[p, :n].cpu().numpy(), dz[p, :n]), p


def test_scene_with_one_unknown_cell(cuda):
    """The scene's masks equal the plain float64 walk's along the numpy rays, and a
    day on it is a number away from the cell."""
    import torch
    from solweig_cuda_b200 import _lib, batched, engine, rays, synthetic
    from solweig_cuda_b200.engine import device_ptr, stream_handle
    c = synthetic.make_scene(57, 83, seed=6)
    dsm = c.dsm.astype(np.float64)
    dsm[20, 31] = NAN
    scene = engine.Scene(dsm, c.trees, c.dem, 1.0, landcover=c.landcover)
    assert np.isnan(scene.amaxvalue) and scene.geo32 is None
    dxdy, dz, lengths, cap = rays.svf_rays(2, dsm.shape, NAN, 1.0)
    t = [torch.from_numpy(np.ascontiguousarray(x)).to(cuda) for x in (dxdy, dz, lengths)]
    lay = engine.sky_layout(2)
    masks = torch.empty_like(scene.masks)
    planes = torch.empty((16,) + dsm.shape, dtype=torch.float64, device=cuda)
    sums = torch.empty((4,) + dsm.shape, dtype=torch.float32, device=cuda)
    counts = torch.empty((lay.struct.nbands,) + dsm.shape, dtype=torch.uint8, device=cuda)
    _lib.check(_lib.lib().solweig_svf(
        device_ptr(scene.dsm), device_ptr(scene.vegdem), device_ptr(scene.vegdem2), device_ptr(scene.flags), 57, 83,
        lay.struct.patches, cap, device_ptr(t[0]), device_ptr(t[1]), device_ptr(t[2]), NAN, ctypes.byref(lay.struct),
        lay.band_weights.ctypes.data_as(ctypes.c_void_p), lay.sectors.ctypes.data_as(ctypes.c_void_p), 0.03,
        device_ptr(masks), device_ptr(planes), device_ptr(sums), device_ptr(counts), stream_handle()), "solweig_svf")
    assert torch.equal(scene.masks, masks)
    met = synthetic.make_met(doy=172, latitude=53.0, longitude=0.0, seed=4)
    tmrt = batched.ChosenDay(scene, 53.0, 0.0, 3.0, 0.0, outputs=("tmrt",)).run_day(met)["tmrt"]
    assert bool(torch.isfinite(tmrt[:, 45:, 60:]).all())


def test_svf_calculator_without_a_highest_object(cuda):
    """A height that no ray exceeds gives the same masks and planes."""
    import torch
    from solweig_cuda_b200 import svf, synthetic
    c = synthetic.make_scene(33, 47, seed=8)
    dsm, top = c.dsm.astype(np.float64), c.trees.astype(np.float64) + c.dsm
    bot, bush = 0.25 * c.trees + c.dsm, np.zeros(dsm.shape)
    a = svf.svf_calculator(2, NAN, dsm, top, bot, bush, 1.0)
    b = svf.svf_calculator(2, float("inf"), dsm, top, bot, bush, 1.0)
    for x, y in zip(a, b):
        assert torch.equal(x, y)
