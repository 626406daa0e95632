"""The device-built visibility rays (``solweig_svf_ray_tables``) against the
numpy tables, bit for bit, and the drop-in sky view factor on rasters whose
heights do and do not fit float32 (packed and float64 walks with ceilings)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("option", [1, 2])
@pytest.mark.parametrize("shape,amax,scale", [((40, 50), 30.0, 1.0), ((1, 1), 5.0, 1.0), ((3, 700), 41.5, 0.5),
                                              ((900, 257), 0.0, 1.0), ((64, 64), -1.0, 1.0), ((300, 300), 1e4, 2.0)])
def test_device_rays_equal_numpy(cuda, option, shape, amax, scale):
    from solweig_cuda_b200 import engine, rays
    dxdy, dz, lengths, _ = rays.svf_rays(option, shape, amax, scale)
    t_dxdy, t_dz, t_len, cap = engine.svf_ray_tables(option, shape, amax, scale, cuda)
    got = t_len.cpu().numpy()
    assert np.array_equal(got, lengths) and got.max() <= cap
    for p, n in enumerate(lengths):
        assert np.array_equal(t_dxdy[p, :n].cpu().numpy(), dxdy[p, :n]), p
        assert np.array_equal(t_dz[p, :n].cpu().numpy(), dz[p, :n]), p


@pytest.mark.parametrize("shift", [0.0, 1e-9, -4.0])
def test_svf_calculator_forms_agree_with_the_plain_walk(cuda, shift):
    """Every mask and plane of svf_calculator (ceilings, packed geometry where
    it fits) equals the plain float64 walk of solweig_svf."""
    import ctypes
    import torch
    from solweig_cuda_b200 import _lib, engine, svf, synthetic
    from solweig_cuda_b200.engine import device_ptr, stream_handle
    c = synthetic.make_scene(57, 83, seed=6)
    dsm, trees = c.dsm.astype(np.float64) + shift, c.trees.astype(np.float64)
    top, bot = trees + dsm, trees * 0.25 + dsm
    top[top == dsm] = 0
    bot[bot == dsm] = 0
    bush = np.logical_not(bot * top) * top
    amax = float(max(dsm.max() - dsm.min(), trees.max()))
    got = svf.svf_calculator(2, amax, dsm, top, bot, bush, 1.0)
    t = [torch.from_numpy(x).to(cuda) for x in (dsm, top, bot)]
    assert (engine.packed_geometry(*t) is None) == (shift != 0.0)
    lay = engine.sky_layout(2)
    dxdy, dz, lengths, cap = engine.svf_ray_tables(2, dsm.shape, amax, 1.0, cuda)
    flags = torch.from_numpy((bush > 1).astype(np.uint8) << 1).to(cuda)
    P = lay.struct.patches
    masks = torch.empty((10,) + dsm.shape, dtype=torch.int32, device=cuda)
    planes = torch.empty((16,) + dsm.shape, dtype=torch.float64, device=cuda)
    sums = torch.empty((4,) + dsm.shape, dtype=torch.float32, device=cuda)
    counts = torch.empty((lay.struct.nbands,) + dsm.shape, dtype=torch.uint8, device=cuda)
    cubes = [torch.empty(dsm.shape + (P,), dtype=torch.float32, device=cuda) for _ in range(3)]
    L = _lib.lib()
    _lib.check(L.solweig_svf(
        device_ptr(t[0]), device_ptr(t[1]), device_ptr(t[2]), device_ptr(flags), dsm.shape[0], dsm.shape[1], P, cap,
        device_ptr(dxdy), device_ptr(dz), device_ptr(lengths), float(max(x.max() for x in (dsm, top, bot))),
        ctypes.byref(lay.struct), lay.band_weights.ctypes.data_as(ctypes.c_void_p),
        lay.sectors.ctypes.data_as(ctypes.c_void_p), 0.03, device_ptr(masks), device_ptr(planes), device_ptr(sums),
        device_ptr(counts), stream_handle()), "solweig_svf")
    _lib.check(L.solweig_svf_unpack(device_ptr(masks), dsm.size, P, *(device_ptr(x) for x in cubes), stream_handle()),
               "solweig_svf_unpack")
    for k, i in enumerate(svf._ORDER):
        assert torch.equal(got[k], planes[i]), k
    for a, b in zip(got[15:18], (cubes[1], cubes[2], cubes[0])):
        assert torch.equal(a, b)
    assert torch.equal(got[18], planes[15])
