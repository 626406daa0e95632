"""Kernels of the day gradient at the edges of their tiles, passes and warps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(rows, cols, hours, objective="utci", seed=3):
    import torch
    from solweig_cuda_b200 import engine, grad, synthetic
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    sc = synthetic.make_scene(rows, cols, seed=seed)
    scene = engine.Scene(sc.dsm, sc.trees, sc.dem, 1.0, landcover=sc.landcover)
    met = synthetic.make_met(doy=172, latitude=53.0, longitude=0.0, seed=4)[24 - hours:] if hours < 24 else \
        synthetic.make_met(doy=172, latitude=53.0, longitude=0.0, seed=4)
    rng = np.random.default_rng(5)
    p = [rng.uniform(a, b, scene.shape).astype(np.float32) for a, b in ((0.1, 0.4), (0.9, 0.98), (0.02, 0.2))]
    return scene, grad.DayGradient(scene, 53.0, 0.0, 3.0, 0.0, hours=hours, objective=objective), p, met


# fewer pixels than a warp, one more than a warp's 32, several blocks; daytime
# hours that fill their passes of four and that do not
@pytest.mark.parametrize("rows,cols,hours", [(5, 6, 24), (3, 11, 7), (37, 41, 9), (70, 65, 24)])
def test_luminance_gradient_is_the_masks_times_the_pixel_adjoints(rows, cols, hours):
    """With the weight on one pixel every patch it sees has the same partial and
    the others none; over all pixels the partials add up (float32 chains of at
    most 512 additions)."""
    scene, dg, p, met = _case(rows, cols, hours, "tmrt")
    P = dg.patches
    bits = np.unpackbits(scene.masks.cpu().numpy().view(np.uint8).reshape(2, -1, rows * cols, 4).transpose(0, 2, 1, 3)
                         .reshape(2, rows * cols, -1), axis=2, bitorder="little")[:, :, :P].astype(bool)
    sky, veg = bits[0] & ~bits[1], bits[0] & bits[1]
    pixels = range(rows * cols) if rows * cols <= 33 else (0, 31, 32, rows * cols // 2, rows * cols - 1)
    total = np.zeros((hours, 4, P))
    for q in pixels:
        w = np.zeros((rows, cols), np.float32)
        w.flat[q] = 1.25
        lum = dg.backward(*p, met, w)[4][:, :, :P]
        total += lum
        for hr in range(hours):
            for i, mask in enumerate((sky[q], sky[q], veg[q], veg[q])):
                assert not lum[hr, i, ~mask].any()
                assert np.unique(lum[hr, i, mask]).size <= 1
        if sky[q].any() and veg[q].any():
            for i in (0, 1):
                a, b = lum[:, i, sky[q]][:, 0], lum[:, i + 2, veg[q]][:, 0]
                assert np.abs(b - 0.03 * a).max() <= 2e-7 * np.abs(a).max()
        assert lum.any()
    if rows * cols <= 33:
        lum = dg.backward(*p, met, np.full((rows, cols), 1.25, np.float32))[4][:, :, :P]
        assert np.abs(lum - total).max() <= 512 * 2.0 ** -24 * np.abs(total).max()


# one tile, a column and a row more, less than a tile both ways, several tiles;
# an odd number of daytime hours and one pass
@pytest.mark.parametrize("rows,cols,hours", [(32, 32, 24), (33, 32, 9), (20, 45, 8), (70, 65, 24)])
def test_transposed_walks_match_differences_at_tile_and_raster_edges(rows, cols, hours):
    """Central differences of the forward in the albedo and emissivity of the
    pixels at the raster's border and along the 32-pixel tiles' edges (relative
    tolerance of the differences as for whole fields: 1e-3)."""
    scene, dg, p, met = _case(rows, cols, hours)
    rng = np.random.default_rng(8)
    weights = rng.uniform(0.5, 1.5, (rows, cols)).astype(np.float32)
    grads = dg.backward(*p, met, weights)[:2]
    edges = np.zeros((rows, cols), bool)
    for r in (0, 1, 31, 32, rows - 1):
        edges[min(r, rows - 1)] = True
    for c in (0, 1, 31, 32, cols - 1):
        edges[:, min(c, cols - 1)] = True
    for i in (0, 1):
        v = np.where(edges, rng.uniform(0.5, 1.0, (rows, cols)), 0.0)
        J = []
        for h in (1e-2, -1e-2):
            q = list(p)
            q[i] = (p[i].astype(np.float64) + h * v).astype(np.float32)
            J.append(float(np.nansum(dg.forward(*q, met).cpu().numpy() * weights)))
        fd = (J[0] - J[1]) / 2e-2
        ad = float((grads[i].cpu().numpy().astype(np.float64) * v).sum())
        assert abs(ad - fd) <= 1e-3 * abs(fd), (i, ad, fd)


@pytest.mark.parametrize("hours", [24, 9])
def test_walks_that_do_not_start_at_their_pixel_take_the_general_path(hours):
    """A table whose walks start one step out has no walk words: the general
    kernels stay consistent with each other."""
    scene, dg, p, met = _case(40, 37, hours)
    table = scene.gvf_dxdy_host.reshape(-1)
    assert np.shares_memory(table, scene.gvf_dxdy_host)
    saved = table.copy()
    try:
        steps = table.reshape(18, 22, 2)
        steps[:, 0] = steps[:, 1]
        rng = np.random.default_rng(8)
        w = rng.uniform(0.5, 1.5, scene.shape).astype(np.float32)
        grad = dg.backward(*p, met, w)[0].cpu().numpy().astype(np.float64)
        v = rng.uniform(0.5, 1.0, scene.shape)
        J = []
        for h in (1e-2, -1e-2):
            a = (p[0].astype(np.float64) + h * v).astype(np.float32)
            J.append(float(np.nansum(dg.forward(a, p[1], p[2], met).cpu().numpy() * w)))
        fd = (J[0] - J[1]) / 2e-2
        assert abs(float((grad * v).sum()) - fd) <= 1e-3 * abs(fd)
    finally:
        table[:] = saved


def test_walk_lengths_alone_need_no_walls_and_any_offset_of_the_halo():
    """solweig_gvf_statics without walls and faces, and with a table whose walks
    start one step out: lengths as a loop over the steps finds them."""
    import ctypes
    import torch
    from solweig_cuda_b200 import _lib
    from solweig_cuda_b200.engine import device_ptr, stream_handle
    scene, _, _, _ = _case(37, 41, 24)
    rows, cols = scene.shape
    table = scene.gvf_dxdy_host.reshape(18, 22, 2).copy()
    table[:, 0] = table[:, 1]
    struct = _lib.SolweigScene.from_buffer_copy(scene.struct)
    struct.walls = struct.gvf_face = None
    hits = torch.empty((4, rows, cols), dtype=torch.int32, device="cuda")
    nosh = torch.empty((rows, cols), dtype=torch.float32, device="cuda")
    _lib.check(_lib.lib().solweig_gvf_statics(ctypes.byref(struct), table.ctypes.data_as(ctypes.c_void_p), 1, 22,
                                              device_ptr(hits), device_ptr(nosh), stream_handle()),
               "solweig_gvf_statics")
    got = hits.cpu().numpy()
    ground = scene.flags.cpu().numpy().reshape(rows, cols) & 1
    rr, cc = np.mgrid[:rows, :cols]
    for j in range(18):
        lim, frozen = np.zeros((rows, cols), int), np.zeros((rows, cols), bool)
        going = ground.astype(bool).copy()
        for m in range(22):
            r, c = rr + table[j, m, 0], cc + table[j, m, 1]
            inside = (r >= 0) & (r < rows) & (c >= 0) & (c < cols)
            free = inside & (ground[np.clip(r, 0, rows - 1), np.clip(c, 0, cols - 1)] == 1)
            frozen |= going & ~inside & (m > 0)
            going &= free
            lim += going
        code = (got[j // 5] >> (6 * (j % 5))) & 63
        assert np.array_equal(code & 31, lim), j
        assert np.array_equal((code & 32) != 0, frozen), j
