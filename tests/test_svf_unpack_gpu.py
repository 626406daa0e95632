"""Visibility cubes from the packed masks: blocks that end inside a pixel, odd
patch counts, and cubes that do not start on 16 bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("pixels,patches", [(1, 1), (1, 153), (7, 153), (129, 145), (1031, 153), (33, 160), (2050, 31)])
def test_unpacked_cubes_equal_the_bits(pixels, patches, offset):
    import torch
    from solweig_cuda_b200 import _lib
    from solweig_cuda_b200.engine import device_ptr, stream_handle
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(pixels + patches)
    words = _lib.MASK_WORDS
    masks = rng.integers(0, 2 ** 32, (2 * words, pixels), dtype=np.uint32)
    dev = torch.from_numpy(masks.view(np.int32)).cuda()
    n = pixels * patches
    store = [torch.full((n + offset + 4,), -7.0, device="cuda") for _ in range(3)]
    cubes = [x[offset:offset + n] for x in store]
    _lib.check(_lib.lib().solweig_svf_unpack(device_ptr(dev), pixels, patches, *(device_ptr(x) for x in cubes),
                                             stream_handle()), "solweig_svf_unpack")
    k = np.arange(patches)
    s, v = (((masks[w0 + (k >> 5)] >> (k & 31)[:, None].astype(np.uint32)) & 1).T.astype(bool) for w0 in (0, words))
    for got, want in zip(cubes, (s, ~(s & v), ~(~s & v))):
        assert np.array_equal(got.cpu().numpy().reshape(pixels, patches), want.astype(np.float32))
    for x in store:  # nothing outside the cubes
        assert (x[:offset] == -7.0).all() and (x[offset + n:] == -7.0).all()
