"""The key that ties a scene's walk words to their step table."""
import ctypes

import numpy as np


def test_keys_differ_with_the_table():
    from solweig_cuda_b200 import _lib, rays
    L = _lib.lib()
    keys = {}
    for scale in (1.0, 0.5, 0.25, 2.0):
        dxdy, first, second = rays.gvf_offsets(scale)
        ptr = dxdy.ctypes.data_as(ctypes.c_void_p)
        key = L.solweig_gvf_table_key(ptr, first, second)
        assert key and key == L.solweig_gvf_table_key(ptr, first, second)
        keys[scale, first, second] = key
        changed = dxdy.copy()
        changed[17, second - 1, 1] += 1
        keys[scale, "changed"] = L.solweig_gvf_table_key(changed.ctypes.data_as(ctypes.c_void_p), first, second)
        if second > 1:  # the same memory read as a shorter walk
            keys[scale, "shorter"] = L.solweig_gvf_table_key(ptr, first, second - 1)
    assert len(set(keys.values())) == len(keys)
    assert L.solweig_gvf_table_key(None, 1, 22) == 0
    dxdy = np.zeros((18, 1, 2), dtype=np.int32)
    assert L.solweig_gvf_table_key(dxdy.ctypes.data_as(ctypes.c_void_p), 1, 0) == 0
    assert L.solweig_gvf_table_key(dxdy.ctypes.data_as(ctypes.c_void_p), 1, 1) != 0
