"""The constants of the sky rays for whatever the patch option is given as."""
import numpy as np
import pytest


@pytest.mark.parametrize("option", [1, 2])
def test_the_option_is_read_as_a_number(option):
    import torch
    from solweig_cuda_b200 import rays
    want = rays.svf_ray_constants(option)
    for given in (float(option), np.int64(option), np.array(option), str(option), torch.tensor(option)):
        got = rays.svf_ray_constants(given)
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
        assert rays.svf_ray_capacity(given, (30, 40), 20.0, 1.0) == rays.svf_ray_capacity(option, (30, 40), 20.0, 1.0)


def test_a_changed_option_is_another_one():
    import torch
    from solweig_cuda_b200 import rays
    option = torch.tensor(1)
    first = rays.svf_ray_constants(option)[1].size
    option.fill_(2)
    assert (first, rays.svf_ray_constants(option)[1].size) == (145, 153)


def test_the_kept_constants_cannot_be_written():
    from solweig_cuda_b200 import rays
    for a in rays.svf_ray_constants(2):
        with pytest.raises(ValueError):
            a[..., 0] = 0
