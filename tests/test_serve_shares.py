"""The numerical rays an SM holds, by which the server shares the SMs: half as
many where a ray has the lanes of two time levels."""
from gray_b200 import api


def test_rays_per_sm():
    f = getattr(api.lib(), "_Z16dyst_rays_per_smb")  # internal: dyst_rays_per_sm(bool)
    assert (f(0), f(1)) == (96, 48)
