"""Frames whose paths do not fit the radiance buffer at once (more than 4 GiB of 16-byte values): rendered
in chunks, the film has the bits of the same samples rendered by calls that each fit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp", [(1024, 1024, 257), (1000, 999, 275), (7000, 7200, 6)])
def test_chunked_frame_equals_its_samples_in_calls(w, h, spp):
    from axomae_b200 import native, scenes
    s = scenes.spheres_scene(64, 64, n_spheres=8, seed=1)
    c = native.Context(0)
    try:
        c.upload(s)
        c.build()
        whole, parts = (np.zeros((h, w, 4), np.float32) for _ in range(2))
        assert w * h * spp * 16 > 4 << 30
        c.render(native.make_frame(s, w, h, spp, 2), film_host=whole)
        step = (spp + 3) // 4
        for b in range(0, spp, step):
            c.render(native.make_frame(s, w, h, spp, 2, sample_begin=b, sample_count=min(step, spp - b), reset=b == 0),
                     film_host=parts)
        assert np.array_equal(whole.view(np.uint32), parts.view(np.uint32))
    finally:
        c.close()
