"""A batch whose paths do not fit the radiance buffer at once (more than 4 GiB of 16-byte values): its films have
the bits of the frames rendered alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batch_beyond_the_radiance_buffer():
    from axomae_b200 import native, scenes
    sizes = [(1024, 1024, 120), (1000, 900, 90), (700, 1200, 110)]
    assert sum(w * h * spp for w, h, spp in sizes) * 16 > 4 << 30
    ctxs, frames, alone = [], [], []
    try:
        for k, (w, h, spp) in enumerate(sizes):
            scene = scenes.spheres_scene(64, 64, n_spheres=4 + k, seed=k)
            c = native.Context(0)
            ctxs.append(c)
            c.upload(scene)
            c.build()
            frames.append(native.make_frame(scene, w, h, spp, 2, seed=k))
            alone.append(np.zeros((h, w, 4), np.float32))
            c.render(frames[-1], film_host=alone[-1])
        films = [np.zeros_like(f) for f in alone]
        native.render_batch(ctxs, frames, films_host=films)
    finally:
        for c in ctxs:
            c.close()
    for a, b in zip(films, alone):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
