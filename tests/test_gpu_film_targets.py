"""Where a render's films go: device buffers shared by the frames of a batch, each frame with its film in
host memory too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(40, 40), (64, 48), (24, 24)]


@pytest.fixture(scope="module")
def batch():
    from axomae_b200 import native, scenes
    ctxs, frames, alone = [], [], []
    for k, (w, h) in enumerate(SIZES):
        scene = scenes.spheres_scene(w, h, n_spheres=4 + k, seed=k)
        c = native.Context(0)
        c.upload(scene)
        c.build()
        film = np.zeros((h, w, 4), np.float32)
        frames.append(native.make_frame(scene, w, h, 2, 4, seed=k))
        c.render(frames[-1], film_host=film)
        ctxs.append(c)
        alone.append(film)
    yield ctxs, frames, alone
    for c in ctxs:
        c.close()


@pytest.mark.parametrize("offsets", [(0, 0, 0), (0, 1600, 900), (0, 20000, 20000 + 4 * 64 * 48 - 4)])
def test_frames_that_share_a_device_film(batch, offsets):
    """Every host film is its own frame's; the device memory holds the films in the order of the frames,
    later ones over earlier ones."""
    import torch
    from axomae_b200 import native
    ctxs, frames, alone = batch
    dev = torch.full((40000,), -1.0, device="cuda")
    want = np.full(40000, -1.0, np.float32)
    for off, film in zip(offsets, alone):
        want[off:off + film.size] = film.ravel()
    host = [np.zeros_like(film) for film in alone]
    torch.cuda.synchronize()
    native.render_batch(ctxs, frames, films_host=host, films_device=[dev.data_ptr() + 4 * off for off in offsets])
    for got, film in zip(host, alone):
        assert np.array_equal(got.view(np.uint32), film.view(np.uint32))
    assert np.array_equal(dev.cpu().numpy().view(np.uint32), want.view(np.uint32))
