"""The kernel that finishes a draining wavefront, at the sizes around its limit (150,000 rays) and on every
BVH width: films bit for bit, and gradients up to the order of their atomic sums, against the waves
alone (trace_mode 2 keeps every ray in them)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _emissive(scene):
    from axomae_b200 import scenes
    scene = dict(scene, textures=list(scene["textures"]), materials=[dict(m) for m in scene["materials"]])
    scene["textures"].append(scenes.solid_u8((0.3, 0.2, 0.1)))
    scene["materials"][1]["emissive"] = len(scene["textures"]) - 1
    return scene


@pytest.mark.parametrize("width", [1, 2, 8])
@pytest.mark.parametrize("w,h,spp,depth,rr,emissive", [(1, 1, 1, 0, -1, False), (33, 17, 3, 6, 2, True),
                                                       (387, 387, 1, 5, -1, False), (388, 388, 1, 5, 1, True),
                                                       (300, 301, 2, 12, -1, False)])
def test_films_equal_the_waves(width, w, h, spp, depth, rr, emissive):
    from axomae_b200 import native, scenes
    s = scenes.mixed_scene(8000, w, h, seed=6)
    s = _emissive(s) if emissive else s
    c = native.Context(0)
    try:
        c.upload(s)
        c.build(width=width)
        fr = native.make_frame(s, w, h, spp, depth, rr_start=rr)
        films, stats = [], []
        for tuning in (dict(), dict(trace_mode=2), dict(queue_capacity=65536)):
            c.set_tuning(**tuning) if tuning else c.set_tuning()
            film = np.zeros((h, w, 4), np.float32)
            stats.append(c.render(fr, film_host=film))
            films.append(film)
        assert np.array_equal(films[0].view(np.uint32), films[1].view(np.uint32))
        assert np.array_equal(films[0].view(np.uint32), films[2].view(np.uint32))
        assert stats[0].traced == stats[1].traced == stats[2].traced
        assert stats[0].waves == stats[1].waves
    finally:
        c.close()


@pytest.mark.parametrize("w,h,spp", [(8, 5, 1), (387, 387, 1), (200, 200, 5)])
def test_gradients_equal_the_waves(w, h, spp):
    import torch
    from axomae_b200 import native, scenes
    s = scenes.spheres_scene(w, h, n_spheres=12, seed=3)
    c = native.Context(0)
    try:
        c.upload(s)
        c.build()
        n, m = c.info()["triangles"], len(s["materials"])
        gen = torch.Generator(device="cuda").manual_seed(1)
        alb = torch.rand((n, 3), generator=gen, device="cuda") * 0.6 + 0.2
        rough = torch.rand((m,), generator=gen, device="cuda") * 0.7 + 0.2
        d_img = torch.randn((h, w, 4), generator=gen, device="cuda")
        torch.cuda.synchronize()
        fr = native.make_frame(s, w, h, spp, 5)
        c.set_diff_params(alb.data_ptr(), rough.data_ptr())
        out = []
        for tuning in (dict(), dict(trace_mode=2)):
            c.set_tuning(**tuning) if tuning else c.set_tuning()
            ga, gr = torch.zeros_like(alb), torch.zeros_like(rough)
            torch.cuda.synchronize()
            c.backward(fr, d_img.data_ptr(), ga.data_ptr(), gr.data_ptr())
            out.append((ga.cpu().numpy(), gr.cpu().numpy()))
        for a, b in zip(out[0], out[1]):
            # the same terms summed in another order: a few thousand float additions each
            np.testing.assert_allclose(a, b, rtol=1e-3, atol=1e-4 * max(1e-6, float(np.abs(b).max())))
    finally:
        c.close()
