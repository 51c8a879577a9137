"""The bakes' size rules: lanes per texel (1 to 8), sample counts that leave a ragged last group, the map
with and without non-finite texels, and the three ways a map becomes a texture.  References: the
oracle's CPU bake (rtol 1e-4, as in test_bake_matches_oracle), or the same bake by another route."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from axomae_b200 import native
    c = native.Context(0)
    yield c
    c.close()


def _map(rng, h, w, ch):
    return rng.lognormal(0, 1, (h, w, ch)).astype(np.float32)


@pytest.mark.parametrize("ow,oh,samples", [(1, 1, 1), (8, 4, 7), (64, 32, 33), (256, 256, 9), (512, 512, 3), (1024, 1024, 2)])
@pytest.mark.parametrize("ch", [3, 4])
@pytest.mark.parametrize("bad", [None, np.inf, np.nan])
def test_bake_lanes_and_nonfinite_maps(ctx, ow, oh, samples, ch, bad):
    import torch
    import oracle_binding
    rng = np.random.default_rng(ow + samples)
    src = _map(rng, 19, 37, ch)
    if bad is not None:
        src[7, 11, 1] = bad
    out = torch.zeros((oh, ow, ch), dtype=torch.float32, device="cuda")
    ts = torch.from_numpy(src).cuda()
    torch.cuda.synchronize()
    ctx.bake_irradiance(ts.data_ptr(), 37, 19, ch, ow, oh, samples, out.data_ptr())
    ref = oracle_binding.bake_irradiance(src, ow, oh, samples)
    np.testing.assert_allclose(out.cpu().numpy()[..., :3], np.asarray(ref).reshape(oh, ow, -1)[..., :3], rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("w,h", [(64, 32), (63, 17), (1, 1)])
@pytest.mark.parametrize("ow,oh,samples", [(4, 2, 5), (256, 256, 9), (1024, 512, 3)])
def test_texunit_bake_does_not_depend_on_where_the_map_lies(ctx, w, h, ow, oh, samples):
    """RGBA at an aligned address (read in place when its rows are aligned too), at one 16 bytes on
    (copied), and RGB (widened): equal bit for bit."""
    import torch
    rng = np.random.default_rng(w + ow)
    src = _map(rng, h, w, 4)
    flat = torch.zeros(h * w * 4 + 4, dtype=torch.float32, device="cuda")
    films = []
    for off, ch in ((0, 4), (4, 4), (0, 3)):
        data = torch.from_numpy(np.ascontiguousarray(src[..., :ch])).cuda().reshape(-1)
        flat[off:off + data.numel()] = data
        out = torch.zeros((oh, ow, 4), dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        ctx.bake_irradiance_texunit(flat.data_ptr() + 4 * off, w, h, ch, ow, oh, samples, out.data_ptr())
        films.append(out.cpu().numpy())
    assert (films[0][..., 3] == 1.0).all() and np.isfinite(films[0]).all()
    assert np.array_equal(films[0], films[1]) and np.array_equal(films[0], films[2])
