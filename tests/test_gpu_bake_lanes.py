"""Every lane count of the two bakes (1, 2, 4 and 8 lanes per output texel, by the texels' number), with sample
counts that leave a group partly empty, against the oracle (rtol 1e-4 for the CPU bake, as in
test_bake_matches_oracle)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FILL = 148 * 2048  # threads that the GPU holds
SIZES = [(256, 256), (512, 256), (512, 512), (1024, 512), (1024, 1024)]


@pytest.fixture(scope="module")
def ctx():
    from axomae_b200 import native
    c = native.Context(0)
    yield c
    c.close()


def test_sizes_reach_every_lane_count():
    """The rules: the fewest lanes that fill the GPU once (CPU bake) and twice (texture unit)."""
    for fill in (FILL, 2 * FILL):
        assert {next(g for g in (1, 2, 4, 8) if g == 8 or w * h * g >= fill) for w, h in SIZES} == {1, 2, 4, 8}


@pytest.mark.parametrize("ow,oh", SIZES)
@pytest.mark.parametrize("samples", [1, 5])
def test_bake(ctx, ow, oh, samples):
    import torch
    import oracle_binding
    src = np.random.default_rng(ow + samples).lognormal(0, 1, (21, 43, 4)).astype(np.float32)
    ts, out = torch.from_numpy(src).cuda(), torch.zeros((oh, ow, 4), device="cuda")
    torch.cuda.synchronize()
    ctx.bake_irradiance(ts.data_ptr(), 43, 21, 4, ow, oh, samples, out.data_ptr())
    ref = np.asarray(oracle_binding.bake_irradiance(src, ow, oh, samples)).reshape(oh, ow, -1)
    np.testing.assert_allclose(out.cpu().numpy()[..., :3], ref[..., :3], rtol=1e-4, atol=1e-6)


@pytest.mark.parametrize("ow,oh", SIZES)
@pytest.mark.parametrize("samples", [1, 5])
def test_texunit_bake(ctx, ow, oh, samples):
    """A filter weight of the texture unit has 8 fractional bits, and rounding in the trigonometry may move each of
    the two by one step: 2 / 256 of the map's range a sample, so as much of their mean, where one sample
    lost or counted twice is a tenth of the range at least.  At a pole the azimuth is all rounding: one texel in
    10,000 is left out."""
    import torch
    import oracle_binding
    src = np.random.default_rng(ow + samples).uniform(0.5, 1.5, (21, 43, 4)).astype(np.float32)
    ts, out = torch.from_numpy(src).cuda(), torch.zeros((oh, ow, 4), device="cuda")
    torch.cuda.synchronize()
    ctx.bake_irradiance_texunit(ts.data_ptr(), 43, 21, 4, ow, oh, samples, out.data_ptr())
    ref = np.asarray(oracle_binding.bake_irradiance_texunit(src, ow, oh, samples)).reshape(oh, ow, 4)
    dev = out.cpu().numpy()
    assert (dev[..., 3] == 1.0).all()
    assert (np.abs(dev[..., :3] - ref[..., :3]).max(-1) <= 2.0 / 256 + 1e-5).mean() >= 0.9999
