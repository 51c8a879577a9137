"""Texture-unit bakes whose output lies over the source map: the map is read as it was before the call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ch", [3, 4])
@pytest.mark.parametrize("w,h,ow,oh,shift", [(64, 32, 64, 32, 0), (256, 128, 128, 64, 0), (64, 32, 256, 128, 0),
                                             (128, 64, 128, 64, 512), (128, 64, 128, 64, 128 * 64 * 4 - 4)])
def test_texunit_bake_over_its_map(w, h, ow, oh, shift, ch):
    """The output begins `shift` floats into the map: the same bits as into memory of its own."""
    import torch
    from axomae_b200 import native
    src = np.random.default_rng(w + ow).lognormal(0, 1, (h, w, ch)).astype(np.float32)
    n = shift + ow * oh * 4
    memory = torch.zeros(max(n, src.size), device="cuda")
    apart = torch.zeros(ow * oh * 4, device="cuda")
    c = native.Context(0)
    try:
        for out in (apart, memory[shift:n]):
            memory[:src.size] = torch.from_numpy(src).cuda().ravel()
            torch.cuda.synchronize()
            c.bake_irradiance_texunit(memory.data_ptr(), w, h, ch, ow, oh, 65, out.data_ptr())
    finally:
        c.close()
    assert torch.isfinite(apart).all() and (apart.view(-1, 4)[:, :3] > 0).all()
    assert torch.equal(apart, memory[shift:n])


def test_texunit_bake_of_a_pinned_host_map():
    """Memory that is not the GPU's own is copied: the same bits as the map in device memory."""
    import torch
    from axomae_b200 import native
    w, h, ow, oh = 128, 64, 64, 32
    src = torch.from_numpy(np.random.default_rng(3).lognormal(0, 1, (h, w, 4)).astype(np.float32))
    maps = [src.cuda(), src.pin_memory()]
    films = [torch.zeros((oh, ow, 4), device="cuda") for _ in maps]
    torch.cuda.synchronize()
    c = native.Context(0)
    try:
        for m, f in zip(maps, films):
            c.bake_irradiance_texunit(m.data_ptr(), w, h, 4, ow, oh, 33, f.data_ptr())
    finally:
        c.close()
    assert (films[0][..., :3] > 0).all() and torch.equal(films[0], films[1])
