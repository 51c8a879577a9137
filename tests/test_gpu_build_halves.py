"""Builds over triangles whose boxes share one centre, so every split is a halving by position, for different
sizes at which a subtree passes to one thread block: the trees may differ, the closest hits may not."""
import numpy as np
import pytest

from test_gpu_build_edges import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [2, 8, 1])
@pytest.mark.parametrize("n", [40, 300, 2000])
def test_hits_do_not_depend_on_the_subtree_size(n, width):
    import torch
    import oracle_binding
    from axomae_b200 import native
    rng = np.random.default_rng(n)
    a = rng.uniform(0.05, 1.5, (n, 3)) * rng.choice([-1, 1], (n, 3))
    verts = np.stack([a, -a, a * rng.uniform(-1, 1, (n, 3))], 1).astype(np.float32)  # boxes -|a| .. |a|
    box = verts.min(1) + verts.max(1)
    assert (box == 0).all()
    scene = _scene(verts)
    m = 4000
    o = rng.uniform(-4, 4, (m, 3)).astype(np.float32)
    d = rng.uniform(-1, 1, (m, 3)) - o
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    p_ref, t_ref, _, _, _ = oracle_binding.OracleScene(scene).trace(o, d)
    assert (p_ref >= 0).mean() > 0.2
    to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    prim = torch.empty(m, dtype=torch.int32, device="cuda")
    t, u, v = (torch.empty(m, dtype=torch.float32, device="cuda") for _ in range(3))
    torch.cuda.synchronize()
    ctx = native.Context(0)
    try:
        ctx.upload(scene)
        for small in (64, 256, 65536):
            ctx.build(width=width, small_subtree=small)
            ctx.trace(to.data_ptr(), td.data_ptr(), m, prim.data_ptr(), t.data_ptr(), u.data_ptr(), v.data_ptr())
            p, tt = prim.cpu().numpy(), t.cpu().numpy()
            assert ((p >= 0) == (p_ref >= 0)).all()
            assert np.array_equal(tt[p >= 0], t_ref[p >= 0])
    finally:
        ctx.close()
