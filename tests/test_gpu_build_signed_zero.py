"""Builds over meshes with negative zeros among their coordinates (what rotations and mirrored meshes leave): the
boxes hold every triangle, so the closest hits are the oracle's."""
import numpy as np
import pytest

from test_gpu_build_edges import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [2, 8, 1])
@pytest.mark.parametrize("n", [200, 3000, 20000])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_hits_match_oracle(n, axis, width):
    import torch
    import oracle_binding
    from axomae_b200 import native
    rng = np.random.default_rng(n + axis)
    verts = (rng.uniform(-1, 1, (n, 1, 3)) + 0.3 * rng.normal(size=(n, 3, 3))).astype(np.float32)
    near = np.nonzero(rng.random(n) < 0.5)[0]  # half of the triangles have one vertex at the plane, the rest beside it
    verts[near, :, axis] = np.abs(verts[near, :, axis]) * rng.choice([-1, 1], (len(near), 1))
    verts[near, 0, axis] = np.float32(-0.0)
    scene = _scene(verts)
    m = 20000
    o = rng.uniform(-3, 3, (m, 3)).astype(np.float32)
    at = verts[rng.integers(0, len(verts), m)].mean(1) + 0.02 * rng.normal(size=(m, 3))
    d = at - o
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    p_ref, t_ref, _, _, _ = oracle_binding.OracleScene(scene).trace(o, d)
    to, td = torch.from_numpy(o).cuda(), torch.from_numpy(d).cuda()
    prim = torch.empty(m, dtype=torch.int32, device="cuda")
    t, u, v = (torch.empty(m, dtype=torch.float32, device="cuda") for _ in range(3))
    torch.cuda.synchronize()
    ctx = native.Context(0)
    try:
        ctx.upload(scene)
        ctx.build(width=width)
        ctx.trace(to.data_ptr(), td.data_ptr(), m, prim.data_ptr(), t.data_ptr(), u.data_ptr(), v.data_ptr())
    finally:
        ctx.close()
    p, tt = prim.cpu().numpy(), t.cpu().numpy()
    assert ((p >= 0) == (p_ref >= 0)).all()
    assert np.array_equal(tt[p >= 0], t_ref[p >= 0])
