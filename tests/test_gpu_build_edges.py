"""BVH builds at the sizes where a subtree changes hands (one primitive, one warp's 32, one CTA's 256, the
level kernels above) and on shapes without a binned split: closest hits against the oracle, whose own
tree is built another way, so only exact ties may differ."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(verts):
    """Independent triangles (n, 3, 3) as one mesh over a constant environment."""
    from axomae_b200 import scenes
    n = verts.shape[0]
    b = scenes._Builder()
    v = verts.reshape(-1, 3).astype(np.float32)
    up = np.tile([0, 1, 0], (3 * n, 1)).astype(np.float32)
    t = np.tile([1, 0, 0], (3 * n, 1)).astype(np.float32)
    uv = np.tile([[0, 0], [1, 0], [0, 1]], (n, 1)).astype(np.float32)
    b.add({"vertices": v, "normals": up, "tangents": t, "bitangents": np.cross(up, t).astype(np.float32), "uv": uv,
           "indices": np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)}, b.lambert((0.5, 0.5, 0.5)))
    env = b.tex(scenes.f32_texture(np.ones((2, 2, 4), np.float32)))
    return b.finish(env, scenes.camera((0.0, 0.0, 5.0), (0.0, 0.0, 0.0), 16, 16))


def _triangles(shape, n, rng):
    size = 0.2 * rng.normal(size=(n, 3, 3))
    if shape == "uniform":
        return rng.uniform(-3, 3, (n, 1, 3)) + size
    if shape == "same":  # every centroid equal: median splits at each level
        return np.tile(rng.normal(size=(1, 3, 3)), (n, 1, 1))
    # positions growing by a factor: each split takes a few primitives off one end, so the tree is deep
    x = 1.01 ** np.arange(n) * 1e-3
    return np.stack([x, np.zeros(n), np.zeros(n)], -1)[:, None, :] + size * x[:, None, None]


@pytest.mark.parametrize("shape", ["uniform", "same", "growing"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 256, 257, 1025, 3000])
def test_hits_match_oracle_at_subtree_sizes(shape, n):
    import torch
    import oracle_binding
    from axomae_b200 import native
    rng = np.random.default_rng(n)
    verts = _triangles(shape, n, rng)
    scene = _scene(verts)
    m = 4000
    o = rng.uniform(-4, 4, (m, 3)).astype(np.float32)
    at = verts.reshape(n, 3, 3)[rng.integers(0, n, m)].mean(1) + 0.02 * rng.normal(size=(m, 3))
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
        for small in (0, 64):
            ctx.build(small_subtree=small)
            info = ctx.info()
            assert info["leaves"] == info["nodes"] + 1 or (n == 1 or info["leaves"] == 1 and info["nodes"] == 1)
            ctx.trace(to.data_ptr(), td.data_ptr(), m, prim.data_ptr(), t.data_ptr(), u.data_ptr(), v.data_ptr())
            p, tt = prim.cpu().numpy(), t.cpu().numpy()
            assert ((p >= 0) == (p_ref >= 0)).all()
            hit = p >= 0
            # the closest distance is the reference's; another primitive only at exactly that distance
            assert np.array_equal(tt[hit], t_ref[hit])
    finally:
        ctx.close()
