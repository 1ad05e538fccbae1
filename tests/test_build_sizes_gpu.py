"""GPU builds at the sizes where the builder changes kernels: leaves (1 to 3
primitives), nodes whose references each try their own plane (up to 32), nodes
binned in one block (up to 512) and by blocks of 1,024 references, each side of
the limit, and nodes whose centroids coincide (split by position). Both drivers; hits against
the brute-force oracle, bit for bit but for exact ties."""
import numpy as np
import pytest

import oracle
from alpine_b200 import gpu, scenes
from parity import compare_closest

pytestmark = pytest.mark.gpu


def _soup(n, kind):
    verts, idx = scenes.triangle_soup(n, seed=n, mu=np.log(0.08))
    v = verts.reshape(n, 3, 3)
    if kind == "line":  # centroids on one axis: the other two have no extent
        v -= v.mean(1, keepdims=True)
        v = (np.round(v * 1024) / 1024).astype(np.float32)
        box = 0.5 * (v.min(1) + v.max(1))
        v += (np.stack([np.linspace(0.1, 0.9, n), np.full(n, 0.5), np.full(n, 0.5)], 1) - box)[:, None, :].astype(np.float32)
    elif kind == "stacks":  # groups of coincident triangles
        v = np.repeat(v[:: max(1, n // 3)], n, axis=0)[:n] if n < 4 else v[np.sort(np.arange(n) % 3)]
    return np.ascontiguousarray(v, np.float32).reshape(-1, 3), idx


@pytest.mark.parametrize("kind", ["soup", "line", "stacks"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 31, 32, 33, 63, 64, 65, 255, 256, 257, 511, 512, 513, 1023, 1025, 2049])
def test_sizes_around_the_builders_limits(n, kind):
    verts, idx = _soup(n, kind)
    tris = oracle.make_tris(verts, idx)
    rays = np.concatenate([scenes.primary_rays(48, 24), scenes.incoherent_rays(800, seed=n)])
    ref = oracle.closest_brute(rays, tris)[:4]
    ctx = gpu.Context(0)
    try:
        ctx.add_mesh(verts, idx)
        for rule in (gpu.COLLAPSE_SAH, gpu.COLLAPSE_GREEDY):
            ctx.set_build_options(rule)
            st = ctx.build()
            # a binary tree whose leaves hold one to three of the n triangles
            leaves = (st["binary_nodes"] + 1) // 2
            assert st["binary_nodes"] % 2 == 1 and -(-n // 3) <= leaves <= n
            hits = ctx.trace(rays)
            compare_closest(rays, tris, hits, *ref)
            assert (ctx.occluded(rays) == oracle.any_brute(rays, tris)).all()
            ctx.build_async()
            ctx.synchronize()
            assert ctx.trace(rays).tobytes() == hits.tobytes()
    finally:
        ctx.close()


@pytest.mark.parametrize("growth", [1.03, 1.04, 1.05])
def test_boxes_whose_areas_overflow(growth):
    """Nested triangles up to 1.05^1500 across: where the SAH costs overflow,
    nodes are halved by position, and the tree stays within the traversal's
    stack under both collapse rules."""
    n = 60000
    base = np.array([[0, 0, 0], [1, 0, 0.1], [0.2, 1, 0.3]], np.float32) - np.float32(0.4)
    v = (base[None] * (growth ** (np.arange(n) % 1500))[:, None, None]).astype(np.float32)
    verts, idx = v.reshape(-1, 3), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    rays = scenes.incoherent_rays(300, seed=12)
    tris = oracle.make_tris(verts, idx)
    ref = oracle.closest_brute(rays, tris)[:4]
    ctx = gpu.Context(0)
    try:
        ctx.add_mesh(verts, idx)
        for rule in (gpu.COLLAPSE_SAH, gpu.COLLAPSE_GREEDY):
            ctx.set_build_options(rule)
            ctx.build()
            compare_closest(rays, tris, ctx.trace(rays), *ref)
            ctx.build_async()
            ctx.synchronize()
            compare_closest(rays, tris, ctx.trace(rays), *ref)
    finally:
        ctx.close()
