"""Trees built on the GPU, from points in path order (no creator tables) and
from shuffled ones, at the sizes where a warp's, a block's or a chunk's points
end: node arrays equal the host producer's, and the leaf boxes equal those
built for the same array uploaded: every ray's visit count depends on them."""
import numpy as np
import pytest

from conftest import S

pytestmark = pytest.mark.gpu


def _points(n, levels, rng, order):
    # clusters with duplicates, so that chains, branches and equal cells occur
    c = rng.uniform(0.0, S, (max(n // 20, 1), 3))
    p = c[rng.integers(0, c.shape[0], n)] + rng.normal(size=(n, 3)) * S * rng.choice([0.0, 1e-3, 0.1], (n, 1))
    p = np.clip(p, 0.0, np.nextafter(np.float32(S), np.float32(0.0))).astype(np.float32)
    if order == "shuffled":
        return p
    from oracle import qbo
    o = qbo.point_octets(p, S, levels).astype(np.int64)
    key = np.zeros(n, np.int64)
    for k in range(levels):
        key = key * 8 + o[:, k]
    idx = np.argsort(key, kind="stable")
    if order == "one out":  # in path order but for one point
        idx[[0, n // 2]] = idx[[n // 2, 0]]
    return p[idx]


@pytest.mark.parametrize("order", ["sorted", "one out", "shuffled"])
@pytest.mark.parametrize("n,levels", [(1, 1), (1, 17), (2, 3), (31, 12), (32, 5), (33, 12), (2047, 12), (2048, 9),
                                      (2049, 16), (6000, 2), (6000, 12), (20000, 17), (3000, 21)])
def test_built_tree_and_boxes(oracle, n, levels, order):
    import qubatron_gb300 as qb
    rng = np.random.default_rng(n + levels)
    p = _points(n, levels, rng, order)
    nodes = qb.build_octree(p, S, levels)
    pos = rng.uniform(0.0, S, (3000, 3)).astype(np.float32)
    d = (p[rng.integers(0, n, 3000)] - pos).astype(np.float32)
    base = (0.0, S, S, S)
    with qb.OctreeGLC(0) as up:
        up.upload_octree(False, nodes)
        want = up.trace_rays(pos, d, base, min(levels, 17))
    for dynamic in (False, True):
        with qb.OctreeGLC(0) as ctx:
            for _ in range(2):  # the second build reuses what the first left
                assert ctx.build_tree(dynamic, p, S, levels, first_index=0) == nodes.shape[0]
            assert np.array_equal(ctx.download_tree(dynamic), nodes), dynamic
            if not dynamic:
                got = ctx.trace_rays(pos, d, base, min(levels, 17))
                for k in ("status", "leaf", "visits"):
                    assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("n,levels", [(262143, 12), (262144, 5), (262144, 12), (300001, 9)])
def test_large_dynamic_tree(n, levels):
    """Around the size from which a few points go ahead of the others."""
    import qubatron_gb300 as qb
    p = _points(n, levels, np.random.default_rng(n), "shuffled")
    p[-1000:] = p[:1000]  # first made by the points that go ahead, and met last
    nodes = qb.build_octree(p, S, levels)
    with qb.OctreeGLC(0) as ctx:
        for _ in range(2):
            assert ctx.build_tree(True, p, S, levels, first_index=0) == nodes.shape[0]
            assert np.array_equal(ctx.download_tree(True), nodes)


def test_dynamic_tree_of_changing_size():
    """Scratch made for one size serves the smaller sizes, whose prefix sums
    have more chunks (up to 262144 points)."""
    import qubatron_gb300 as qb
    p = _points(300001, 8, np.random.default_rng(1), "shuffled")
    with qb.OctreeGLC(0) as ctx:
        for n in (300001, 262144, 262145, 257, 256, 1, 200000):
            nodes = qb.build_octree(p[:n], S, 8)
            assert ctx.build_tree(True, p[:n], S, 8, first_index=0) == nodes.shape[0]
            assert np.array_equal(ctx.download_tree(True), nodes), n


@pytest.mark.parametrize("kind", ["whole", "stubs", "twice", "outside", "root"])
@pytest.mark.parametrize("n,levels", [(1, 3), (40, 1), (700, 8), (5000, 12)])
def test_uploaded_boxes(oracle, kind, n, levels):
    """Boxes of uploaded arrays: childless nodes above the deepest level, and
    arrays that get none (a node with two parents, an index outside)."""
    import qubatron_gb300 as qb
    rng = np.random.default_rng(n)
    p = _points(n, levels, rng, "shuffled")
    nodes = qb.build_octree(p, S, levels).copy()
    if kind == "root":
        nodes = nodes[:1].copy()
        nodes[:, :8] = 0
    links = np.argwhere(nodes[:, :8] > 0)
    if kind == "stubs":
        for k in rng.integers(0, len(links), len(links) // 4):
            nodes[tuple(links[k])] = 0
    elif kind == "twice" and len(links) > 1:
        leaf = nodes[tuple(links[-1])]  # an edge to a leaf cell, given a second parent
        node, octet = links[len(links) // 2]
        if node != links[-1][0]:
            nodes[node, octet] = leaf
    elif kind == "outside":
        nodes[tuple(links[-1])] = nodes.shape[0] + 5
    pos = rng.uniform(0.0, S, (2000, 3)).astype(np.float32)
    d = (p[rng.integers(0, n, 2000)] - pos).astype(np.float32)
    one = np.full((1, 3), 0.5, np.float32)
    ref = oracle.trace_rays(oracle.Scene(nodes, one.repeat(n, 0), one.repeat(n, 0), boxes=True), (0.0, S, S, S), levels,
                            pos, d)
    with qb.OctreeGLC(0) as ctx:
        ctx.upload_octree(False, nodes)
        got = ctx.trace_rays(pos, d, (0.0, S, S, S), levels)
    for k in ("status", "leaf", "visits"):
        assert np.array_equal(got[k], ref[k]), k


@pytest.mark.parametrize("n,cells", [(1, 1), (33, 1), (257, 1), (4097, 7), (30000, 5000)])
def test_removals_with_duplicates(oracle, n, cells):
    """Many points of few leaves: the first in input order of each removes it."""
    import qubatron_gb300 as qb
    rng = np.random.default_rng(n)
    p = _points(6000, 9, rng, "shuffled")
    nodes = qb.build_octree(p, S, 9)
    shots = np.concatenate([p[rng.integers(0, cells, n)], rng.uniform(0.0, S, (n // 3, 3)).astype(np.float32)])
    want_nodes = nodes.copy()
    want = oracle.remove_points(want_nodes, shots, S, 9)
    with qb.OctreeGLC(0) as ctx:
        ctx.upload_octree(False, nodes)
        mod, octind, removed = ctx.remove_points(False, shots, S, 9)
        assert np.array_equal(ctx.download_tree(False)[:, :9], want_nodes[:, :9])
    assert np.array_equal(mod, want[0]) and np.array_equal(octind, want[1]) and removed == (want[0] >= 0).sum()
