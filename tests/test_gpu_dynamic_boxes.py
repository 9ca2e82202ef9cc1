"""Leaf boxes of dynamic trees built on the GPU: every ray's visit counts
equal those on the same array uploaded, whose boxes boxes.cu makes, at the
sizes where a warp's, a block's or a chunk's points end, from which points go
ahead of the others, and with scratch left by builds of other sizes."""
import numpy as np
import pytest

from conftest import S
from test_gpu_build_boxes import _points

pytestmark = pytest.mark.gpu

BASE = (0.0, S, S, S)
ROOT_ONLY = np.zeros((1, 12), np.int32)


def _rays(p, n, rng):
    pos = rng.uniform(0.0, S, (n, 3)).astype(np.float32)
    return pos, (p[rng.integers(0, p.shape[0], n)] - pos).astype(np.float32)


def _check(ctx, up, p, levels, rng):
    """Tree 1 of ctx built from p, against the host producer's array in up."""
    import qubatron_gb300 as qb
    nodes = qb.build_octree(p, S, levels)
    assert ctx.build_tree(True, p, S, levels, first_index=0) == nodes.shape[0]
    assert np.array_equal(ctx.download_tree(True), nodes)
    up.upload_octree(True, nodes)
    pos, d = _rays(p, 3000, rng)
    got, want = (c.trace_rays(pos, d, BASE, min(levels, 17)) for c in (ctx, up))
    for k in ("status", "leaf", "visits"):
        assert np.array_equal(got[k], want[k]), (k, p.shape[0], levels)
    assert (want["visits"][:, 1] > 0).any()


@pytest.fixture
def pair():
    import qubatron_gb300 as qb
    with qb.OctreeGLC(0) as ctx, qb.OctreeGLC(0) as up:
        for c in (ctx, up):
            c.upload_octree(False, ROOT_ONLY)
        yield ctx, up


@pytest.mark.parametrize("order", ["sorted", "shuffled"])
@pytest.mark.parametrize("n,levels", [(1, 1), (1, 17), (2, 3), (31, 12), (32, 5), (33, 12), (2047, 12), (2048, 9),
                                      (2049, 16), (6000, 2), (20000, 17), (262143, 12), (262144, 5), (300001, 9)])
def test_built_dynamic_boxes(oracle, pair, n, levels, order):
    rng = np.random.default_rng(n + levels)
    p = _points(n, levels, rng, order)
    for _ in range(2):  # the second build reuses what the first left
        _check(*pair, p, levels, rng)


def test_boxes_after_other_sizes(pair):
    rng = np.random.default_rng(2)
    p = _points(300001, 12, rng, "shuffled")
    for n, levels in ((300001, 12), (257, 12), (262144, 8), (1, 3), (200000, 12), (33, 17), (262145, 5)):
        _check(*pair, p[:n], levels, rng)


@pytest.mark.parametrize("n,levels", [(40, 2), (700, 8), (5000, 12)])
def test_two_parents_leave_no_boxes(oracle, n, levels):
    """A node reached from two parents rules the boxes out: the walk is the
    shader's, visit counts included."""
    import qubatron_gb300 as qb
    rng = np.random.default_rng(n)
    nodes = qb.build_octree(_points(n, levels, rng, "shuffled"), S, levels).copy()
    links = np.argwhere(nodes[:, :8] > 0)
    leaf = nodes[tuple(links[-1])]  # an edge to a leaf cell, given a second parent
    node, octet = links[len(links) // 2]
    assert node != links[-1][0] and nodes[node, octet] != leaf
    nodes[node, octet] = leaf
    pos = rng.uniform(0.0, S, (2000, 3)).astype(np.float32)
    d = rng.normal(size=(2000, 3)).astype(np.float32)
    with qb.OctreeGLC(0) as ctx:
        ctx.upload_octree(False, nodes)
        got = ctx.trace_rays(pos, d, BASE, levels)
        ctx.set_option(qb._lib.OPT_BOX_PRUNE, 0)
        plain = ctx.trace_rays(pos, d, BASE, levels)
    for k in ("status", "leaf", "visits"):
        assert np.array_equal(got[k], plain[k]), k
