"""A captured dynamic frame holds the addresses of the build's scratch and of
the tree's leaf-box records. When a call in between replaces one of them, while
everything else the frame depends on comes out equal again, the replay is
refused, and a new capture gives the eager frame."""
import numpy as np
import pytest

from conftest import LEVELS, S
from helpers import upload_scene
from test_gpu_dynamic_graph import Rig, _host, _outputs, _views, env  # noqa: F401 (a fixture)

pytestmark = pytest.mark.gpu


def _refused_then_equal(torch, ctx, rig, g, views, gbufs):
    import qubatron_gb300 as qb
    with pytest.raises(qb.QbcError) as e:
        g.launch()
    assert e.value.code == -4 and "qbc_graph_launch" in str(e.value)
    g.update(views)
    rig.pose(torch, 3)
    g.launch()
    ctx.synchronize()
    replay = _host(gbufs)
    ebufs, eouts = _outputs(torch, views)
    ctx.dynamic_update(rig.update)
    ctx.render_views(views, eouts, on_device=True)
    ctx.synchronize()
    for a, b in zip(replay, _host(ebufs)):
        for k in a:
            assert np.array_equal(a[k], b[k]), k


def test_scratch_replaced(env, floor50k_scene):  # noqa: F811
    """More points at few levels, whose nodes fit the tree's buffers: only the
    per-point scratch grows."""
    torch, ctx = env
    s = floor50k_scene
    upload_scene(ctx, s.nodes, s.colors, s.normals)
    rig, views = Rig(torch, ctx), _views()
    gbufs, gouts = _outputs(torch, views)
    rig.pose(torch, 0)
    g = ctx.graph_capture_dynamic(rig.update, views, gouts)
    try:
        g.launch()
        ctx.synchronize()
        more = np.random.default_rng(0).uniform(0.0, S * 0.99, (2 * rig.n, 3)).astype(np.float32)
        ctx.build_tree(True, more, S, 3)
        ctx.dynamic_update(rig.update)
        _refused_then_equal(torch, ctx, rig, g, views, gbufs)
    finally:
        g.close()


def test_records_replaced(env, floor50k_scene):  # noqa: F811
    """The walk without boxes names no records, but the build writes them: an
    uploaded tree's larger ones take their place."""
    torch, ctx = env
    import qubatron_gb300 as qb
    s = floor50k_scene
    upload_scene(ctx, s.nodes, s.colors, s.normals)
    p = np.random.default_rng(1).uniform(0.0, S * 0.99, (60_000, 3)).astype(np.float32)
    big = qb.build_octree(p, S, LEVELS)
    ctx.upload_octree(True, big)
    rig, views = Rig(torch, ctx, n=2000), _views()
    gbufs, gouts = _outputs(torch, views)
    rig.pose(torch, 0)
    ctx.set_option(qb._lib.OPT_BOX_PRUNE, 0)
    g = ctx.graph_capture_dynamic(rig.update, views, gouts)
    try:
        g.launch()
        ctx.synchronize()
        ctx.upload_octree(True, big)
        ctx.set_option(qb._lib.OPT_BOX_PRUNE, 1)
        bufs, outs = _outputs(torch, views)
        ctx.render_views(views, outs, on_device=True)
        ctx.set_option(qb._lib.OPT_BOX_PRUNE, 0)
        ctx.dynamic_update(rig.update)
        _refused_then_equal(torch, ctx, rig, g, views, gbufs)
    finally:
        g.close()


def test_failed_update_keeps_the_refusal(env, floor50k_scene):  # noqa: F811
    """An update that fails leaves the frame captured before, and with it the
    refusal to replay it in the changed state."""
    torch, ctx = env
    import qubatron_gb300 as qb
    L = qb._lib
    s = floor50k_scene
    upload_scene(ctx, s.nodes, s.colors, s.normals)
    views = _views()
    _, outs = _outputs(torch, views)
    ctx.render_views_ex(views, outs, True, two_pass=True, log=True)
    g = ctx.graph_capture(views, outs, two_pass=True, proposals=L.PROPOSE_LOGGED)
    try:
        g.launch()
        ctx.render_views_ex(views[:1], outs[:1], True, two_pass=True, log=True)  # the log is of other views now
        ctx.set_option(L.OPT_SERVICE_MIN, 7)
        with pytest.raises(qb.QbcError):
            g.update(views)
        with pytest.raises(qb.QbcError) as e:
            g.launch()
        assert e.value.code == -4 and "qbc_graph_launch" in str(e.value)
        ctx.render_views_ex(views, outs, True, two_pass=True, log=True)
        g.update(views)
        g.launch()
        ctx.synchronize()
    finally:
        g.close()


def test_failed_update_keeps_the_tree(env, floor50k_scene):  # noqa: F811
    """... and the dynamic tree uploaded since, which the recorded update would
    have replaced: its node count and its frames are still those."""
    torch, ctx = env
    import qubatron_gb300 as qb
    L = qb._lib
    s = floor50k_scene
    upload_scene(ctx, s.nodes, s.colors, s.normals)
    p = np.random.default_rng(4).uniform(0.3 * S, 0.7 * S, (40_000, 3)).astype(np.float32)
    big = qb.build_octree(p, S, LEVELS)
    ctx.upload_octree(True, big)  # the tree's buffers hold it from now on
    rig, views = Rig(torch, ctx, n=2000), _views()
    _, outs = _outputs(torch, views)
    rig.pose(torch, 0)
    ctx.dynamic_update(rig.update)
    ctx.render_views_ex(views, outs, True, two_pass=True, log=True)
    g = ctx.graph_capture_dynamic(rig.update, views, outs, two_pass=True, proposals=L.PROPOSE_LOGGED)
    try:
        ctx.upload_model(True, rig.ch.colors[:1].repeat(40_000, 0), rig.ch.rest_normals[:1].repeat(40_000, 0))
        ctx.upload_octree(True, big)
        want = [f.arrays for f in ctx.render_host(views, ("rgba8", "flags", "leaf"))]
        ctx.render_views_ex(views[:1], outs[:1], True, two_pass=True, log=True)  # the log is of other views now
        with pytest.raises(qb.QbcError):
            g.update(views)
        assert ctx.tree_nodes(1) == big.shape[0] and ctx.model_points(1) == 40_000
        got = [f.arrays for f in ctx.render_host(views, ("rgba8", "flags", "leaf"))]
        for a, b in zip(got, want):
            for k in a:
                assert np.array_equal(a[k], b[k]), k
    finally:
        g.close()
