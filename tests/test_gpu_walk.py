"""The walk on t values (walker_fast.cuh) against the walk on the shader's
own arithmetic and the oracle, where the two come closest to differing: rays
through lattice points and along diagonals, which meet several bisecting
planes at one t, rays that graze cube edges by a few ulps, axis-parallel rays,
origins outside the basecube, and cameras on bisecting planes. Every output is
compared bit for bit, with and without a visits stream (two kernels)."""
import ctypes as C

import numpy as np
import pytest

from conftest import LEVELS, S
from helpers import bits, compare_frame, oracle_scene, upload_scene

pytestmark = pytest.mark.gpu

BASE = (0.0, S, S, S)


@pytest.fixture(scope="module")
def scene(lib):
    from qubatron_gb300 import scenes
    return scenes.make_scene(scenes.scaled_spec("room20m", 200_000))


@pytest.fixture(scope="module")
def character(lib):
    from qubatron_gb300 import build_octree, scenes
    ch = scenes.make_character(30_000)
    p, n = scenes.skin_reference(ch, scenes.pose_bones(ch, 3))
    return build_octree(p), ch.colors, n


def _rays(kind, n, rng):
    """n rays that meet planes of the octree together."""
    step = S / 2 ** rng.integers(1, LEVELS + 1, (n, 1))
    pos = np.round(rng.uniform(0.02 * S, 0.98 * S, (n, 3)) / step) * step
    if kind == "lattice":  # from lattice point to lattice point
        d = np.round(rng.uniform(0.0, S, (n, 3)) / step) * step - pos
    elif kind == "diagonal":  # equal components: all three planes at one t
        d = rng.choice([-1.0, 1.0], (n, 3)) * rng.uniform(0.5, 2.0, (n, 1))
    elif kind == "grazing":  # through a lattice line, off by a few ulps
        d = rng.choice([-1.0, 1.0], (n, 3)) * (1.0 + rng.integers(-4, 5, (n, 3)) * 2.0**-23)
        pos = pos * (1.0 + rng.integers(-2, 3, (n, 3)) * 2.0**-23)
    elif kind == "parallel":  # one or two zero components, or tiny ones
        d = rng.normal(size=(n, 3)) * rng.choice([0.0, 1e-7, 1.0], (n, 3), p=[0.3, 0.2, 0.5])
        d[:, 0] += (np.abs(d).sum(1) == 0.0)
    else:  # outside: towards lattice points from beyond the basecube
        out = rng.uniform(-1.5 * S, 2.5 * S, (n, 3))
        d = pos - out
        pos = out
    return pos.astype(np.float32), d.astype(np.float32)


def _trace(ctx, pos, d, visits):
    from qubatron_gb300 import _lib
    n = pos.shape[0]
    out = {"status": np.zeros(n, np.int32), "leaf": np.zeros((n, 2), np.int32), "model": np.zeros((n, 2), np.int32),
           "isp": np.zeros((n, 4), np.float32), "col": np.zeros((n, 4), np.float32),
           "nrm": np.zeros((n, 4), np.float32), "visits": np.zeros((n, 2), np.uint32)}
    h = _lib.RayHits(**{k: a.ctypes.data for k, a in out.items() if visits or k != "visits"})
    _lib.check(ctx._lib.qbc_trace_rays(ctx.handle, C.c_void_p(pos.ctypes.data), C.c_void_p(d.ctypes.data), n,
                                       (C.c_float * 4)(*BASE), LEVELS, C.byref(h), 0))
    return out


@pytest.mark.parametrize("two_trees", [False, True])
@pytest.mark.parametrize("kind", ["lattice", "diagonal", "grazing", "parallel", "outside"])
def test_rays(oracle, scene, character, kind, two_trees):
    import qubatron_gb300 as qb
    from qubatron_gb300 import _lib as L
    pos, d = _rays(kind, 30_000, np.random.default_rng(7))
    dyn = character if two_trees else (None, None, None)
    with qb.OctreeGLC(0) as ctx:
        upload_scene(ctx, scene.nodes, scene.colors, scene.normals, *dyn)
        plain, counted = _trace(ctx, pos, d, False), _trace(ctx, pos, d, True)
        ctx.set_option(L.OPT_BOX_PRUNE, 0)
        shader = _trace(ctx, pos, d, True)
    ref = oracle.trace_rays(oracle_scene(oracle, scene.nodes, scene.colors, scene.normals, *dyn, boxes=True), BASE,
                            LEVELS, pos, d)
    for k in ("status", "leaf", "model", "isp", "col", "nrm"):
        assert np.array_equal(bits(plain[k]), bits(shader[k])), k
        assert np.array_equal(bits(counted[k]), bits(shader[k])), k
    for k in ("status", "leaf", "model", "visits"):
        assert np.array_equal(counted[k], ref[k]), k


@pytest.mark.parametrize("two_trees", [False, True])
def test_cameras_on_bisecting_planes(oracle, scene, character, two_trees):
    import qubatron_gb300 as qb
    dyn = character if two_trees else (None, None, None)
    streams = ("rgba8", "rgba32f", "flags", "leaf", "isp")
    ref_scene = oracle_scene(oracle, scene.nodes, scene.colors, scene.normals, *dyn, boxes=True)
    with qb.OctreeGLC(0) as ctx:
        upload_scene(ctx, scene.nodes, scene.colors, scene.normals, *dyn)
        for pos, ang in (((900.0, 450.0, 1350.0), (0.0, 0.0, 0.0)), ((900.0, 900.0, 1799.0), (0.0, -0.3, 0.0)),
                         ((-500.0, 700.0, 900.0), (1.5707963, 0.0, 0.0)), ((1125.0, 675.0, 787.5), (0.7853982, 0.1, 0.0))):
            v = qb.view_setup(161, 97, pos, ang, 0.4, 10, LEVELS, S, 1, 0.0)
            ref = oracle.render(ref_scene, oracle.QboView.from_bytes(v.to_bytes()))
            plain = ctx.render_host([v], streams)[0].arrays
            counted = ctx.render_host([v], streams + ("visits",))[0].arrays
            compare_frame(counted, ref, f"{pos}", visits=True)
            compare_frame({**plain, "visits": counted["visits"]}, ref, f"{pos} without visits")
            # bytes alone are shaded by another route
            assert np.array_equal(ctx.render_host([v], ("rgba8",))[0]["rgba8"], ref["rgba8"]), pos


@pytest.mark.parametrize("shoot", [0, 1, 2, -1])
def test_bytes_alone(oracle, scene, shoot):
    """A frame of bytes alone where its shading must fall back: texels beyond
    [0, 1], zero, tiny, huge and non-finite normals, shoot outside 0 and 1."""
    import qubatron_gb300 as qb
    rng = np.random.default_rng(3)
    n = scene.colors.shape[0]
    col = scene.colors * rng.choice([0.0, 1.0, -1.0, 3.0, 1e4], (n, 3), p=[0.1, 0.6, 0.1, 0.1, 0.1]).astype(np.float32)
    with np.errstate(invalid="ignore"):
        nrm = scene.normals * rng.choice([1.0, 0.0, 1e-20, 1e20, 1e-30, np.inf, np.nan], (n, 1),
                                         p=[0.4, 0.1, 0.1, 0.1, 0.1, 0.1, 0.1]).astype(np.float32)
    v = qb.view_setup(201, 113, (903.7, 421.3, 1302.9), (0.2, -0.3, 0.0), 0.4, 10, LEVELS, S, shoot, 0.0)
    ref = oracle.render(oracle_scene(oracle, scene.nodes, col, nrm), oracle.QboView.from_bytes(v.to_bytes()))
    with qb.OctreeGLC(0) as ctx:
        upload_scene(ctx, scene.nodes, col, nrm)
        assert np.array_equal(ctx.render_host([v], ("rgba8",))[0]["rgba8"], ref["rgba8"])


@pytest.mark.parametrize("two_trees", [False, True])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 129, 1000, 3649, 20_000])
def test_few_rays(oracle, scene, character, n, two_trees):
    """So few rays that lanes without one take parts of the others' walks:
    results and visit counts are those of one lane's walk."""
    import qubatron_gb300 as qb
    from qubatron_gb300 import _lib as L
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.05 * S, 0.95 * S, (n, 3)).astype(np.float32)
    d = rng.normal(size=(n, 3)).astype(np.float32)
    d[::3] *= np.float32([1.0, 1e-3, 1.0])  # along the floor: long walks
    lp, ld = _rays("lattice", n, rng)
    pos[::5], d[::5] = lp[::5], ld[::5]
    dyn = character if two_trees else (None, None, None)
    with qb.OctreeGLC(0) as ctx:
        upload_scene(ctx, scene.nodes, scene.colors, scene.normals, *dyn)
        plain, counted = _trace(ctx, pos, d, False), _trace(ctx, pos, d, True)
        ctx.set_option(L.OPT_BOX_PRUNE, 0)
        shader = _trace(ctx, pos, d, True)
    ref = oracle.trace_rays(oracle_scene(oracle, scene.nodes, scene.colors, scene.normals, *dyn, boxes=True), BASE,
                            LEVELS, pos, d)
    for k in ("status", "leaf", "model", "isp", "col", "nrm"):
        assert np.array_equal(bits(plain[k]), bits(shader[k])), k
        assert np.array_equal(bits(counted[k]), bits(shader[k])), k
    for k in ("status", "leaf", "model", "visits"):
        assert np.array_equal(counted[k], ref[k]), k


@pytest.mark.parametrize("n", [1, 2, 5200, 5240, 5243, 5300])
def test_host_outputs(scene, n):
    """Any choice of outputs, around the size up to which they are copied
    together (512 KB with all of them)."""
    import qubatron_gb300 as qb
    from qubatron_gb300 import _lib
    pos, d = _rays("lattice", n, np.random.default_rng(n))
    with qb.OctreeGLC(0) as ctx:
        upload_scene(ctx, scene.nodes, scene.colors, scene.normals)
        want = _trace(ctx, pos, d, True)
        for names in (("status",), ("leaf", "isp"), ("visits", "model"), ("col", "nrm", "status"), ()):
            got = {k: np.full_like(want[k], 77) for k in names}
            h = _lib.RayHits(**{k: a.ctypes.data for k, a in got.items()})
            _lib.check(ctx._lib.qbc_trace_rays(ctx.handle, C.c_void_p(pos.ctypes.data), C.c_void_p(d.ctypes.data), n,
                                               (C.c_float * 4)(*BASE), LEVELS, C.byref(h), 0))
            for k in names:
                assert np.array_equal(bits(got[k]), bits(want[k])), (names, k)
