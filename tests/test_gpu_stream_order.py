"""Ray queries on host arrays read them in stream order: arrays that work queued
earlier on the context's stream has still to fill (pinned ones by a copy,
pageable ones by a host function) give the rays they then hold, whatever the
number of rays (small calls copy through a buffer of the context's, larger
ones array by array)."""
import ctypes as C

import numpy as np
import pytest

from conftest import LEVELS, S
from helpers import bits, upload_scene

pytestmark = pytest.mark.gpu

OUT = {"status": ((), np.int32), "leaf": ((2,), np.int32), "model": ((2,), np.int32), "isp": ((4,), np.float32),
       "col": ((4,), np.float32), "nrm": ((4,), np.float32), "visits": ((2,), np.uint32)}


def _cudart():
    """The CUDA runtime this process has loaded (PyTorch's)."""
    with open("/proc/self/maps") as f:
        paths = {line.split()[-1] for line in f if "libcudart.so" in line}
    if not paths:
        pytest.skip("no shared CUDA runtime loaded")
    return C.CDLL(paths.pop())


@pytest.mark.parametrize("pinned", [("pos", "dir"), ("pos",), ("dir",), ()])
@pytest.mark.parametrize("n", [1, 1000, 5200, 8000])
def test_rays_filled_on_the_stream(floor50k_scene, n, pinned):
    torch = pytest.importorskip("torch")
    import qubatron_gb300 as qb
    from qubatron_gb300 import _lib
    s = floor50k_scene
    rng = np.random.default_rng(n)
    new = {"pos": rng.uniform(0.05 * S, 0.95 * S, (n, 3)).astype(np.float32),
           "dir": rng.normal(size=(n, 3)).astype(np.float32)}
    old = {"pos": np.full((n, 3), 0.5 * S, np.float32), "dir": np.ones((n, 3), np.float32)}
    with qb.OctreeGLC(0) as ctx:
        upload_scene(ctx, s.nodes, s.colors, s.normals)
        want = ctx.trace_rays(new["pos"], new["dir"], (0.0, S, S, S), LEVELS)
        stream = torch.cuda.Stream()
        ctx.set_stream(stream.cuda_stream)
        host = {k: torch.from_numpy(old[k].copy()).pin_memory() for k in pinned}
        src = {k: torch.from_numpy(new[k]).cuda() for k in pinned}
        torch.cuda.synchronize()
        got = {k: np.zeros((n, *shape), dt) for k, (shape, dt) in OUT.items()}
        h = _lib.RayHits(**{k: a.ctypes.data for k, a in got.items()})
        if not pinned:
            host = {k: torch.from_numpy(old[k]) for k in new}
        at = {k: host[k].data_ptr() if k in host else new[k].ctypes.data for k in new}
        fill = C.CFUNCTYPE(None, C.c_void_p)(lambda _: [np.copyto(old[k], new[k]) for k in new] and None)
        with torch.cuda.stream(stream):
            torch.cuda._sleep(20_000_000)  # some 10 ms before the arrays are filled
            for k in pinned:
                host[k].copy_(src[k], non_blocking=True)
            if not pinned:
                assert _cudart().cudaLaunchHostFunc(C.c_void_p(stream.cuda_stream), fill, None) == 0
        _lib.check(ctx._lib.qbc_trace_rays(ctx.handle, C.c_void_p(at["pos"]), C.c_void_p(at["dir"]), n,
                                           (C.c_float * 4)(0.0, S, S, S), LEVELS, C.byref(h), 0))
        torch.cuda.synchronize()
        ctx.set_stream(None)
    for k in OUT:
        assert np.array_equal(bits(got[k]), bits(want[k])), k
