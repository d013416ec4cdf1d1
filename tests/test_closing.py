"""Objects and their context, closed in either order."""
import ctypes as C

import pytest

from rvpoint_b200 import datasets as D

pytestmark = pytest.mark.gpu


def live(L):
    d, p = C.c_longlong(0), C.c_longlong(0)
    L.rvp_debug_live_bytes(C.byref(d), C.byref(p))
    return d.value, p.value


@pytest.mark.parametrize("context_first", [False, True])
def test_memory_is_given_back(gpu_ctx, context_first):
    from rvpoint_b200 import api
    from rvpoint_b200.learned import PlaneScorer
    base = live(gpu_ctx.L)
    ctx = api.Context(0)
    c = D.room_cloud(n=3000, seed=1)
    h, o = api.SpatialHash(ctx), api.Octree(ctx)
    h.setInputCloud(c, 0.1)
    h.build()
    o.setInputCloud(c)
    o.build()
    things = [h, o, api.Pipeline(10_000, 2, ctx=ctx), PlaneScorer(3000, 1, ctx=ctx)]
    assert live(gpu_ctx.L)[0] > base[0]
    for t in [ctx] + things if context_first else things + [ctx]:
        t.close()
    assert live(gpu_ctx.L) == base
    for t in things:  # closed: a second time does nothing
        t.close()


def test_closed_with_their_context(gpu_ctx):
    from rvpoint_b200 import _lib, api
    ctx = api.Context(0)
    c = D.room_cloud(n=100, seed=1)
    h = api.SpatialHash(ctx)
    h.setInputCloud(c, 0.1)
    h.build()
    ctx.close()
    with pytest.raises(_lib.RvpError):
        h.knn(c.x, c.y, c.z, 3)
