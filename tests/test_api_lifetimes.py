"""The Python wrapper's objects go before their context, however they go: closed by hand,
through the context, or collected with it in one garbage cycle (as after an exception whose
traceback holds them). The native library is replaced by a recorder."""
import ctypes
import gc

import pytest

from illume_gb300 import _capi as C
from illume_gb300 import api


@pytest.fixture
def gone(monkeypatch):
    order = []

    class Lib:
        def __getattr__(self, name):
            if name.endswith("_destroy"):
                return lambda h: order.append((name.split("_")[1], h.value))
            return lambda *args: C.OK

    lib = Lib()
    lib.illume_context_create = lambda device, budget, out: setattr(out._obj, "value", 1) or C.OK
    lib.illume_renderer_create = lambda ctx, scene, params, out: setattr(out._obj, "value", 3) or C.OK
    lib.illume_server_create = lambda ctx, budget, jobs, out: setattr(out._obj, "value", 4) or C.OK
    monkeypatch.setattr(C, "lib", lambda: lib)
    return order


def make():
    ctx = api.Context()
    scene = api.HostScene(ctx, ctypes.c_void_p(2))
    return ctx, scene, api.Renderer(ctx, scene, params=C.RenderParams()), api.Server(ctx)


def test_one_garbage_cycle(gone):
    gc.disable()
    try:
        ring = list(make())
        ring.append(ring)
        ring[0].ring = ring   # the context first in the cycle
        del ring
        gc.collect()
    finally:
        gc.enable()
    assert gone[-1] == ("context", 1)
    assert sorted(gone[:-1]) == [("renderer", 3), ("scene", 2), ("server", 4)]


def test_closed_through_the_context_and_by_hand(gone):
    ctx, scene, renderer, server = make()
    renderer.close()
    ctx.close()
    for x in (renderer, server, scene, ctx):
        x.close()
    assert gone == [("renderer", 3), ("server", 4), ("scene", 2), ("context", 1)]


def test_many_children(gone):
    ctx = api.Context()
    for i in range(500):
        api.HostScene(ctx, ctypes.c_void_p(100 + i)).close()
    kept = api.HostScene(ctx, ctypes.c_void_p(7))
    assert len(ctx._children) < 40
    ctx.close()
    assert gone[-2:] == [("scene", 7), ("context", 1)] and len(gone) == 502 and not kept.handle
