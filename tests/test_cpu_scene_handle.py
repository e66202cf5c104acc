"""A scene lives as long as its handle: against a fake of the C library."""
import ctypes as C
import gc

import pytest

import agentray
import agentray.scenes as S


class _FakeLib:
    def __init__(self):
        self.made, self.destroyed = 0, []

    def ar_scene_create(self, ctx, desc, out):
        self.made += 1
        out._obj.value = 1000 + self.made
        return 0

    def ar_scene_destroy(self, handle):
        self.destroyed.append(handle.value)
        return 0


class _Context:
    handle = C.c_void_p(1)


@pytest.fixture
def fake(monkeypatch):
    fake = _FakeLib()
    monkeypatch.setattr(agentray, "lib", lambda: fake)
    yield fake
    for scene in [o for o in gc.get_objects() if isinstance(o, agentray.Scene)]:
        scene.handle = C.c_void_p()  # a failed test's frames keep it: not to reach the library


def test_a_handle_in_use_keeps_its_scene(fake):
    # As in check(lib().ar_render(ctx.handle, Scene(ctx, data).handle, ...)): the call
    # holds the handle, and nothing the scene.
    def call(handle):
        gc.collect()
        return handle.value, list(fake.destroyed)

    seen = call(agentray.Scene(_Context, S.cornell_box(1)[0]).handle)
    assert seen == (1001, [])
    gc.collect()
    assert fake.destroyed == [1001]


def test_a_scene_is_destroyed_once(fake):
    data = S.cornell_box(1)[0]
    a, b = agentray.Scene(_Context, data), agentray.Scene(_Context, data)
    kept = a.handle
    a.close()
    assert fake.destroyed == [1001] and not kept
    a.close()
    del a, kept, b
    gc.collect()
    assert sorted(fake.destroyed) == [1001, 1002]


def test_the_library_takes_the_handle(fake):
    # as c_void_p in an argument list and by reference, as the signatures say
    fn = C.CFUNCTYPE(C.c_int, C.c_void_p, C.POINTER(C.c_void_p))(lambda h, p: int(h == 7 and p[0] == 7))
    h = agentray._SceneHandle(7)
    assert fn(h, C.byref(h)) == 1
    h.value = None
