"""A tuning that is read and set again changes nothing: fields the caller left
open stay open (frames in flight have defaults of their own, which a value set
for all frames would replace), fields that were changed hold, and a tuning made
from values alone holds as it is given."""
import ctypes as C

import pytest

import vrg

pytestmark = pytest.mark.gpu

FIELDS = [k for k, _ in vrg.Tuning._fields_ if k != "reserved"]
ALL = (1 << len(FIELDS)) - 1


def _open(t):
    return t.reserved[0]


@pytest.mark.parametrize("batched", [False, True], ids=["single", "batched"])
def test_set_of_get_is_neutral(gpu_ctx, batched):
    r = vrg.BatchRenderer(gpu_ctx, [(40, 30), (16, 9)], 3) if batched else vrg.Renderer(gpu_ctx, 80, 56, 3)

    def get():
        t = vrg.Tuning()
        vrg.check(gpu_ctx.lib.vrg_renderer_get_tuning(r.h, C.byref(t)), "vrg_renderer_get_tuning")
        return t
    try:
        base = get()
        assert _open(base) == ALL and all(v > 0 for v in base.as_dict().values())
        r.set_tuning(base)
        assert get().as_dict() == base.as_dict() and _open(get()) == ALL
        for k, name in enumerate(FIELDS[:-1]):  # one field changed: it holds, the others stay open
            t = get()
            v = {"stream_block": 64}.get(name, 1)
            setattr(t, name, v)
            r.set_tuning(t)
            assert getattr(get(), name) == v and _open(get()) == ALL & ~(1 << k), name
            r.set_tuning(get())  # and again
            assert getattr(get(), name) == v and _open(get()) == ALL & ~(1 << k), name
            setattr(t, name, 0)
            r.set_tuning(t)
            assert get().as_dict() == base.as_dict() and _open(get()) == ALL
        r.set_tuning(vrg.Tuning(*[getattr(base, k) for k in FIELDS]))  # the values alone: they hold
        assert get().as_dict() == base.as_dict() and _open(get()) == 0
        r.set_tuning(vrg.Tuning())
        assert _open(get()) == ALL
    finally:
        r.close()
