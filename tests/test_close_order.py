"""A plan or batch closed after its context (the garbage collector's order in a cycle)
leaves the library alone: its context's memory is gone. No GPU: handles are made up
and the destroy calls are counted."""
import ctypes

import pytest


class _Lib:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        return lambda *a: self.calls.append(name)


@pytest.mark.parametrize("cls,call", [("Plan", "awc_plan_destroy"), ("Batch", "awc_batch_destroy")])
def test_close_after_the_context(pkg, monkeypatch, cls, call):
    fake = _Lib()
    monkeypatch.setattr(pkg._lib, "lib", lambda: fake)

    def make():
        ctx = object.__new__(pkg.Context)
        ctx._h = ctypes.c_void_p(1)
        x = object.__new__(getattr(pkg, cls))
        x.ctx, x._h = ctx, ctypes.c_void_p(2)
        return ctx, x

    ctx, x = make()
    x.close()
    x.close()
    assert fake.calls == [call]
    ctx.close()
    fake.calls.clear()
    ctx, x = make()
    ctx.close()
    x.close()
    assert fake.calls == ["awc_destroy"]
