"""The order in which Python's finalisers destroy the library's handles: a
context that is collected in one cycle with its objects (as at interpreter exit)
takes them along, and none is destroyed after it."""
import gc

import pytest

from _loader import load

mzk = load()


class FakeLib:
    """Hands out handles and records what is destroyed."""

    def __init__(self):
        self.next, self.destroyed = 100, []

    def __getattr__(self, name):
        def call(*args):
            if name.endswith("_destroy") or name == "mzk_device_free":
                self.destroyed.append((name, args[-1]))
            for a in args:
                if hasattr(a, "_obj"):  # an output by reference
                    self.next += 1
                    a._obj.value = self.next if name != "mzk_domain_shape" else 4
            return 0
        return call


@pytest.fixture
def fake(monkeypatch):
    f = FakeLib()
    monkeypatch.setattr(mzk, "lib", lambda: f)
    return f


def objects():
    ctx = mzk.Context(0)
    return ctx, mzk.EvaluationDomain(ctx, 5, 4), ctx.alloc(64), mzk.ProvingServer(ctx)


def expected(ctx, dom, buf, srv):
    return [("mzk_server_destroy", srv.h), ("mzk_domain_destroy", dom.h), ("mzk_device_free", buf.ptr),
            ("mzk_ctx_destroy", ctx.h)]


def test_collected_in_a_cycle(fake):
    cycle = {}
    cycle["self"], cycle["all"] = cycle, objects()
    want = expected(*cycle["all"])
    del cycle
    gc.collect()
    assert fake.destroyed == want


def test_closed_by_the_caller(fake):
    all_ = objects()
    want = expected(*all_)
    all_[0].close()
    del all_
    gc.collect()
    assert fake.destroyed == want


def test_objects_first(fake):
    ctx, dom, buf, srv = objects()
    want = expected(ctx, dom, buf, srv)
    srv.close()
    dom.close()
    buf.free()
    del dom, buf, srv
    ctx.close()
    assert fake.destroyed == want
