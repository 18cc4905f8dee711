"""Closing a context closes what renders its volumes before the volumes."""


def test_context_closes_servers_and_batches_first(monkeypatch):
    import weakref
    import livre_gb300 as lv
    order = []

    class Lib:
        def lv_ctx_destroy(self, handle):
            order.append("Context")

    monkeypatch.setattr(lv, "lib", lambda: Lib())
    ctx = lv.Context.__new__(lv.Context)
    ctx.handle = object()
    ctx._children = weakref.WeakSet()
    children = []
    for cls in (lv.Volume, lv.TransferFunction, lv.Batch, lv.Server):
        monkeypatch.setattr(cls, "close", lambda self: order.append(type(self).__name__))
        children += [cls.__new__(cls) for _ in range(5)]
    for child in children:
        ctx._children.add(child)
    ctx.close()
    assert order[:5] == ["Server"] * 5 and order[5:10] == ["Batch"] * 5
    assert sorted(order[10:20]) == ["TransferFunction"] * 5 + ["Volume"] * 5
    assert order[20:] == ["Context"]
