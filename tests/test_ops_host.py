"""Host side of the ops: what the launchers are told, without a GPU."""
from types import SimpleNamespace

from pie_b200 import ops


def test_products_over_expanded_weights_say_so(monkeypatch):
    """The GEMM requests weights ahead of its predecessor's end unless it is told that the predecessor wrote them, as the
    expansion of an fp8 weight does."""
    calls = []
    monkeypatch.setattr(ops, "dequant_fp8", lambda q, out=None: calls.append("expand"))
    monkeypatch.setattr(ops, "gemm", lambda x, w, **kw: calls.append(kw.get("fresh_w", False)))
    monkeypatch.setattr(ops, "_FP8_SCRATCH", {(0, (64, 24)): "scratch"})
    on_device = SimpleNamespace(is_cuda=True, shape=(3, 24))
    ops.gemm_fp8w(on_device, SimpleNamespace(shape=(64, 24), device=SimpleNamespace(index=0)), mode="dequant")
    assert calls == ["expand", True]
