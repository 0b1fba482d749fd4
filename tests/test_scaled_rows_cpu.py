"""Undivided rows go only to parts that read them: a part derived from one that does, with a ``forward`` or ``add_norm`` of its
own, gets normalised rows."""
from types import SimpleNamespace

from kindi_b200.parts.attention import CausalSelfAttention
from kindi_b200.parts.base import LazyBranch
from kindi_b200.parts.mlp import SwiGLU
from kindi_b200.parts.norm import RMSNorm


def test_derived_parts_do_not_take_undivided_rows(monkeypatch):
    from kindi_b200.kernels import linear as L
    monkeypatch.setattr(L, "takes_scaled", lambda *a, **k: True)
    monkeypatch.setattr(L, "stream_product", lambda *a, **k: ("rows", "squares"))
    ctx = SimpleNamespace()
    for base, attrs in ((CausalSelfAttention, dict(wqkv=None)), (SwiGLU, dict(wgu=None, group=L.GATE_UP_GROUP))):
        own = type("Own", (base,), {"forward": lambda self, ctx, y: y})
        kept = type("Kept", (base,), {})
        for cls, takes in ((base, True), (kept, True), (own, False)):
            part = cls.__new__(cls)
            part.__dict__.update(attrs)
            assert part.takes_scaled_rows(ctx) is takes, cls
    for cls, takes in ((RMSNorm, True), (type("Own", (RMSNorm,), {"add_norm": lambda self, *a, **k: None}), False)):
        norm = cls.__new__(cls)
        norm.__dict__.update(weight=None, eps=1e-5)
        assert (norm.add_norm_scaled(ctx, None, LazyBranch(ctx, None, None)) is not None) is takes, cls
