"""What classes derived from the library's parts inherit."""
import pytest

from camelid_b200.parts import attention, feedforward, latent_attention, recurrent, window_attention


@pytest.mark.parametrize("base,method", [(feedforward.DenseFeedForward, "_activations"), (window_attention.WindowAttention, "attend"),
                                         (latent_attention.LatentAttention, "attend"), (recurrent.Retention, "read_out")])
def test_a_class_that_takes_the_rows_itself_gets_complete_ones(base, method):
    """A method that knows of no scale, in the class itself, further down or beside it; one that takes the scale says so again."""
    own = {method: lambda self, ctx, x, *more, **named: x}
    derived, beside = type("Derived", (base,), own), type("Beside", (type("Mixin", (), own), base), {})
    assert base.accepts_row_scale and not derived.accepts_row_scale and not beside.accepts_row_scale
    assert not type("Further", (derived,), {}).accepts_row_scale
    assert type("Plain", (base,), {"load": lambda self, *a: None}).accepts_row_scale
    assert type("Again", (base,), {**own, "accepts_row_scale": True}).accepts_row_scale


def test_classes_of_the_library_keep_what_they_say():
    assert feedforward.DenseGelu.accepts_row_scale and feedforward.SwiGLU.accepts_row_scale
    assert type("Derived", (attention.GroupedQueryAttention,), {"forward": lambda self, ctx, x, residual: None}).accepts_row_scale


def test_a_derived_part_with_matrices_of_its_own_is_taken_at_its_word():
    part = type("Derived", (feedforward.SwiGLU,), {})({"hidden_size": 16, "intermediate_size": 32})
    assert part.w_gate_up is None and part.scales_sums(None, 4)


def test_sums_that_wait_already_are_not_replaced(monkeypatch):
    """A part from outside may leave sums pending while a product is deferred: the product is added plainly then."""
    from types import SimpleNamespace

    import torch

    from camelid_b200.parts import linear
    h, w = torch.zeros((2, 5000)), torch.zeros((5000, 8))
    ctx = SimpleNamespace(deferred=(torch.zeros((2, 8)), w, h), pending="theirs")
    ran = []
    monkeypatch.setattr(linear, "_few", lambda *a, **k: True)
    monkeypatch.setattr(linear, "partial_sums", lambda *a: "ours")
    monkeypatch.setattr(linear, "linear", lambda ctx, x, w, out, epilogue: ran.append(out is h))
    linear.deferred_sums(ctx, h)
    assert ctx.pending == "theirs" and ctx.deferred is None and ran == [True]
    ctx = SimpleNamespace(deferred=(torch.zeros((2, 8)), w, h), pending=None)
    linear.deferred_sums(ctx, h)
    assert ctx.pending == "ours" and ctx.deferred is None and ran == [True]
