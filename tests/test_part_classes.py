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
