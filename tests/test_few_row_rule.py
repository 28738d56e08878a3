"""Which products of few rows run on the kernel whose blocks own whole sums, at shapes that were measured on both."""
import pytest

from camelid_b200.csrc import ops


@pytest.mark.parametrize("n,k,plain,with_act", [(4736, 64, True, True), (6144, 64, False, True), (28672, 64, False, False), (6144, 256, True, True),
                                                (11008, 256, False, True), (28672, 256, False, False), (16384, 384, True, True), (65536, 384, False, False),
                                                (28672, 512, True, True), (50304, 512, False, False), (50304, 768, True, False), (50304, 640, False, False), (128256, 640, False, False),
                                                (128256, 1024, True, True), (128256, 2048, True, True), (16384, 2048, True, True), (2048, 8192, True, True), (28672, 5120, False, False),
                                                (20480, 5120, True, True), (28672, 4608, True, True)])
def test_the_faster_kernel(n, k, plain, with_act):
    assert (ops.few_pays(n, k, True), ops.few_pays(n, k, False)) == (plain, with_act)


@pytest.mark.parametrize("rows,top,experts,hidden,ff,few", [(1, 8, 8, 2048, 2048, True), (4, 2, 8, 2048, 2048, True), (8, 2, 8, 2048, 2048, False),
                                                            (8, 2, 32, 2048, 2048, True), (8, 2, 16, 1536, 2048, True), (8, 2, 4, 2048, 1024, False),
                                                            (8, 2, 8, 2048, 1024, True), (16, 1, 4, 1024, 1024, True), (8, 2, 2, 256, 128, True),
                                                            (9, 2, 64, 256, 128, False)])
def test_the_faster_form_of_routed_products(rows, top, experts, hidden, ff, few):
    assert ops.few_pairs_pay(rows, top, experts, hidden, ff) == few


def test_weights_that_always_pay():
    assert all(ops.few_pays(ops.FEW_ALWAYS // k, k, plain) for k in range(1024, 20000, 8) for plain in (True, False))
