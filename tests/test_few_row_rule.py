"""Which products of few rows run on the kernel whose blocks own whole sums, at shapes that were measured on both."""
import pytest

from camelid_b200.csrc import ops


@pytest.mark.parametrize("n,k,plain,with_act", [(4736, 64, True, True), (6144, 64, False, True), (28672, 64, False, False), (6144, 256, True, True),
                                                (11008, 256, False, True), (28672, 256, False, False), (16384, 384, True, True), (65536, 384, False, False),
                                                (28672, 512, True, True), (50304, 512, False, False), (50304, 768, True, False), (50304, 640, False, False), (128256, 640, False, False),
                                                (128256, 1024, True, True), (128256, 2048, True, True), (16384, 2048, True, True), (2048, 8192, True, True)])
def test_the_faster_kernel(n, k, plain, with_act):
    assert (ops.few_pays(n, k, True), ops.few_pays(n, k, False)) == (plain, with_act)
