"""Barycentric weights on both sides of the domain size from which a thread takes eight rows (2^16): points of the
extension field, on the domain (with their conjugates and antipodes) and off the circle, unaligned columns. Words
equal the oracle's."""
import pytest

import test_gpu_octets as octets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_n", [15, 16, 17, 19])
@pytest.mark.parametrize("offset", [0, 1])
def test_weights(log_n, offset):
    octets.test_weights(log_n, offset)


@pytest.mark.parametrize("j", [0, 1, 5, 40000])
@pytest.mark.parametrize("turn", [0, 1, 2, 3])
def test_weights_at_domain_points(j, turn):
    octets.test_weights_at_domain_points(16, j, turn)


def test_weights_off_the_circle():
    octets.test_weights_off_the_circle(16)
