"""DEEP quotients on both sides of the row count from which a thread takes eight rows (2^16): one and several sample
points, accumulations lifted by every kind of ratio, unaligned columns. Words equal the oracle's."""
import pytest

import test_gpu_octets as octets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sub_log,blowup,acc_logs", [(15, 1, [15, 3]), (16, 1, [16]), (16, 2, [16, 15, 1]), (17, 1, [9, 17, 16, 2])])
@pytest.mark.parametrize("offset", [0, 1])
def test_quotients(sub_log, blowup, acc_logs, offset):
    octets.test_quotients(sub_log, blowup, acc_logs, offset)
