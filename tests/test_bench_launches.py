"""The launches that bench.py states for a batch call follow the batch entry's
own limits (cudec_b200/csrc/batch.cu)."""
import os
import re

import pytest

import bench

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cudec_b200",
                   "csrc", "batch.cu")


@pytest.mark.parametrize("sms", [148, 132])
def test_lz_launches(sms):
    text = open(SRC).read()
    medium = int(re.search(r"kMediumMax = (\d+)", text).group(1))
    beside = eval(re.search(r"kWideBeside = ([^;]+);", text).group(1))
    for n, want in ((1, 1), (medium * sms, 1), (medium * sms + 1, 2), (beside, 2), (beside + 1, 1)):
        assert bench.lz_launches(n, sms) == want, n
