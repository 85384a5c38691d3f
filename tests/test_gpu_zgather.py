"""The fused z FFT + gather of FP64 plans where a launch takes four slots per block: from H = 24
on with more than two blocks of one slot per SM, below from 2048 of them, with a remainder of
slots and of fields.  Fields, truths and tolerances as in test_gpu_rows.py (a transform of n
points is within about 4 log2(n) eps of the largest value: 1.5e-14 at 48^3 points, bar 2e-13)."""
import pytest

from test_gpu_rows import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sg,n,batch", [(229, 16, 347), (230, 24, 263), (229, 32, 211), (229, 48, 151), (225, 64, 231),
                                        (229, 96, 13), (221, 48, 49), (47, 64, 37)])
def test_four_slots_fp64(cf, O, prep, sg, n, batch):
    check(cf, O, prep, sg, (n, n, n), 8, batch)
