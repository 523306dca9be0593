"""The table's matmul on host arrays at decode rows: every way x and y cross the bus gives the device call's bytes."""
import ctypes as C

import numpy as np
import pytest

import turboexl3_b200 as t3
from turboexl3_b200 import synth
from turboexl3_b200 import table as tb

from gpu_util import bits16, dev

pytestmark = pytest.mark.gpu


# x read in place by the GEMV (up to 53 blocks of 256 inputs at one row) / rotated ahead (from 54 on, and past 8 rows); y written in
# place (128 KB) / by the copy engine; and the staged path
@pytest.mark.parametrize("in_dim,out_dim,rows", [(256, 1920, 1), (256, 2048, 1), (256, 6784, 1), (256, 6912, 1), (256, 2048, 32), (384, 24576, 3),
                                                 (2176, 2048, 32)])
def test_host_arrays_give_the_device_bytes(in_dim, out_dim, rows):
    trellis, suh, svh = synth.linear(2400 + rows, in_dim, out_dim, 32)
    block = tb.Block('{"format":"exl3","codebook":"mul1"}')
    verdict, weight = block.load_tensor(trellis, suh, svh, in_dim)
    assert verdict.ok, verdict.why
    x = synth.activations(2401 + rows, rows, in_dim)
    want = bits16(t3.linear(dev(x), dev(trellis), dev(suh), dev(svh)))
    for _ in range(2):
        verdict, y = tb.matmul(weight, x)
        assert verdict.ok, verdict.why
        assert np.array_equal(y.view(np.uint16), want)
    assert t3.device_error() == 0
    tb.table().release(C.byref(weight))
    block.close()
