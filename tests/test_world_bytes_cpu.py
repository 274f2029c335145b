"""What a world's step borrows from a lane's pool: a pool of a given size
holds the worlds it held when the solve's levels were a float an array."""
import ctypes as C

import pytest

from worldinagrain_b200 import abi

# (width, height): the bytes a step borrowed then
THEN = {(8, 8): 26624, (16, 16): 91648, (32, 32): 361728, (75, 52): 1394944, (64, 64): 1459712, (256, 256): 23421952,
        (1024, 1024): 374817792, (8192, 2): 6041088}


@pytest.mark.parametrize("size", list(THEN))
def test_a_step_borrows_no_more(size):
    from worldinagrain_b200 import fluid
    f = fluid.lib().wig_batch_world_bytes_split
    f.argtypes = [C.POINTER(abi.WorldDesc), C.POINTER(C.c_uint64), C.POINTER(C.c_uint64)]
    f.restype = C.c_int
    d, kept, borrowed = abi.WorldDesc(*size, 0, 0), C.c_uint64(), C.c_uint64()
    assert f(C.byref(d), C.byref(kept), C.byref(borrowed)) == 0
    assert borrowed.value <= THEN[size]
