"""What Plan.run takes as a number of iterations.  Without a problem the engine
refuses the call itself (a null handle): an argument that gets that far was
accepted."""
import ctypes as C
import types

import numpy as np
import pytest


def run(iterations):
    from cuda_fot_b200 import fot
    nothing = types.SimpleNamespace(problem=types.SimpleNamespace(_h=C.c_void_p()), _h=C.c_void_p())
    with pytest.raises(fot.FotError):
        fot.Plan.run(nothing, iterations)


@pytest.mark.parametrize("iterations", [0, 1, 2 ** 32 - 1, True, np.int64(3), np.uint32(3), C.c_uint32(3)])
def test_accepted(iterations):
    run(iterations)


@pytest.mark.parametrize("iterations", [2 ** 64, 2 ** 64 + 3, -2 ** 63 - 1, 1.0, np.float64(2.0), "3", None])
def test_refused(iterations):
    with pytest.raises((C.ArgumentError, TypeError)):
        run(iterations)
