"""How the similarity matrix without a kept workspace is cut into launches (csrc/cuda/cos_sim.cu): one, and one copy of the result,
up to 2048 x 4096 pairs; one whatever the size where the result takes the place of an input."""
import ctypes as C

import pytest

import fastface_b200 as ff


@pytest.mark.parametrize("n,m,over,launches", [(1, 1, 0, 1), (2048, 1400, 0, 1), (700, 4000, 0, 1), (2048, 4096, 0, 1), (2049, 4096, 0, 2),
                                               (2048, 4097, 0, 2), (5000, 10000, 0, 9), (5000, 10000, 1, 1)])
def test_launches(built_lib, n, m, over, launches):
    lib = ff.load_library()
    lib.ffcu_test_cos_plain_launches.restype = C.c_longlong
    lib.ffcu_test_cos_plain_launches.argtypes = [C.c_int] * 3
    assert lib.ffcu_test_cos_plain_launches(n, m, over) == launches
