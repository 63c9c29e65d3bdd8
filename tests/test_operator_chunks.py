"""The operator's z-chunk rule, on the host: no even split of the layers is
cheaper by the rule's own measure, slender columns of one tile included."""
import ctypes as C

import pytest


@pytest.fixture(scope="module")
def chunk(built_lib):
    fn = getattr(C.CDLL(str(built_lib)), "_ZN4hexa15op_chunk_layersExixd")
    fn.restype, fn.argtypes = C.c_int, [C.c_longlong, C.c_int, C.c_longlong, C.c_double]
    return fn


def cost(tiles, nz, ctas, start, kc):
    return -(-tiles * -(-nz // kc) // ctas) * (kc + start)


@pytest.mark.parametrize("tiles", [1, 2, 3, 7, 40, 108, 152, 153, 600])
@pytest.mark.parametrize("nz", [1, 2, 25, 97, 193, 1025, 2001, 10001])
@pytest.mark.parametrize("start", [0.6, 2.0])
def test_chunks_fill_the_gpu(chunk, tiles, nz, start):
    kc = chunk(tiles, nz, 152, start)
    assert 1 <= kc <= nz
    got = cost(tiles, nz, 152, start, kc)
    best = min(cost(tiles, nz, 152, start, k) for k in range(1, nz + 1))
    # chunks of many waves (over four items a CTA) are not tried: their starts cost what they save
    assert got <= 1.02 * best
    assert got <= cost(tiles, nz, 152, start, min(16, nz))  # the shortest chunk in use before
