"""The filter's tile plan, on the host: the threads that stage a tile reach every
node of it and of its halo, and fit the CTA; tiles and chunks cover the grid."""
import ctypes as C

import pytest


class Grid(C.Structure):
    _fields_ = [(n, C.c_int) for n in ("nx", "ny", "nz", "NX", "NY", "NZ")]


class Plan(C.Structure):
    _fields_ = [(n, C.c_int) for n in ("tx", "ty", "threads", "stage", "ntx", "nty", "kchunk")]
    _fields_ += [("items", C.c_longlong), ("blocks", C.c_int)]


@pytest.fixture(scope="module")
def plan(built_lib):
    fn = getattr(C.CDLL(str(built_lib)), "_ZN4hexa9helm_planERKNS_4GridE")
    fn.restype, fn.argtypes = Plan, [C.POINTER(Grid)]
    return lambda nx, ny, nz: fn(C.byref(Grid(nx, ny, nz, nx + 1, ny + 1, nz + 1)))


# each range of cross-sections holds some whose tile has an odd number of nodes just past a multiple of 64
@pytest.mark.parametrize("xs,ys", [(range(1, 140), range(1, 40)), (range(1, 12), range(1, 300)),
                                   (range(120, 520, 7), range(1, 260, 3))])
def test_staging_covers_the_tile(plan, xs, ys):
    for nx in xs:
        for ny in ys:
            p = plan(nx, ny, 9)
            nodes = (p.tx + 2) * (p.ty + 2)
            assert 2 * p.stage >= nodes and p.stage <= p.threads, (nx, ny, p.tx, p.ty)
            assert p.stage % 32 == 0 and p.threads % 32 == 0 and p.threads <= 288
            assert p.ntx * p.tx > nx and p.nty * p.ty > ny and p.tx * p.ty <= p.threads
            assert -(-10 // p.kchunk) * p.ntx * p.nty == p.items


def test_the_tile_of_an_odd_node_count_is_picked(plan):
    for dims in [(52, 4), (104, 4), (105, 4)]:
        for nx, ny in (dims, dims[::-1]):
            p = plan(nx, ny, 3)
            assert {p.tx, p.ty} == {53, 5} and p.stage >= 193
