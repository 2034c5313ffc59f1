"""Places of a join's build rows: every slot of the largest tables, and every number in a group, comes back."""
import ctypes as C

import pytest

from test_cuda_errors_cpu import build


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = build(str(tmp_path_factory.mktemp("place")), """
extern "C" uint64_t place(uint64_t slot, unsigned number) { return place_of(slot, number); }
extern "C" uint64_t slot(uint64_t place) { return place_slot(place); }
extern "C" unsigned number(uint64_t place) { return place_number(place); }
""", "xlb_place.h")
    so.place.restype = so.slot.restype = C.c_uint64
    return so


@pytest.mark.parametrize("slots", [1 << 10, 1 << 31, 1 << 32, 1 << 33])  # (for up to 2^9, 2^30, 2^31 and 2^32 rows)
def test_places_come_back(lib, slots):
    for slot in (0, 1, slots // 2, slots - 1, slots):  # (the last one: key 0)
        for number in (0, 1, 31, 63):
            p = C.c_uint64(lib.place(C.c_uint64(slot), C.c_uint(number)))
            assert lib.slot(p) == slot and lib.number(p) == number
