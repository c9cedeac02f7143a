"""The mesh kernel's queue of large triangles (LargeQueue, mesh.cu) on the
host: what reaches the slot's list, and how far the list's length counts once
it is full.  The length is a 32-bit number and one triangle can enter
thousands of bands of rows, so a mesh of noise could carry it past 2^31 if
every entry went on being counted; a warp that meets a full list counts no
more, which leaves at most one group of 32 per warp beyond the capacity."""
import ctypes

import numpy as np
import pytest

import device_host

CODE = """
#include "device_types.hpp"
using namespace rvsb;
constexpr int QUEUE = 64, kEntryPixels = 8192, kBiasBits = 0x4B400000;
%s
extern "C" int push_warps(int warps, int rounds, int capacity, int width, int height, int* length, uint4* list) {
    // `warps` warps, one after the other, in which every lane enters `rounds`
    // triangles with a box of width x height pixels.
    DevStatus st{};
    SlotBuffers B{};
    B.status = &st;
    B.large = list;
    B.large_capacity = capacity;
    for (int w = 0; w < warps; ++w) {
        uint4 q[QUEUE] = {};
        run_warp([&](int lane) {
            LargeQueue queue{q, 0};
            for (int r = 0; r < rounds; ++r)
                queue.push(B, lane, true, (uint32_t)((w * rounds + r) * 32 + lane), 1, false,
                           make_int4(kBiasBits, kBiasBits, kBiasBits + width - 1, kBiasBits + height - 1));
            if (queue.n > 0) queue.flush(B, lane, queue.n);
        });
    }
    *length = st.n_large;
    return 0;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return device_host.build(str(tmp_path_factory.mktemp("queue")), CODE % device_host.extract("mesh.cu", "struct LargeQueue {"))


def _push(lib, warps, rounds, capacity, width, height):
    length = ctypes.c_int()
    guard = 64
    entries = np.full((capacity + guard, 4), 0xffffffff, np.uint32)
    lib.push_warps(warps, rounds, capacity, width, height, ctypes.byref(length),
                   entries.ctypes.data_as(ctypes.c_void_p))
    assert (entries[capacity:] == 0xffffffff).all()
    return length.value, entries[:capacity]


@pytest.mark.parametrize("width,height", [(8, 4), (8192, 5), (100, 200)])
def test_every_band_reaches_the_list(lib, width, height):
    """Boxes of at most 8192 pixels, exactly a row, and two and a half bands
    of 81 rows: all entries arrive, and a triangle's bands tile its rows."""
    n, entries = _push(lib, 2, 2, 4096, width, height)
    per = -(-height // max(1, 8192 // width))
    assert n == 2 * 2 * 32 * per
    rows = {}
    for tri, view, x, y in entries[:n].tolist():
        assert view == 1 and x == (width - 1) << 16
        rows.setdefault(tri, []).append((y & 0xffff, y >> 16))
    assert sorted(rows) == list(range(2 * 2 * 32))
    for bands in rows.values():
        bands.sort()
        assert bands[0][0] == 0 and bands[-1][1] == height - 1
        assert all(a[1] + 1 == b[0] for a, b in zip(bands, bands[1:]))


def test_a_full_list_stops_counting(lib):
    """Three warps of 64 triangles of 64 bands each, 12,288 entries, into a
    list of 100: overflow is seen, and counted at most once per warp."""
    warps, capacity = 3, 100
    n, _ = _push(lib, warps, 2, capacity, 8192, 64)
    assert capacity < n <= capacity + 32 * (warps + 1)


def test_a_list_filled_to_the_last_entry_is_no_overflow(lib):
    n, entries = _push(lib, 2, 2, 128, 8, 4)
    assert n == 128
    assert sorted(entries[:, 0].tolist()) == list(range(128))
