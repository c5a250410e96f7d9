"""Results copied to host memory in chunks: sizes and destinations where the
chunks and the threads' parts of them begin and end. Bytes must be equal and
nothing beyond them written."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HUGE = 1 << 21


@pytest.fixture(scope="module")
def big(n34):
    # 5.9M triangles: k is 24 MB (two chunks), the triangles 71 MB (five)
    ctx = n34.Context()
    ctx.upload(n34.graph_from_edges(*n34.gen_rgg(60000, 32, 3)))
    r = ctx.run("ondemand")
    yield ctx, int(r["triangle_count"])
    ctx.close()


@pytest.mark.parametrize("offset", [0, 4, HUGE - 4, HUGE, HUGE + 4, 12340])
def test_destinations(n34, big, offset):
    ctx, T = big
    k0, t0 = ctx.copy_k(T, with_tris=True)
    room = np.full((16 * T + 4 * HUGE) // 4, 0xA5A5A5A5, np.uint32)
    base = (-room.ctypes.data) % HUGE + offset
    k = room[base // 4:base // 4 + T]
    tb = base + 4 * T + 64
    tris = room[tb // 4:tb // 4 + 3 * T]
    assert n34.lib().nucleus34_ctx_copy_k(ctx._h, k.ctypes.data_as(C.POINTER(C.c_int32)),
                                          tris.ctypes.data_as(C.POINTER(C.c_uint32))) == 0
    assert np.array_equal(k.view(np.int32), k0) and np.array_equal(tris.reshape(-1, 3), t0)
    k[:] = tris[:] = 0xA5A5A5A5
    assert np.all(room == 0xA5A5A5A5)


# k of 8 MB and one chunk, each with one word less and one more, out of a batch
# whose graphs lie behind one another; then once more without cached buffers
@pytest.mark.parametrize("words", [2 ** 21 - 1, 2 ** 21, 2 ** 21 + 1, 2 ** 22 - 1, 2 ** 22, 2 ** 22 + 1])
def test_sizes(n34, words):
    # disjoint triangles: one k each, every one 0 but a K4's four
    tri = np.arange(3 * (words - 4), dtype=np.uint32).reshape(-1, 3)
    q = np.uint32(3 * (words - 4))
    s = np.concatenate([tri[:, 0], tri[:, 0], tri[:, 1], np.array([q, q, q, q + 1, q + 1, q + 2], np.uint32)])
    d = np.concatenate([tri[:, 1], tri[:, 2], tri[:, 2], np.array([q + 1, q + 2, q + 3, q + 2, q + 3, q + 3], np.uint32)])
    with n34.Context() as ctx:
        ctx.upload(n34.graph_from_edges(s, d))
        assert ctx.run("ondemand")["triangle_count"] == words
        for _ in range(2):
            k = ctx.copy_k(words)
            assert np.count_nonzero(k) == 4 and np.all(k[-4:] == 1)
            assert n34.lib().nucleus34_release_cached_memory(0) == 0
