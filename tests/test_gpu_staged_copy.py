"""Results of 20 MB and more to pageable memory, which go in chunks through pinned
buffers: sizes at the threshold and at the chunks' ends, destinations at every kind
of offset to the 2 MB parts, out of a context and out of a batch. Compared with the
same result copied to pinned memory, which takes no chunks."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

HUGE = 1 << 21          # the threads' parts end at multiples of it
STAGED = 20 << 20       # threshold, bytes
HEAD, CHUNK = 14 << 20, 16 << 20  # first chunk of a destination at a multiple of HUGE, and the others


def i32(p):
    return p.ctypes.data_as(C.POINTER(C.c_int32))


def u32(p):
    return p.ctypes.data_as(C.POINTER(C.c_uint32))


def cliques(triangles, seed):
    """Disjoint K3, K4 and K5 in random order (1, 4, 10 triangles; k of 0, 1, 2)."""
    r = np.random.default_rng(seed)
    size = r.integers(3, 6, triangles)
    count = np.array([0, 0, 0, 1, 4, 10])
    blocks = int(np.searchsorted(np.cumsum(count[size]), triangles - 10))
    size = size[:blocks]
    size = np.concatenate([size, np.full(triangles - int(count[size].sum()), 3)])
    first = np.concatenate([[0], np.cumsum(size)[:-1]])
    s, t = [], []
    for n in (3, 4, 5):
        i, j = np.triu_indices(n, 1)
        at = first[size == n][:, None]
        s.append((at + i).ravel())
        t.append((at + j).ravel())
    return np.concatenate(s).astype(np.uint32), np.concatenate(t).astype(np.uint32)


def check(copy, words, offset):
    """copy(pointer) against the copy to pinned memory; nothing else is written."""
    pinned = torch.empty(words, dtype=torch.int32).pin_memory().numpy().view(np.uint32)
    copy(pinned)
    assert np.unique(pinned).size > 1
    room = np.full(words + 3 * HUGE // 4, 0xA5A5A5A5, np.uint32)
    at = ((-room.ctypes.data) % HUGE + offset) // 4
    copy(room[at:at + words])
    assert np.array_equal(room[at:at + words], pinned)
    assert np.all(room[:at] == 0xA5A5A5A5) and np.all(room[at + words:] == 0xA5A5A5A5)


@pytest.mark.parametrize("byte_count", [STAGED, HEAD + CHUNK, HEAD + 2 * CHUNK])
@pytest.mark.parametrize("more", [-4, 0, 4])
def test_k_at_the_chunk_ends(n34, byte_count, more):
    words = (byte_count + more) // 4
    with n34.Context() as ctx:
        ctx.upload_edges(*cliques(words, 1))
        assert ctx.run("ondemand")["triangle_count"] == words
        for offset in (0, 4, HUGE - 4):
            check(lambda p: n34._check(n34.lib().nucleus34_ctx_copy_k(ctx._h, i32(p), None), "copy_k"), words, offset)
        assert n34.lib().nucleus34_release_cached_memory(0) == 0
        check(lambda p: n34._check(n34.lib().nucleus34_ctx_copy_k(ctx._h, i32(p), None), "copy_k"), words, 0)


@pytest.mark.parametrize("lead", [4, HUGE // 2, HUGE - 4])
@pytest.mark.parametrize("more", [-4, 0, 4])
def test_chunk_ends_of_other_destinations(n34, lead, more):
    """A destination `lead` bytes below a multiple of 2 MB has a first chunk longer
    by as much."""
    words = (HEAD + lead + CHUNK + more) // 4
    with n34.Context() as ctx:
        ctx.upload_edges(*cliques(words, 2))
        assert ctx.run("ondemand")["triangle_count"] == words
        check(lambda p: n34._check(n34.lib().nucleus34_ctx_copy_k(ctx._h, i32(p), None), "copy_k"), words, HUGE - lead)


@pytest.mark.parametrize("triangles", [STAGED // 12, STAGED // 12 + 1, (HEAD + CHUNK) // 12, (HEAD + CHUNK) // 12 + 1])
def test_triangle_list(n34, triangles):
    with n34.Context() as ctx:
        ctx.upload_edges(*cliques(triangles, 3))
        assert ctx.run("ondemand")["triangle_count"] == triangles
        for offset in (0, 12):
            check(lambda p: n34._check(n34.lib().nucleus34_ctx_copy_k(ctx._h, None, u32(p)), "copy_k"),
                  3 * triangles, offset)


def test_batch(n34):
    """The middle one of three graphs, 21 MB of k."""
    graphs = [n34.graph_from_edges(*n34.gen_ws(1000 + i, 10, 0.1, i)) for i in (1, 2)]
    big = n34.graph_from_edges(*cliques(STAGED // 4 + 300001, 4))
    alone = n34.decompose(big, variant="ondemand", n_quds=0)
    with n34.batch_decompose([graphs[0], big, graphs[1]]) as b:
        k, tris = b.copy_k(1, with_tris=True)
        check(lambda p: n34._check(n34.lib().nucleus34_batch_copy_k(b._h, 1, i32(p), None), "batch_copy_k"), len(k), 4)
    assert k.nbytes > STAGED and np.array_equal(k, alone.k) and np.array_equal(tris, alone.tris)
