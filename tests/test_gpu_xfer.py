"""Copies between pageable host memory and the device through the context's
pinned chunks (csrc/spk_xfer.cu): the reads a count uploads and the lists it
downloads are the same bytes whether the host buffers are pageable numpy
arrays (copied in 4 MiB pieces by several host threads) or pinned memory
(copied directly).  Integer data, compared bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def spk(spk_lib):
    return spk_lib


def pinned_copy(a):
    import torch
    t = torch.from_numpy(np.ascontiguousarray(a)).pin_memory()
    return t, t.numpy()


def test_pageable_and_pinned_uploads_agree(spk):
    """A read set of 38 MB (several upload pieces, each over the direct-copy
    size) counted from pageable and from pinned host buffers: same lists,
    edges and statistics; the downloads into pageable arrays equal those into
    pinned ones, and a piece-sized tail (not a multiple of the chunk) is
    whole."""
    from spk import synth
    p = synth.c2(0.3).packed
    assert p.data.size > 32 << 20
    hold = [pinned_copy(x) for x in (p.data, p.offsets, p.lengths)]
    pinned = tuple(h[1] for h in hold)
    a = spk.count(p, [31, 55], bloom_bits=1 << 28)
    b = spk.count(pinned, [31, 55], bloom_bits=1 << 28)
    for ki in range(2):
        ia, ib = a.info(ki), b.info(ki)
        for key in ("occurrences", "n_table", "n_list", "n_solid", "n_edges", "cutoff", "twice_popcount"):
            assert ia[key] == ib[key], key
        ka, ca = a.kmers(ki)
        kb, cb = b.kmers(ki)
        assert ka.nbytes > 8 << 20  # the download goes through the pinned chunks
        np.testing.assert_array_equal(ka, kb)
        np.testing.assert_array_equal(ca, cb)
        np.testing.assert_array_equal(a.edges(ki), b.edges(ki))
        # the same list into pinned output arrays
        m = ka.shape[0]
        tk, hk = pinned_copy(np.zeros((m + 3, ka.shape[1]), np.uint64))
        tc, hc = pinned_copy(np.zeros(m + 3, np.uint32))
        gk, gc = b.kmers(ki, out=(hk, hc))
        np.testing.assert_array_equal(gk, ka)
        np.testing.assert_array_equal(gc, ca)
    a.close()
    b.close()


def test_per_thread_stream_keeps_its_order(spk):
    """A context on cudaStreamPerThread (handle 2): copies of pageable memory
    above the chunked size still follow, and are followed by, the kernels of the
    calling thread's stream, which a sleeping kernel holds up for some ms."""
    import torch
    rng = np.random.default_rng(8)
    keys = rng.integers(0, 1 << 62, size=9 << 20, dtype=np.uint64)  # 72 MiB of keys, 9 MiB of flags
    keys[1::2] = keys[::2]  # each key twice: the second insert promotes it
    bits = 1 << 27          # 16 MiB per tier
    want = spk.TwoTierFilter(bits, ctx=spk.Context(0))
    promoted, tiers, solid = want.insert_batch(keys), want.download(), want.is_solid_batch(keys)
    ctx = spk.Context(0)
    ctx.set_stream(2)
    per_thread = torch.cuda.ExternalStream(2)

    def busy():
        with torch.cuda.stream(per_thread):
            torch.cuda._sleep(40_000_000)

    f = spk.TwoTierFilter(bits, ctx=ctx)
    busy()
    np.testing.assert_array_equal(f.insert_batch(keys), promoted)
    busy()
    for a, b in zip(f.download(), tiers):
        np.testing.assert_array_equal(a, b)
    busy()
    np.testing.assert_array_equal(f.is_solid_batch(keys), solid)
    f.close()
    want.close()
