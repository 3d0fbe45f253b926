"""Entry points whose pageable copies are large enough (8 MiB) for the context's
pinned chunks (csrc/spk_xfer.cu): filter, ingest, corrector and tier downloads,
with sizes that leave a partial last piece.  Integer data, compared bit for bit
with the oracle, or with the same work in batches too small for the chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHUNKED = 8 << 20


@pytest.fixture(scope="module")
def spk(spk_lib):
    return spk_lib


def test_filter(spk):
    """Inserts and queries of u64 and Kmer256 keys in one call and in calls of
    under 8 MiB (a batch equals per-key calls in order); flags of over 8 MiB and
    tiers whose size is no whole number of pieces."""
    rng = np.random.default_rng(1)
    bits = 70_000_001
    a, b = spk.TwoTierFilter(bits), spk.TwoTierFilter(bits)
    n = (8 << 20) + 12_345
    keys = rng.integers(0, 1 << 62, size=n, dtype=np.uint64)
    keys[n // 2:] = keys[rng.integers(0, n // 2, size=n - n // 2)]
    step = 700_001
    got = a.insert_batch(keys)
    assert got.nbytes > CHUNKED
    np.testing.assert_array_equal(got, np.concatenate([b.insert_batch(keys[i:i + step]) for i in range(0, n, step)]))
    q = rng.permutation(keys)
    np.testing.assert_array_equal(a.is_solid_batch(q),
                                  np.concatenate([b.is_solid_batch(q[i:i + step]) for i in range(0, n, step)]))
    wide = rng.integers(0, 1 << 62, size=(300_007, 4), dtype=np.uint64)
    wide[150_000:] = wide[:150_007]
    assert wide.nbytes > CHUNKED
    step = 200_000
    for f in ("insert_kmer256_batch", "is_solid_kmer256_batch"):
        np.testing.assert_array_equal(
            getattr(a, f)(wide),
            np.concatenate([getattr(b, f)(wide[i:i + step]) for i in range(0, wide.shape[0], step)]))
    for x, y in zip(a.download(), b.download()):
        assert x.nbytes > CHUNKED and x.nbytes % (4 << 20)
        np.testing.assert_array_equal(x, y)


def test_ingest_and_store(spk, ora):
    """A FASTQ text of 80 MB whose store has over 8 MiB of packed bases and of
    offsets, against the oracle's store."""
    rng = np.random.default_rng(2)
    n, length = 1_100_003, 31
    head = np.frombuffer(b"@r\n", np.uint8)
    bases = np.frombuffer(b"ACGT", np.uint8)[rng.integers(0, 4, size=(n, length))]
    mid = np.frombuffer(b"\n+\n", np.uint8)
    qual = np.full((n, length), ord("I"), np.uint8)
    text = np.concatenate([np.tile(head, (n, 1)), bases, np.tile(mid, (n, 1)), qual,
                           np.full((n, 1), ord("\n"), np.uint8)], axis=1).tobytes()
    want = ora.Packed.from_texts(text).arrays()
    dev = spk.ingest(text)
    got, side = dev.download()
    assert len(text) > CHUNKED and got.data.nbytes > CHUNKED and got.offsets.nbytes > CHUNKED and not side
    np.testing.assert_array_equal(got.data, want[0])
    np.testing.assert_array_equal(got.offsets, want[1])
    np.testing.assert_array_equal(got.lengths, want[2])
    dev.close()


def test_corrector(spk):
    """Packed reads and offsets of over 8 MiB corrected in one call and in calls
    of under 8 MiB (reads are corrected one by one)."""
    rng = np.random.default_rng(3)
    k, length, n = 21, 32, 1_200_001
    g = rng.integers(0, 4, 50_000, dtype=np.uint8)
    start = rng.integers(0, g.size - length, n)
    codes = g[start[:, None] + np.arange(length)[None, :]]
    hit = rng.random(n) < 0.2
    at = rng.integers(0, length, n)
    codes[hit, at[hit]] = (codes[hit, at[hit]] + 1) % 4
    q = codes.reshape(n, length // 4, 4)
    data = ((q[:, :, 0] << 6) | (q[:, :, 1] << 4) | (q[:, :, 2] << 2) | q[:, :, 3]).reshape(-1)
    offs = np.arange(n, dtype=np.uint64) * (length // 4)
    lens = np.full(n, length, np.uint32)
    assert data.nbytes > CHUNKED and offs.nbytes > CHUNKED
    # the genome's k-mers, inserted twice
    gp = np.packbits(((g[:, None] >> np.array([1, 0], np.uint8)) & 1).reshape(-1))
    r = spk.count((gp, np.zeros(1, np.uint64), np.array([g.size], np.uint32)), [k], bloom_bits=1 << 24,
                  list_min_count=1, min_count=1, flags=0x10)
    kmers, _ = r.kmers(0, 1)
    wide = np.zeros((kmers.shape[0], 4), np.uint64)
    wide[:, :kmers.shape[1]] = kmers
    f = spk.TwoTierFilter(1 << 24)
    f.insert_kmer256_batch(wide)
    f.insert_kmer256_batch(wide)
    got, flags, nc = f.correct_reads((data, offs, lens), k)
    step = 400_000
    total = 0
    for i in range(0, n, step):
        m = min(step, n - i)
        d = data[i * 8:(i + m) * 8]
        w, wf, wn = f.correct_reads((d, offs[:m], lens[:m]), k)
        np.testing.assert_array_equal(got.data[i * 8:(i + m) * 8], w.data)
        np.testing.assert_array_equal(flags[i:i + m], wf)
        total += wn
    assert nc == total


def test_result_tiers(spk, ora):
    """Tiers of 12.5 MB of a count."""
    from spk import synth
    p = synth.sample(5_000, 30.0, seed=4, ks=(31,)).packed
    bits = 100_000_001
    r = spk.count(p, [31], bloom_bits=bits, flags=spk.SPK_F_KEEP_BLOOM)
    o = ora.count(p.data, p.offsets, p.lengths, 31, bits, mode=ora.MODE_TWICE)
    seen, twice = r.bloom(0)
    assert seen.nbytes > CHUNKED and seen.nbytes % (4 << 20)
    for a, b in zip((seen, twice), o.bloom()):
        np.testing.assert_array_equal(a, b)
