"""The default job where one minimizer bin holds far more than its share: the
minimizer partition gives such a job up and it is counted another way, with the
same results."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def spk(spk_lib):
    return spk_lib


def pack(codes):
    """2-bit bytes of equally long reads (rows of base codes)."""
    n, length = codes.shape
    pad = np.zeros((n, -(-length // 4) * 4), np.uint8)
    pad[:, :length] = codes
    q = pad.reshape(n, -1, 4)
    return (q[:, :, 0] << 6) | (q[:, :, 1] << 4) | (q[:, :, 2] << 2) | q[:, :, 3]


def check(spk, ora, r, rows, k, bits, hot=None):
    """Result r (list_min_count 1, tiers kept) against the oracle on rows.  hot: the
    count of the one k-mer that rows hold three times in place of all its reads."""
    data = pack(rows)
    n, nb = data.shape
    offs, lens = np.arange(n, dtype=np.uint64) * nb, np.full(n, rows.shape[1], np.uint32)
    o = ora.count(data.reshape(-1), offs, lens, k, bits, mode=ora.MODE_TWICE, threads=os.cpu_count() or 1)
    tk, tc = o.table(1)
    if hot is not None:
        tc = np.where(tc == 3, hot, tc).astype(np.uint32)
    gk, gc = r.kmers(0, 1)
    np.testing.assert_array_equal(gk, tk)
    np.testing.assert_array_equal(gc, tc)
    for a, b in zip(r.bloom(0), o.bloom()):
        np.testing.assert_array_equal(a, b)
    info = r.info(0)
    assert info["cutoff"] == ora.cutoff(tc, 5.0)
    sk, _ = r.solid(0)
    np.testing.assert_array_equal(r.edges(0), ora.edges(sk, k))


def test_more_records_than_a_reference_holds(spk, ora):
    """34 million reads of one 33-mer among others: the batch of its minimizer has
    more than 2^25 records, which one CTA finds while the others count."""
    import torch
    k, n, bits = 33, 34_000_000, 1 << 24
    rng = np.random.default_rng(5)
    rest = np.repeat(rng.integers(0, 4, size=(200_000, k), dtype=np.uint8), 2, axis=0)  # each k-mer twice
    hot = rng.integers(0, 4, size=(1, k), dtype=np.uint8)
    nb = -(-k // 4)
    m = rest.shape[0]
    data = torch.zeros((n + m) * nb + 64, dtype=torch.uint8, device="cuda")
    view = data[:(n + m) * nb].view(n + m, nb)
    view[:n] = torch.from_numpy(pack(hot)).cuda()
    view[n:] = torch.from_numpy(pack(rest)).cuda()
    offs = torch.arange(n + m, device="cuda", dtype=torch.int64) * nb
    lens = torch.full((n + m,), k, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    r = spk.count_device(data.data_ptr(), (n + m) * nb, offs.data_ptr(), lens.data_ptr(), n + m, [k], bloom_bits=bits,
                         list_min_count=1, flags=spk.SPK_F_EDGES | spk.SPK_F_KEEP_BLOOM)
    assert r.info(0)["occurrences"] == n + m
    check(spk, ora, r, np.concatenate([rest, np.repeat(hot, 3, axis=0)]), k, bits, hot=n)


def small_hash_mmer(m):
    """An m-mer of a small hash (sk_hash in csrc/spk_superk.cuh), as base codes: the
    minimizer of nearly every window that holds it."""
    rng = np.random.default_rng(m)
    code = rng.integers(0, 1 << (2 * m), size=1 << 20, dtype=np.uint64)
    rev, x = np.zeros_like(code), code.copy()
    for _ in range(m):
        rev = (rev << np.uint64(2)) | (np.uint64(3) - (x & np.uint64(3)))
        x >>= np.uint64(2)
    h = (np.minimum(code, rev).astype(np.uint32) ^ np.uint32(0x2545F491)) * np.uint32(0x9E3779B1)
    h = (h ^ (h >> np.uint32(15))) * np.uint32(0x2C1B3C6D)
    h ^= h >> np.uint32(13)
    c = int(code[np.argmin(h)])
    return np.array([(c >> (2 * (m - 1 - i))) & 3 for i in range(m)], np.uint8)


def planted(k, n, seed):
    """n reads of random bases around one m-mer: every window of every read has it
    as its minimizer, and nearly every one is a k-mer of its own."""
    m = 15 if k > 32 else 13 if k >= 27 else 11
    rows = np.random.default_rng(seed).integers(0, 4, size=(n, 2 * k - m), dtype=np.uint8)
    rows[:, k - m:k] = small_hash_mmer(m)
    return rows


@pytest.mark.parametrize("k,n,given_up", [(21, 1_000, 0), (21, 3_000, 1), (55, 300, 0), (55, 3_000, 1),
                                          (31, 3_000, 1), (127, 100, 0), (77, 2_000, 1), (127, 3_000, 1)])
def test_one_minimizer_of_many_kmers(spk, ora, k, n, given_up):
    """A bin with a few times a table's k-mers is counted in parts; one with many
    times that is not (its parts would each read all of it: the work grew with the
    square of the reads) but by spans or, for a small set, in the table."""
    rows = planted(k, n, seed=k)
    rng = np.random.default_rng(k + 1)
    # (k > 64: enough occurrences for the super-k-mers to take the set)
    extra = rng.integers(0, 4, size=(0 if k <= 64 else 20_000, rows.shape[1]), dtype=np.uint8)
    rows = np.concatenate([rows, rows[: n // 2], extra])
    data = pack(rows)
    nb = data.shape[1]
    offs, lens = np.arange(rows.shape[0], dtype=np.uint64) * nb, np.full(rows.shape[0], rows.shape[1], np.uint32)
    r = spk.count((data.reshape(-1), offs, lens), [k], bloom_bits=1 << 24, list_min_count=1,
                  flags=spk.SPK_F_EDGES | spk.SPK_F_KEEP_BLOOM)
    assert r.info(0)["part_rescatters"] == given_up
    check(spk, ora, r, rows, k, 1 << 24)


@pytest.mark.parametrize("k", [21, 55])
def test_correcting_count_gives_up_too(spk, ora, k):
    """The correcting count of such reads takes the reference's two passes."""
    rows = np.repeat(planted(k, 3_000, seed=k), 2, axis=0)
    rows[::7, 3] = (rows[::7, 3] + 1) % 4
    data = pack(rows)
    nb = data.shape[1]
    n = rows.shape[0]
    offs, lens = np.arange(n, dtype=np.uint64) * nb, np.full(n, rows.shape[1], np.uint32)
    bits = 1 << 22
    o = ora.count(data.reshape(-1), offs, lens, k, bits, mode=ora.MODE_TWICE, correct=True)
    tk, tc = o.table(1)
    r = spk.count((data.reshape(-1), offs, lens), [k], bloom_bits=bits, list_min_count=1,
                  flags=spk.SPK_F_EDGES | spk.SPK_F_KEEP_BLOOM | spk.SPK_F_CORRECT)
    gk, gc = r.kmers(0, 1)
    np.testing.assert_array_equal(gk, tk)
    np.testing.assert_array_equal(gc, tc)
    for a, b in zip(r.bloom(0), o.bloom()):
        np.testing.assert_array_equal(a, b)
    assert r.info(0)["n_corrected_reads"] == o.stats()["corrected_reads"]


def test_deep_locus(spk, ora):
    """One locus of 400 bases read 60,000 times with errors: few minimizers, each
    with thousands of records and of k-mers."""
    rng = np.random.default_rng(9)
    g = rng.integers(0, 4, 400, dtype=np.uint8)
    start = rng.integers(0, 400 - 120, 60_000)
    rows = g[start[:, None] + np.arange(120)[None, :]]
    e = rng.random(rows.shape) < 0.004
    rows[e] = (rows[e] + 1) % 4
    data = pack(rows)
    nb = data.shape[1]
    n = rows.shape[0]
    offs, lens = np.arange(n, dtype=np.uint64) * nb, np.full(n, 120, np.uint32)
    r = spk.count((data.reshape(-1), offs, lens), [55], bloom_bits=1 << 24, list_min_count=1,
                  flags=spk.SPK_F_EDGES | spk.SPK_F_KEEP_BLOOM)
    check(spk, ora, r, rows, 55, 1 << 24)


def test_more_bloom_operations_than_room(spk, ora):
    """Distinct k-mers that fit the singletons' buffer and the list's, but whose Bloom
    operations overflow theirs (1.4 of the slots): counted once more with room."""
    rng = np.random.default_rng(6)
    slots, k, bits = 1 << 17, 31, 1 << 24
    once = rng.integers(0, 4, size=(int(0.93 * slots) // 101, 131), dtype=np.uint8)
    more = rng.integers(0, 4, size=(int(0.47 * slots) // 101, 131), dtype=np.uint8)
    rows = np.concatenate([once, np.repeat(more, 5, axis=0)])
    assert slots / 2 < 0.3 * rows.shape[0] * 101 < slots
    data = pack(rows)
    n, nb = data.shape
    offs, lens = np.arange(n, dtype=np.uint64) * nb, np.full(n, 131, np.uint32)
    r = spk.count((data.reshape(-1), offs, lens), [k], bloom_bits=bits, list_min_count=1,
                  flags=spk.SPK_F_EDGES | spk.SPK_F_KEEP_BLOOM)
    info = r.info(0)
    assert info["table_regrows"] == 1 and info["part_rescatters"] == 0
    check(spk, ora, r, rows, k, bits)
