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
