"""Timed cases of the k-mer counting library: what a program built on it has it do.

Every case goes through the public entry points (the ``spk`` package and the
C ABI behind it) and returns whole outputs: the solid list, the edge list, the
unitigs, the packed store.  Inputs are synthetic paired-end-like reads of the
shapes the benchmark and the tests use (uniform or GC-skewed genomes with a few
inserted repeats, substitution errors rising along the read, 20-150x), drawn
from the seed on the GPU.

Kinds
  count   one counting job on reads already in device memory (the serving and
          multi-k form: reads stay resident), the solid list and the edges
          into pinned buffers that the caller keeps
  host    the same job from pageable host arrays, as a first call has them
  multik  one call over several k, as the per-k assembly loop makes it
  batch   independent uneven samples through the batch pipeline
  unitigs a count followed by the unitig compaction of its solid k-mers
  correct the count with read error correction
  ingest  FASTQ texts to the packed store, brought back to the host
  filter  the two-tier Bloom filter on its own: batched inserts and queries
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "spades-rs_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import spk  # noqa: E402

MI = 1 << 20


def listed():
    return [
        # the smallest calls: a plasmid- or amplicon-sized sample, where launches and readbacks count
        dict(name="amplicon_k31", kind="count", k=31, genome=10_000, cov=30.0, read_len=150, ragged=False,
             gc=0.5, bloom_bits=16 * MI),
        # the plain single-sample configuration (1 Mb, 30x, k = 21, one-limb keys)
        dict(name="small_k21", kind="count", k=21, genome=1_000_000, cov=30.0, read_len=150, ragged=False,
             gc=0.5, bloom_bits=512 * MI),
        # the large isolate, device-resident: the headline job (5 Mb, 100x, k = 55)
        dict(name="isolate_k55", kind="count", k=55, genome=5_000_000, cov=100.0, read_len=150, ragged=False,
             gc=0.5, bloom_bits=512 * MI),
        # three-limb keys on reads of uneven length (trimmed reads and N-split sub-reads)
        dict(name="ragged_k77", kind="count", k=77, genome=2_000_000, cov=60.0, read_len=150, ragged=True,
             gc=0.45, bloom_bits=512 * MI),
        # the largest k on longer reads (2 x 250 bp), a Bloom that is no power of two
        dict(name="long_k127", kind="count", k=127, genome=1_500_000, cov=70.0, read_len=250, ragged=False,
             gc=0.55, bloom_bits=300_000_000),
        # a first call on host arrays (pageable), GC-poor genome, two-limb keys just above one limb
        dict(name="host_k33", kind="host", k=33, genome=3_000_000, cov=60.0, read_len=150, ragged=True, gc=0.35,
             bloom_bits=512 * MI),
        # the per-k loop of a multi-k assembly
        dict(name="multik", kind="multik", k=0, genome=1_200_000, cov=50.0, read_len=150, ragged=False, gc=0.5,
             bloom_bits=512 * MI),
        # uneven samples (0.05-1.2 Mb, 20-200x, GC 30-70%) at k = 33 as one batch
        dict(name="batch_k33", kind="batch", k=33, genome=500_000, cov=80.0, read_len=150, ragged=False, gc=0.5,
             bloom_bits=512 * MI, samples=12),
        # count and graph step: solid k-mers to unitigs
        dict(name="unitigs_k55", kind="unitigs", k=55, genome=3_000_000, cov=60.0, read_len=150, ragged=False,
             gc=0.5, bloom_bits=512 * MI),
        # the error-correcting count (the default of the assembler's pipeline test, k = 31)
        dict(name="correct_k31", kind="correct", k=31, genome=1_000_000, cov=40.0, read_len=150, ragged=True,
             gc=0.5, bloom_bits=512 * MI),
        # FASTQ pairs to the store (both texts; 0.5 Mb at 60x)
        dict(name="ingest", kind="ingest", k=0, genome=500_000, cov=60.0, read_len=150, ragged=False, gc=0.5,
             bloom_bits=0),
        # the filter alone: 1 M inserts (each key up to a few times), then queries half of which were inserted
        dict(name="filter", kind="filter", k=55, genome=1_000_000, cov=1.0, read_len=0, ragged=False, gc=0.5,
             bloom_bits=64 * MI),
    ]


def _logu(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["count"] * 5 + ["host", "multik", "batch", "unitigs", "correct", "ingest", "filter"])
    k = rng.choice([21, 25, 31, 33, 41, 55, 63, 77, 89, 99, 127])
    read_len = rng.choice([100, 125, 150, 250])
    if k >= read_len - 20:
        read_len = 250
    bases = _logu(rng, 3e5, 4e8 if kind == "count" and k <= 64 else 1.5e8)
    cov = _logu(rng, 20, 150)
    c = dict(kind=kind, k=k, genome=int(min(max(bases / cov, 5_000), 5e6)) | 1, cov=round(cov, 2), read_len=read_len,
             ragged=rng.random() < 0.4, gc=round(rng.uniform(0.3, 0.7), 3),
             bloom_bits=rng.choice([16 * MI, 64 * MI, 100_000_000, 512 * MI, 512 * MI]))
    if kind == "multik":
        c.update(k=0, genome=min(c["genome"], 1_200_000), cov=min(c["cov"], 50.0))
    elif kind == "batch":
        c.update(samples=rng.randint(3, 12), k=rng.choice([21, 33, 55]), read_len=150,
                 genome=int(_logu(rng, 50_000, 350_000)), cov=min(c["cov"], 80.0))
    elif kind == "correct":
        c.update(k=rng.choice([21, 31, 55]), genome=min(c["genome"], 1_000_000), cov=min(c["cov"], 40.0), read_len=150)
    elif kind == "unitigs":
        c.update(k=rng.choice([21, 31, 55, 63]), cov=max(c["cov"], 60.0), genome=min(c["genome"], 1_500_000),
                 read_len=rng.choice([150, 250]))
    elif kind == "ingest":
        c.update(k=0, ragged=False, bloom_bits=0, genome=min(c["genome"], 500_000), cov=min(c["cov"], 60.0))
    elif kind == "filter":
        c.update(genome=int(_logu(rng, 1, 1_000_000)), cov=1.0, read_len=0, ragged=False,
                 bloom_bits=rng.choice([16 * MI, 64 * MI, 100_000_000]))
    return c


# ---- inputs ---------------------------------------------------------------
def _gen(seed, stream=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1_000_003 + stream) & 0x7FFFFFFF)
    return g


def _genome(case, g):
    n = case["genome"]
    u = torch.rand(n, generator=g, device="cuda")
    gc = case["gc"]
    at = (1 - gc) / 2
    codes = (u >= at).to(torch.uint8) + (u >= at + gc / 2).to(torch.uint8) + (u >= at + gc).to(torch.uint8)
    for i in range(20 if n >= 200_000 else 0):  # repeat copies of 1-5 kb at 99% identity
        ln = 1000 + int(torch.randint(0, 4001, (1,), generator=g, device="cuda"))
        a, b = torch.randint(0, n - ln, (2,), generator=g, device="cuda").tolist()
        seg = codes[a:a + ln].clone()
        m = torch.rand(ln, generator=g, device="cuda") < 0.01
        seg = torch.where(m, (seg + 1) % 4, seg)
        codes[b:b + ln] = seg
    return codes


def _read_codes(case, g, codes, n, length):
    """n reads of `length` bases (codes), substitutions rising from 0.1% to 1.0% along the read."""
    start = (torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (codes.numel() - length + 1)).long()
    idx = start[:, None] + torch.arange(length, device="cuda")[None, :]
    fwd = codes[idx]
    rev = (3 - fwd).flip(1)
    minus = torch.rand(n, generator=g, device="cuda") < 0.5
    r = torch.where(minus[:, None], rev, fwd)
    rate = torch.linspace(0.001, 0.010, length, device="cuda")[None, :]
    err = torch.rand((n, length), generator=g, device="cuda") < rate
    sub = torch.randint(1, 4, (n, length), generator=g, device="cuda", dtype=torch.uint8)
    return torch.where(err, (r + sub) % 4, r)


def _pack(codes):
    n, length = codes.shape
    nb = (length + 3) // 4
    pad = torch.zeros((n, nb * 4), dtype=torch.uint8, device="cuda")
    pad[:, :length] = codes
    q = pad.view(n, nb, 4)
    return (q[:, :, 0] << 6) | (q[:, :, 1] << 4) | (q[:, :, 2] << 2) | q[:, :, 3]


def _reads(case, seed, stream=0):
    """Packed reads on the device: (data with 64 spare bytes, bytes, offsets, lengths)."""
    g = _gen(seed, stream)
    codes = _genome(case, g)
    length = min(case["read_len"], codes.numel())
    n = max(2, int(case["genome"] * case["cov"] / length))
    parts, lens = [], []
    for a in range(0, n, 400_000):
        m = min(400_000, n - a)
        r = _read_codes(case, g, codes, m, length)
        ln = torch.full((m,), length, dtype=torch.int32, device="cuda")
        if case["ragged"]:  # a third of the reads trimmed or split
            cut = torch.rand(m, generator=g, device="cuda") < 0.33
            t = torch.randint(21, length + 1, (m,), generator=g, device="cuda", dtype=torch.int32)
            ln = torch.where(cut, t, ln)
            r = torch.where(torch.arange(length, device="cuda")[None, :] < ln[:, None], r, torch.zeros_like(r))
            p = _pack(r)
            p = p[torch.arange(p.shape[1], device="cuda")[None, :] < ((ln + 3) // 4)[:, None]]
        else:
            p = _pack(r).reshape(-1)
        parts.append(p)
        lens.append(ln)
    lengths = torch.cat(lens)
    nb = (lengths.long() + 3) // 4
    offsets = torch.cumsum(nb, 0) - nb
    nbytes = int(nb.sum())
    data = torch.zeros(nbytes + 64, dtype=torch.uint8, device="cuda")
    data[:nbytes] = torch.cat(parts)
    return data, nbytes, offsets, lengths


def _host(reads):
    data, nbytes, offsets, lengths = reads
    return spk.PackedReads(data[:nbytes].cpu().numpy(), offsets.cpu().numpy().astype(np.uint64),
                           lengths.cpu().numpy().astype(np.uint32))


def _zeros(*shape, dtype=np.uint64):
    """A pinned, cleared host array (the caller's; kept from call to call)."""
    t = torch.zeros(math.prod(shape), dtype={8: torch.int64, 4: torch.int32, 1: torch.uint8}[np.dtype(dtype).itemsize],
                    pin_memory=True)
    return t.numpy().view(dtype).reshape(shape)


def _out_buffers(case, k, edges=True):
    """Buffers for the solid list and the edges of one sample; what a job does not fill stays zero."""
    n = 2 * case["genome"] + 65_536
    out = dict(cap=n, keys=_zeros(n, spk.nlimbs(k)), counts=_zeros(n, dtype=np.uint32))
    if edges:
        out["edges"] = _zeros(n, spk.nlimbs(k + 1))
    return out


def _fastq(case, seed):
    g = _gen(seed)
    codes = _genome(case, g)
    length = min(case["read_len"], codes.numel())
    n = max(2, int(case["genome"] * case["cov"] / length / 2))
    texts = []
    for mate in (1, 2):
        r = _read_codes(case, g, codes, n, length)
        letters = torch.tensor(list(b"ACGT"), dtype=torch.uint8, device="cuda")[r.long()]
        isn = torch.rand((n, length), generator=g, device="cuda") < 0.0005  # bases set to N
        letters = torch.where(isn, torch.full_like(letters, ord("N")), letters)
        qual = torch.randint(33 + 20, 33 + 41, (n, length), generator=g, device="cuda", dtype=torch.uint8)
        ids = torch.arange(n, device="cuda")
        digits = torch.stack([(ids // 10 ** d) % 10 + 48 for d in range(8, -1, -1)], 1).to(torch.uint8)

        def col(s):
            return torch.tensor(list(s), dtype=torch.uint8, device="cuda")[None, :].expand(n, len(s))

        rec = torch.cat([col(b"@read"), digits, col(b"/%d\n" % mate), letters, col(b"\n+\n"), qual, col(b"\n")], 1)
        texts.append(rec.contiguous().cpu().numpy().tobytes())
    return texts


def _samples(case):
    """Genome size, GC and coverage of each sample of a batch (the seed draws the bases and the reads)."""
    g = np.random.default_rng(case["genome"])
    out = []
    for _ in range(case["samples"]):
        f = math.exp(g.uniform(math.log(0.1), math.log(2.4)))
        out.append(dict(case, genome=max(5_000, int(case["genome"] * f)), gc=float(g.uniform(0.3, 0.7)),
                        cov=float(case["cov"] * g.uniform(0.25, 2.5))))
    return out


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, ctx=spk.default_context())
    if kind in ("count", "correct", "unitigs", "multik"):
        st["reads"] = _reads(case, seed)
        st["ks"] = [case["k"]] if case["k"] else [21, 33, 55, 77]
        st["out"] = [_out_buffers(case, k, edges=kind != "unitigs") for k in st["ks"]]
        if kind == "unitigs":
            n = case["genome"] // 2 + 65_536
            st["unitigs"] = [_zeros(16 * case["genome"] + 65_536, dtype=np.uint8), _zeros(n), _zeros(n, dtype=np.float64),
                             _zeros(n)]
    elif kind == "host":
        st["packed"] = _host(_reads(case, seed))
        st["out"] = [_out_buffers(case, case["k"])]
    elif kind == "batch":
        st["samples"] = [_host(_reads(c, seed, 1 + i)) for i, c in enumerate(_samples(case))]
        st["out"] = [_out_buffers(c, case["k"], edges=False) for c in _samples(case)]
    elif kind == "ingest":
        st["texts"] = _fastq(case, seed)
        n = len(st["texts"][0]) // case["read_len"]  # reads of both files, with room for N-split pieces
        st["store"] = [_zeros(n * (case["read_len"] // 4 + 2), dtype=np.uint8), _zeros(n), _zeros(n, dtype=np.uint32)]
    elif kind == "filter":
        g = np.random.default_rng(seed)
        n = case["genome"]
        uniq = g.integers(0, 1 << 64, size=(n, 4), dtype=np.uint64)
        lo, hi = 2 * min(case["k"], 64), 2 * max(case["k"] - 64, 0)  # bits of Kmer256.lo and .hi
        for limb, bits in enumerate((min(lo, 64), max(lo - 64, 0), min(hi, 64), max(hi - 64, 0))):
            uniq[:, limb] &= np.uint64((1 << bits) - 1)
        st["keys"] = np.ascontiguousarray(uniq[g.integers(0, max(1, n // 2), size=n)])
        st["queries"] = np.ascontiguousarray(uniq[g.permutation(n)])
    torch.cuda.synchronize()
    return st


# ---- one pass -------------------------------------------------------------
def _stats(info):
    return np.array([info[f] for f in ("cutoff", "occurrences", "admitted_occurrences", "n_table", "n_solid", "n_edges",
                                       "n_singletons", "n_distinct", "seen_popcount", "twice_popcount")], dtype=np.int64)


def _ptr(a):
    return a.ctypes.data_as(ctypes.POINTER({8: ctypes.c_uint64, 4: ctypes.c_uint32, 1: ctypes.c_uint8}[a.itemsize]))


def _ok(rc):
    if rc:
        raise spk.SpkError(rc, "call failed")


def _lists(out, r, i):
    """The solid list (already there when the count copied it) and the edges of the i-th k into the caller's buffers."""
    info = r.info(i)
    if not info["solid_copied"]:
        r.solid(i, out=(out["keys"], out["counts"]))
    res = [out["keys"], out["counts"]]
    if "edges" in out:
        m = ctypes.c_size_t(out["cap"])
        _ok(spk.lib().spk_result_edges(r.h, i, _ptr(out["edges"]), ctypes.byref(m)))
        res.append(out["edges"])
    return res + [_stats(info)]


def run(st):
    case = st["case"]
    kind, bits = case["kind"], case["bloom_bits"]
    if kind in ("count", "correct", "unitigs", "multik", "host"):
        kw = dict(ctx=st["ctx"], bloom_bits=bits)
        if kind != "unitigs":
            kw["solid_out"] = (st["out"][0]["keys"], st["out"][0]["counts"])
        if kind == "correct":
            kw["flags"] = spk.SPK_F_EDGES | spk.SPK_F_CORRECT
        if kind == "host":
            r = spk.count(st["packed"], [case["k"]], **kw)
        else:
            data, nbytes, offsets, lengths = st["reads"]
            r = spk.count_device(data.data_ptr(), nbytes, offsets.data_ptr(), lengths.data_ptr(), lengths.numel(),
                                 st["ks"], **kw)
        if kind == "unitigs":
            seqs, lens, cov, nk = st["unitigs"]
            nb, n = ctypes.c_uint64(seqs.size), ctypes.c_uint64(lens.size)
            _ok(spk.lib().spk_result_unitigs(r.h, 0, seqs.ctypes.data_as(ctypes.c_char_p), ctypes.byref(nb), _ptr(lens),
                                             cov.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), _ptr(nk),
                                             ctypes.byref(n)))
            res = [seqs, lens, cov, nk, _stats(r.info(0))]
        else:
            res = [_lists(out, r, i) for i, out in enumerate(st["out"])]
        r.close()
        return res
    if kind == "batch":
        jobs = [spk.Job(p, [case["k"]], dict(bloom_bits=bits)) for p in st["samples"]]
        res = []
        for i, r in spk.count_batch_iter(jobs, ctx=st["ctx"]):
            res.append(_lists(st["out"][i], r, 0))
            r.close()
        return res
    if kind == "ingest":
        d = spk.ingest(st["texts"][0], st["texts"][1], ctx=st["ctx"])
        info = d.info()
        data, offsets, lengths = st["store"]
        if info["data_len"] > data.size or info["n_reads"] > offsets.size:
            raise MemoryError("the store is larger than the caller's buffers")
        _ok(spk.lib().spk_packed_download(d.h, data.ctypes.data, offsets.ctypes.data, lengths.ctypes.data, None, None))
        d.close()
        return [data, offsets, lengths, info["n_reads"], info["data_len"], info["pe_count"], info["n_sidecar"]]
    f = spk.TwoTierFilter(bits, ctx=st["ctx"])
    promoted = f.insert_kmer256_batch(st["keys"])
    solid = f.is_solid_kmer256_batch(st["queries"])
    res = [promoted, solid, *f.download()]
    f.close()
    return res


# ---- what a pass cannot do without ------------------------------------------
def _count_bytes(case, k):
    n_reads = case["genome"] * case["cov"] / case["read_len"]
    read_bytes = n_reads * ((case["read_len"] * (0.85 if case["ragged"] else 1.0) + 3) // 4 + 12)
    lists = case["genome"] * (8 * spk.nlimbs(k) + 4 + 8 * spk.nlimbs(k + 1))
    return read_bytes + 2 * case["bloom_bits"] / 8 + lists


def work(case):
    kind = case["kind"]
    if kind == "multik":
        b = sum(_count_bytes(case, k) for k in (21, 33, 55, 77))
    elif kind == "batch":
        b = case["samples"] * _count_bytes(case, case["k"])
    elif kind == "ingest":
        n = case["genome"] * case["cov"] / case["read_len"]
        b = n * (2 * case["read_len"] + 20) + n * (case["read_len"] / 4 + 12)
    elif kind == "filter":
        b = case["genome"] * (2 * 32 + 2) + 2 * case["bloom_bits"] / 8
    else:
        b = _count_bytes(case, case["k"])
    return {"bytes": int(b), "flops": 0}


def exact(case, seed):
    """Outputs are whole numbers and bytes (keys, counts, edges, packed bases, bits); the unitigs' mean
    coverages are ratios of such numbers, whose 64-bit graph walk in numpy takes minutes."""
    return None
