"""The correcting count on a device with little memory left: its counted lists do
not fit, and it takes the reference's two passes, which need less, to the same
result.  In a process of its own, whose device memory pool starts empty."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np, torch, spk
from spk import synth
k, bits = int(sys.argv[2]), 1 << 26
flags = spk.SPK_F_EDGES | spk.SPK_F_CORRECT
warm = synth.sample(3_000, 20.0, seed=1, ks=(k,)).packed  # loads the kernels
spk.count(warm, [k], bloom_bits=1 << 20, flags=flags).close()
p = synth.sample(400_000, 100.0, seed=2, ks=(k,)).packed
free = torch.cuda.mem_get_info()[0]
filler = torch.empty(free - (int(sys.argv[3]) << 20), dtype=torch.uint8, device="cuda")

def run():
    r = spk.count(p, [k], bloom_bits=bits, list_min_count=1, flags=flags)
    return r, r.info(0), r.kmers(0, 1), r.edges(0)

r1, i1, l1, e1 = run()
del filler
torch.cuda.empty_cache()
r2, i2, l2, e2 = run()
# (the table of the two passes has room for the admitted k-mers alone)
assert i1["table_capacity"] < i2["table_capacity"], (i1["table_capacity"], i2["table_capacity"])
for name in ("cutoff", "occurrences", "n_table", "n_solid", "n_edges", "n_singletons", "n_corrected_reads", "seen_popcount",
             "twice_popcount"):
    assert i1[name] == i2[name], name
assert np.array_equal(l1[0], l2[0]) and np.array_equal(l1[1], l2[1]) and np.array_equal(e1, e2)
print("same", i1["n_table"])
"""


@pytest.mark.parametrize("k,left_mib", [(31, 300), (55, 500)])
def test_little_memory(spk_lib, k, left_mib):
    r = subprocess.run([sys.executable, "-c", CHILD, os.path.join(ROOT, "spades-rs_b200"), str(k), str(left_mib)],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same" in r.stdout, r.stdout + r.stderr[-3000:]
