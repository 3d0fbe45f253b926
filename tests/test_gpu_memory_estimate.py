"""The memory estimate that admits batch and serving jobs (spk_job_hbm_estimate)
against what counts hold: the high-water mark of the device memory pool, in a
process of its own.  The estimate is not under it, or jobs admitted side by side
would not fit, and not far above (a quarter of the slots taken as solid k-mers,
request sizes rounded up, the kept lists: up to two and a half times)."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import sys
sys.path.insert(0, sys.argv[1])
import ctypes, torch, spk
from spk import synth
torch.zeros(1, device="cuda")
rt = ctypes.CDLL([l.split()[-1] for l in open("/proc/self/maps") if "libcudart" in l][0])
pool, used_high = ctypes.c_void_p(), 8  # cudaMemPoolAttrUsedMemHigh
assert rt.cudaDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0
ctx = spk.default_context()
for genome, cov in ((1_000_000, 100.0), (2_000_000, 20.0)):
    p = synth.sample(genome, cov, seed=2, ks=(21,)).packed
    for k in (21, 31, 55, 77):
        for flags in (spk.SPK_F_EDGES, spk.SPK_F_EDGES | spk.SPK_F_CORRECT):
            est = spk.Server.estimate(spk.Job(p, [k], dict(flags=flags)))
            v = ctypes.c_uint64(0)
            assert rt.cudaMemPoolSetAttribute(pool, used_high, ctypes.byref(v)) == 0
            spk.count(p, [k], flags=flags).close()
            assert rt.cudaMemPoolGetAttribute(pool, used_high, ctypes.byref(v)) == 0
            print("k=%d x%g flags=%#x estimate %.0f MB, high-water mark %.0f MB" % (k, cov, flags, est / 1e6, v.value / 1e6))
            assert v.value <= est <= 2.5 * v.value
print("done")
"""


def test_estimate_covers_the_high_water_mark(spk_lib):
    r = subprocess.run([sys.executable, "-c", CHILD, os.path.join(ROOT, "spades-rs_b200")], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "done" in r.stdout, r.stdout + r.stderr[-3000:]
